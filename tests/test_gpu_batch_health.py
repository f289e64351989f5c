"""A member whose field is no longer finite ends a batch's call with
MGPU_E_NONFINITE, but only where the members' control blocks are read: the
other members have made the call's steps by then (its first 50 of more)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["run", "bench_steps"])
@pytest.mark.parametrize("steps,made", [(3, 3), (12, 12), (50, 50), (57, 50)])
def test_members_make_their_steps_beside_a_failed_one(call, steps, made):
    from mgpu import case, common_setup, lib
    cd = common_setup.build_common(case.small_nozzle())
    cd.ints["NSTEPS_MAX"], cd.reals["CONLIM"] = 10 ** 6, 1e-9
    good, bad, alone = (lib.Problem(cd) for _ in range(3))
    ro = cd.arrays["RO"].copy()
    ro[2, 10, 3] = np.nan
    bad.set("RO", ro)
    batch = lib.Batch([good, bad])
    made = steps if call == "bench_steps" else made
    if steps >= 5:
        with pytest.raises(lib.MgpuError) as e:
            getattr(batch, call)(steps)
        assert e.value.code == -5
    else:
        getattr(batch, call)(steps)            # no tail yet: nothing has looked at the field
    alone.run(made)
    for n in ("RO", "ROE", "ROVX", "STEP"):
        assert np.array_equal(good.get(n), alone.get(n)), n
