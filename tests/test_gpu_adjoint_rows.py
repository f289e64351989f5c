"""The transposed step where the last row ends before J = JM: the planes past
it are damped by that row's mean |STORE| too, and their part of its adjoint
counts."""
import numpy as np
import pytest

from helpers import rel_linf
from test_gpu_adjoint import ADJ_STATE, _state_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("past", [0, 3, 6])
def test_planes_past_the_last_row(past):
    from mgpu import case, common_setup, lib
    import oracle as O
    O.build()
    cd = common_setup.build_common(case.small_nozzle())
    cd.arrays["JMIX"][-1] = cd.jm - past
    of = O.Oracle(cd)
    of.setup_calls()
    for _ in range(30):
        of.step()
    for n, a in list(cd.arrays.items()):
        if a.dtype == np.float32:
            cd.arrays[n] = of.get(n, double=False).astype(np.float32)
    cd.ints["NSTEP"], cd.ints["FROZEN"] = 30, 1
    rng = np.random.default_rng(7)
    seeds = {n: rng.standard_normal(cd.arrays[n].shape) * _state_mask(n, cd) for n in ADJ_STATE}
    # the adjoint of the last planes, through which the row's mean is reached
    seeds["DRO"][:, :-past - 1, :] *= 0.0
    oa = O.Oracle(cd, ad=True)
    oa.ad_begin()
    oa.step()
    oa.ad_reverse(seeds)
    gp = lib.Problem(cd, setup_calls=False)
    gp.adjoint_prepare()
    gp.adjoint_objective("none")
    for n in ADJ_STATE:
        gp.adjoint_set(n, seeds[n].astype(np.float32))
    gp.adjoint_iterate(1)
    # as the transposed steps of whole rows: FP32 chains with atomics
    bad = {}
    for n in ADJ_STATE:
        m = _state_mask(n, cd)
        e = rel_linf(gp.adjoint_get(n) * m, oa.ad_grad(n) * m)
        if e > 1e-3:
            bad[n] = e
    assert not bad
