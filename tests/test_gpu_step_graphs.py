"""A march's step graphs all exist before its first step: a run that ends
between two tails, on a step of a kind it has not come to before, takes no more
device memory and does not capture its stream, which another thread may use for
reports meanwhile.  A batch's graphs are all captured with the CTA sizes its
members have, tuned after the batch was made or before."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _deck(steps, nlos=None):
    from mgpu import case, common_setup
    cd = common_setup.build_common(case.small_stage())
    cd.ints["NSTEPS_MAX"], cd.reals["CONLIM"] = steps, 1e-9
    if nlos is not None:
        cd.ints["NLOS"] = nlos
    return cd


def _free():
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("nlos", [1, 3, 5, 10])
def test_no_memory_is_taken_between_the_first_step_and_the_last(nlos):
    from mgpu import lib
    ps = [lib.Problem(_deck(23, nlos)) for _ in range(24)]
    for p in ps:
        p.step()
    free = _free()
    for p in ps:
        assert p.run(100)[0] == 1 and p.step(check=False).nstep == 24
    assert _free() == free


def test_batch_takes_no_memory_after_it_is_made():
    from mgpu import lib
    ps = [lib.Problem(_deck(23 if q % 2 else 27, 3)) for q in range(24)]
    b = lib.Batch(ps)
    b.run(1)
    free = _free()
    for n in (4, 17, 6, 5):                  # kinds 0 to 3, members ended and not
        b.run(n)
    assert _free() == free


def test_reports_of_another_thread_do_not_break_a_march():
    from mgpu import lib
    want = lib.Problem(_deck(23))
    want.run(100)
    for _ in range(10):
        p = lib.Problem(_deck(23))
        p.integrals_noalloc()
        p.step()
        stop, errors = threading.Event(), []

        def report():
            try:
                while not stop.is_set():
                    p.integrals_noalloc()
            except Exception as e:             # noqa: BLE001
                errors.append(e)

        t = threading.Thread(target=report)
        t.start()
        rc = p.run(100)[0]
        stop.set()
        t.join()
        assert rc == 1 and not errors
        assert np.array_equal(p.get("ROE"), want.get("ROE"))


@pytest.mark.parametrize("threads", [128, 512])
def test_a_member_tuned_after_the_batch_was_made_stays_bitwise_alone(threads):
    from mgpu import case, common_setup, lib
    ps = []
    for t in (threads, threads, 0):            # planes of four and more cells a thread, whose sums show the size
        cd = common_setup.build_common(case.turbine_stage(im=33, jm_row=49, km=33))
        cd.ints["TS_THREADS"] = t
        ps.append(lib.Problem(cd))
    p, q, other = ps
    b = lib.Batch([p, other])
    b.run(2)
    q.run(2)
    chosen = p.autotune()[0]
    for _ in range(60):                        # timing decides: until both are tuned alike
        if q.autotune()[0] == chosen:
            break
    else:
        pytest.skip("the tuner's choices differ")
    b.run(13)
    q.run(13)
    for n in ("RO", "ROE", "ROVX", "DRO"):
        assert np.array_equal(p.get(n), q.get(n)), n
