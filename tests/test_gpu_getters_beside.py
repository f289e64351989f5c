"""A progress reader on another thread (mgpu_get_real, mgpu_get_int) leaves the
march as it is: which steps run LOSS and the tail does not depend on it."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["DAMP", "NSTEP"])
def test_a_reader_beside_a_march_does_not_change_it(name):
    from mgpu import case, common_setup, lib
    cd = common_setup.build_common(case.small_stage())
    cd.ints["NLOS"], cd.ints["NSTEPS_MAX"], cd.reals["CONLIM"] = 3, 10 ** 6, 1e-9
    want, p = lib.Problem(cd), lib.Problem(cd)
    want.run(1350)
    stop, errors = threading.Event(), []

    def read():
        L, v = lib.load(), ctypes.c_int32()
        try:
            while not stop.is_set():
                if name == "NSTEP":
                    assert L.mgpu_get_int(p.h, b"NSTEP", ctypes.byref(v)) == 0
                else:
                    p.get_real(name)
        except Exception as e:                 # noqa: BLE001
            errors.append(e)

    p.step()
    t = threading.Thread(target=read)
    t.start()
    for n in (99, 250, 250):
        p.run(n)
    for _ in range(30):                        # queues the steps up to each tail without waiting in between
        p.bench_steps(25, flush_l2=False)
    stop.set()
    t.join()
    assert not errors
    for f in ("RO", "ROE", "XFORCE", "STEP"):
        assert np.array_equal(p.get(f), want.get(f)), f
