"""The adjoint takes every plane whose three copies fit 200 KB of shared memory
(3 IM KM <= 51200 floats), the smoothing weights beside them, and no larger."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("im,km,taken", [(128, 133, True), (110, 154, True), (133, 129, False)])
def test_largest_planes(im, km, taken):
    from mgpu import case, common_setup, lib
    cd = common_setup.build_common(case.small_nozzle(im=im, km=km))
    cd.ints["FROZEN"] = 1
    p = lib.Problem(cd)
    p.run(2)
    if not taken:
        with pytest.raises(lib.MgpuError) as e:
            p.adjoint_prepare()
        assert e.value.code == -4
        return
    p.adjoint_prepare()
    p.adjoint_objective("mass_flow_in")
    p.adjoint_iterate(2)
    g = p.adjoint_get("RO")
    assert np.isfinite(g).all() and np.abs(g).max() > 0.0
