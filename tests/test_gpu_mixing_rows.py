"""The pitchwise sums at a mixing plane are formed eight lanes a row, four
rows a warp, in double-float (the default precision split), or by one thread
a row in the reference's order.  The two differ by the FP32 rounding of at
most 33 terms, 2e-6 of a cell's change: after one step the fields agree to
1e-5 of the density, the energy and the largest momentum.  A row or a term
left out or taken twice is 1e-3 of them.  The sizes leave rows fewer than a
warp's four, rows past a round's last, and terms that do not divide by eight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("im,km", [(9, 7), (10, 6), (16, 9), (18, 34), (34, 12)])
def test_mixing_plane_rows_against_the_reference_order(im, km):
    from mgpu import case, common_setup, lib
    got = {}
    for order in (0, 1):
        cd = common_setup.build_common(case.small_stage(im=im, jm_row=25, km=km))
        cd.ints["REDUCE_ORDER"] = order
        p = lib.Problem(cd)
        p.run(1)
        got[order] = {n: p.get(n) for n in ("RO", "ROE", "ROVX", "RORVT", "ROVR")}
        p.close()
    scale = {n: np.abs(a).max() for n, a in got[1].items()}
    scale["ROVR"] = max(scale["ROVX"], scale["ROVR"])
    for n, a in got[0].items():
        assert np.isfinite(a).all(), n
        assert np.abs(a - got[1][n]).max() <= 1e-5 * scale[n], n
