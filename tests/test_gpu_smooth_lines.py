"""The smoothing kernel takes two lines of a plane at a time, half the plane
apart, in segments of four points.  The sizes leave an odd last line in I and
in K, a last segment of one to four points, and lines of a single segment.
One step of the small stage against the oracle: the operations are the
reference's, so the fields agree to the bar of one step, 1e-5, of the density,
the energy and the largest momentum (a wrong weight or neighbour is 1e-3)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("im,km", [(9, 6), (10, 9), (11, 10), (12, 7), (15, 13), (18, 33)])
def test_one_step_matches_the_oracle(im, km):
    from mgpu import case, common_setup, lib
    import oracle as O
    cd = common_setup.build_common(case.small_stage(im=im, jm_row=25, km=km))
    gpu, ref = lib.Problem(cd), O.Oracle(cd)
    ref.setup_calls()
    gpu.step()
    ref.step()
    want = {n: np.asarray(ref.get(n, double=False)).ravel() for n in ("RO", "ROE", "ROVX", "RORVT", "ROVR")}
    scale = {n: np.abs(a).max() for n, a in want.items()}
    scale["ROVR"] = max(scale["ROVR"], scale["ROVX"])
    for n, a in want.items():
        assert np.abs(gpu.get(n).ravel() - a).max() <= 1e-5 * scale[n], n
    gpu.close()
