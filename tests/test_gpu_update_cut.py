"""TSTEP's damping and corner gather marches along J over tiles of K, cut by
the grid's size; a member of a batch takes the kernel over pairs of J planes
instead.  Both form every value by the same operations: a problem alone and
the same problem as a batch of one have bitwise the same state.  The sizes
leave remainders in the K tiles (3 rows a thread), in the planes a CTA marches
(1 to 16), in the last warp of a tile and in the last pair of planes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("im,jm_row,km", [(23, 49, 23), (37, 66, 34), (33, 61, 50), (65, 49, 47), (73, 60, 58), (96, 48, 9)])
def test_batch_of_one_is_bitwise_the_problem_alone(im, jm_row, km):
    from mgpu import case, common_setup, lib
    cd = common_setup.build_common(case.turbine_stage(im=im, jm_row=jm_row, km=km))
    alone, member = lib.Problem(cd), lib.Problem(cd)
    alone.run(6)
    lib.Batch([member]).run(6)
    for n in ("RO", "ROVX", "ROVR", "RORVT", "ROE", "DRO", "DROVX"):
        assert np.array_equal(alone.get(n), member.get(n)), n
