"""TSTEP's damping and corner gather runs over pairs of J planes where a plane
has at most 512 points, and otherwise marches along J over tiles of K cut by
the grid's size (TS_PAIR = 0: always).  Both form every value by the same
operations, so the state is bitwise the same.  The sizes leave remainders in
the K tiles (3 rows a thread), in the planes a CTA marches (1 to 16), in the
last warp of a tile and in the last pair of planes.  A batch of one steps the
larger sizes, where both march, as the problem alone does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("RO", "ROVX", "ROVR", "RORVT", "ROE", "DRO", "DROVX")


@pytest.mark.parametrize("im,jm_row,km", [(9, 25, 7), (10, 31, 13), (16, 40, 32), (23, 49, 22), (37, 48, 13), (50, 51, 10)])
def test_march_is_bitwise_the_pair_update(im, jm_row, km):
    from mgpu import case, common_setup, lib
    make = case.small_stage if jm_row < 40 else case.turbine_stage
    cd = common_setup.build_common(make(im=im, jm_row=jm_row, km=km))
    got = []
    for pair in (0, 1):
        cd.ints["TS_PAIR"] = pair
        p = lib.Problem(cd)
        p.run(6)
        got.append({n: p.get(n) for n in FIELDS})
        p.close()
    for n in FIELDS:
        assert np.array_equal(got[0][n], got[1][n]), n


@pytest.mark.parametrize("im,jm_row,km", [(23, 49, 23), (37, 66, 34), (33, 61, 50), (65, 49, 47), (73, 60, 58), (96, 48, 9)])
def test_batch_of_one_is_bitwise_the_problem_alone(im, jm_row, km):
    from mgpu import case, common_setup, lib
    cd = common_setup.build_common(case.turbine_stage(im=im, jm_row=jm_row, km=km))
    alone, member = lib.Problem(cd), lib.Problem(cd)
    alone.run(6)
    lib.Batch([member]).run(6)
    for n in FIELDS:
        assert np.array_equal(alone.get(n), member.get(n)), n
