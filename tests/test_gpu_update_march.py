"""TSTEP's update marches along J over tiles of K: whatever its cut (TS_ROWS rows
and TS_PLANES planes of a CTA), the state is bitwise that of the kernel over
pairs of planes, which runs where a plane has at most 512 points, and on larger
planes that of the smallest cut (one plane and three rows of a CTA: no carry
from plane to plane).  The cuts leave a last tile of one row, a last march of
one plane, a tile larger than the plane and one CTA for several planes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("RO", "ROVX", "ROVR", "RORVT", "ROE", "DRO", "DROVX")
CUTS = [(3, 1), (3, 2), (3, 3), (3, 7), (3, 16), (6, 7), (6, 16), (9, 5), (21, 3), (0, 16), (0, 7), (6, 0), (0, 0)]


def _deck(make, size):
    from mgpu import common_setup
    return common_setup.build_common(make(im=size[0], jm_row=size[1], km=size[2]))


def _state(cd, pair, rows, planes):
    from mgpu import lib
    cd.ints["TS_PAIR"], cd.ints["TS_ROWS"], cd.ints["TS_PLANES"] = pair, rows, planes
    p = lib.Problem(cd)
    p.run(6)
    got = {n: p.get(n) for n in FIELDS}
    p.close()
    return got


@pytest.mark.parametrize("size", [(9, 25, 7), (10, 31, 13), (16, 40, 32), (23, 49, 22), (50, 51, 10)])
def test_every_cut_is_bitwise_the_pair_update(size):
    from mgpu import case
    cd = _deck(case.small_stage if size[1] < 40 else case.turbine_stage, size)
    want = _state(cd, 1, 0, 0)
    for rows, planes in CUTS:
        if rows // 3 * size[0] > 288:
            continue
        got = _state(cd, 0, rows, planes)
        for n in FIELDS:
            assert np.array_equal(got[n], want[n]), (rows, planes, n)


@pytest.mark.parametrize("size", [(37, 48, 34), (73, 60, 58)])
def test_every_cut_of_larger_planes_is_bitwise_the_smallest(size):
    from mgpu import case
    cd = _deck(case.turbine_stage, size)
    want = _state(cd, 0, 3, 1)
    for rows, planes in CUTS[1::2]:
        if rows // 3 * size[0] > 288:
            continue
        got = _state(cd, 1, rows, planes)
        for n in FIELDS:
            assert np.array_equal(got[n], want[n]), (rows, planes, n)


def test_cuts_that_no_cta_can_have_are_refused():
    from mgpu import case, common_setup, lib
    for rows, planes in ((4, 0), (-3, 0), (99, 0), (0, 17), (0, -1)):
        cd = common_setup.build_common(case.small_stage())
        cd.ints["TS_ROWS"], cd.ints["TS_PLANES"] = rows, planes
        with pytest.raises(lib.MgpuError) as e:
            lib.Problem(cd)
        assert e.value.code == -1
