"""A batch's members lie on a few chains, one after the other on each; a member
computes bitwise what it computes alone, whichever chain and place it has.
Batches of fewer members than the least number of chains, of one more, and of
many small members, with a member of another size among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,im,jm_row,km", [(2, 9, 25, 7), (5, 65, 121, 49), (9, 33, 97, 33), (11, 9, 25, 7)])
def test_members_on_chains_are_bitwise_alone(n, im, jm_row, km):
    from mgpu import case, common_setup, lib
    make = case.small_stage if jm_row < 40 else case.turbine_stage
    decks = [common_setup.build_common(make(im=im, jm_row=jm_row, km=km))] * (n - 1)
    decks.insert(n // 2, common_setup.build_common(case.small_stage(im=11, jm_row=25, km=9)))
    members = [lib.Problem(cd) for cd in decks]
    members[-1].run(2)                      # at another step than the others: mixed steps
    batch = lib.Batch(members)
    batch.run(7)
    batch.run(5)
    want = {}
    for i, cd in enumerate(decks):
        key = (id(cd), i == n - 1)
        if key not in want:
            p = lib.Problem(cd)
            p.run(14 if i == n - 1 else 12)
            want[key] = {f: p.get(f) for f in ("RO", "ROVX", "ROE")}
            p.close()
        for f, a in want[key].items():
            assert np.array_equal(members[i].get(f), a), (i, f)
