"""Reports of one handle from several threads at a time are each the report
asked for: the buffer that they are formed in belongs to one at a time."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_stage_tables_of_several_threads():
    from mgpu import case, common_setup, lib
    cd = common_setup.build_common(case.compressor_4stage(im=9, jm_row=25, km=7))
    p = lib.Problem(cd)
    p.run(20)

    def table(s):
        r = p.integrals() if s == 0 else p.stage(s)
        return [getattr(r, f) for f, _ in r._fields_]

    stages = range(cd.ints["NSTAGES"] + 2)
    want = {s: table(s) for s in stages}
    wrong = []

    def report(s):
        for _ in range(400):
            if table(s) != want[s]:
                wrong.append(s)

    ts = [threading.Thread(target=report, args=(s,)) for s in stages]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong
