"""Two coincidence handles on one device, run from two host threads at once:
their kernels are in flight together, each with its own frame table.  The
frames, their number and their lengths differ, so that a table of the other
handle would give other cells and members.  Every output equals that of the
same handle's run alone."""
import threading

import pytest

from test_gpu_coinc import _same
from test_gpu_coinc_tiles import N, REFR, _cfg

RUNS = 30


@pytest.mark.gpu
def test_two_handles_at_once(gpu_ok):
    from polgraw_gb300 import lib as L
    from polgraw_gb300 import synth
    handles, alone = [], []
    for frames, per_frame, seed in ((range(1, 25), 9000, 5), (range(3, 6), 70001, 6)):
        fr = list(frames)
        recs = synth.coinc_triggers(fr, per_frame, N=N, refr=REFR, seed=seed, lines=3, sky=8, signals=200)
        h = L.Coinc(_cfg())
        for f in fr:
            h.add_frame(f, recs[f])
        handles.append(h)
        alone.append(h.run(cells=True))
    assert all(a.summary.ncoin > 0 for a in alone)
    together = [[], []]
    start = threading.Barrier(2)

    def runs(k):
        start.wait()
        for _ in range(RUNS):
            together[k].append(handles[k].run(cells=True))

    threads = [threading.Thread(target=runs, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert len(together[k]) == RUNS
        for r in together[k]:
            _same(r, alone[k])
