"""Searches with an output capacity of zero records: the call learns the number
of records from the library and comes back with room for them."""
import numpy as np
import pytest

from polgraw_gb300 import workloads
from polgraw_gb300.lib import Context, Opts, Range, Segments


@pytest.mark.gpu
def test_no_capacity(gpu_ok):
    s = workloads.segment_settings(10771, dt=8.0, band=100, fftpad=1, nifo=1)
    arr, keep = workloads.segment_detectors(10771, 3, dets=("H1",), dt=8.0)
    o, r = Opts(8.0, 0, 0, 1), Range()
    r.spndr[:], r.nr[:], r.mr[:], r.pmr[:] = (0, 3), (-9, 9), (-9, 9), (1, 1)
    want = Context(s, arr, 1).job_core(1, 3, -2, o, r)
    assert len(want[0]) > 0
    c = Context(s, arr, 1)
    calls = (lambda: Context(s, arr, 1).job_core(1, 3, -2, o, r, cap=0),
             lambda: Context(s, arr, 1).search_batch([(1, 3, -2)], o, r, cap=0),
             lambda: Segments([c]).search([[(1, 3, -2)]], [o], [r], cap=0)[0])
    for call in calls:
        rec, idx, fnum = call()
        assert fnum == want[2] and np.array_equal(rec, want[0]) and np.array_equal(idx, want[1])
