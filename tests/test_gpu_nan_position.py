"""A position that is not a number in the ephemeris of a search: the resampled
series is zero at that sample, as outside the data, in the FP32 forms every
other sample is a number, and the searches after it are as before.  (The FP64
form's prelude phase is NaN there, and the transform takes it everywhere.)"""
import math

import numpy as np
import pytest

from polgraw_gb300 import workloads
from polgraw_gb300.lib import Context, Opts, PHASE_NAMES


@pytest.mark.gpu
@pytest.mark.parametrize("N,at", [(2, 1), (10771, 0), (10771, 5000), (10771, 10770)])
def test_nan_position(N, at, gpu_ok):
    s = workloads.segment_settings(max(N, 3000), dt=8.0, band=100, fftpad=1, nifo=2)
    s.N = N
    arr, keep = workloads.segment_detectors(N, 3, dets=("H1", "L1"), dt=8.0)
    ctx = [Context(s, arr, 2, precision=p, phase_mode=PHASE_NAMES[m]) for p, m in
           ((0, "fixed"), (0, "f64"), (0, "ff"), (1, "fixed"))]
    before = [c.prelude(1, 3, -2) for c in ctx]
    good = keep[1].copy()
    keep[1].reshape(N, 3)[at] = [math.nan, 1.0, 2.0]
    for c, b in zip(ctx, before):
        # the detector's constants hold the first position too
        assert c.lib.pa_set_data(c.ctx, arr, 2) == 0
        xa, xb, aa, bb = c.prelude(1, 3, -2)
        assert xa[0, at] == 0 and xb[0, at] == 0
        if c.cfg.precision == 0 and at > 0:
            assert np.isfinite(xa).all() and np.isfinite(xb).all()
        if at > 0:
            assert np.array_equal(xa[1], b[0][1]) and aa == b[2]
        c.fstat(1, 3, -2, 5, Opts(20.0, 0, 0, 1))
    keep[1][:] = good
    for c, b in zip(ctx, before):
        assert c.lib.pa_set_data(c.ctx, arr, 2) == 0
        for x, y in zip(c.prelude(1, 3, -2), b):
            assert np.array_equal(x, y)
