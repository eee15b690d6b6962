"""Followup data whose ephemeris has one position that is not a number, in a gap
(the data there are zero), and positions that leave a chunk's parabola far behind
before it, smooth ones after: the mixed form takes the FP64 phase of every
sample, the gap adds nothing, and F is that of the same data with a number
there.  Tolerance as in test_gpu_followup_sums.py."""
import math

import numpy as np
import pytest

from polgraw_gb300.lib import Followup, make_detectors
from test_gpu_followup_sums import points, setup

N = 5000


@pytest.mark.gpu
@pytest.mark.parametrize("at", [1500, 2048, 2560, 4999])  # inside a chunk; its first, middle and last sample
def test_nan_position_in_a_gap(at, gpu_ok):
    s, dets, keep = setup(N, 8.0, 2)
    x, pos = keep[0], keep[1].reshape(N, 3)
    x[at] = 0.0
    pos[:1000] += np.random.default_rng(5).normal(0.0, 0.05, (1000, 3))
    p = points(9, N)
    ref = Followup(s, dets, 2, precision=1).fstatnet(p)
    pos[at, 1] = math.nan
    got = Followup(s, dets, 2, precision=0).fstatnet(p)
    assert np.isfinite(ref[:, 5]).all()
    assert np.max(np.abs(got[:, 5] - ref[:, 5]) / (2 - ref[:, 5])) <= 1e-5
