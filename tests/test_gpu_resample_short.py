"""The FP32 forms' spline (k_resample) on data of a few samples, whose second
derivatives the sum over 16 points to each side meets the ends of more than
once: against the all-FP64 form, with shifts of a good part of a sample.
Tolerance as in test_gpu_resample.py."""
import numpy as np
import pytest

from polgraw_gb300 import workloads
from polgraw_gb300.lib import Context


@pytest.mark.gpu
@pytest.mark.parametrize("N", [2, 3, 4, 5, 8, 9, 10, 17, 40])
def test_short_series(N, gpu_ok):
    s = workloads.segment_settings(3000, dt=8.0, band=100, fftpad=1, nifo=2)
    s.N = N
    arr, keep = workloads.segment_detectors(N, 3, dets=("H1", "L1"), dt=8.0)
    rng = np.random.default_rng(N)
    for pos in keep[1::2]:
        pos.reshape(N, 3)[1:] += rng.uniform(-0.9, 0.9, (N - 1, 3))
    ref, got = (Context(s, arr, 2, precision=q).prelude(1, 3, -2) for q in (1, 0))
    for r, g in zip(ref[:2], got[:2]):
        top = np.abs(r).max(axis=1, keepdims=True)
        assert (top > 0).all() and np.array_equal(r == 0, g == 0)
        assert np.max(np.abs(g - r) / top) <= 1e-5
