"""The resampled series of the FP32 forms (k_prelude_mod, the resampling
transforms on pairs, k_resample) against the all-FP64 form of the same library:
lengths at the edges of a block's 112 samples and 128 threads, one to three
detectors, and shifts that are smooth, jump between neighbouring samples (a
block then takes several turns), or leave the series at either end (zeros).

Tolerance, against the largest value of an array: two FP32 transforms err by
6e-8 sqrt(2 log2 L) = 3.5e-7 of the rms each, the phase's sine and cosine and the
antenna factors by 1e-6 of a value; the largest of 1e5 errors is below five
standard deviations of that, and the largest value above three rms: 1e-5."""
import numpy as np
import pytest

from polgraw_gb300 import workloads
from polgraw_gb300.lib import Context


@pytest.mark.gpu
@pytest.mark.parametrize("shifts", ["smooth", "jumps", "outside"])
@pytest.mark.parametrize("N,dets", [(2688, ("H1",)), (2689, ("H1", "L1")), (8191, ("H1", "L1", "V1")),
                                    (10771, ("H1", "L1")), (43008, ("H1",))])
def test_resampled_series(N, dets, shifts, gpu_ok):
    dt = 8.0 if N < 30000 else 2.0
    s = workloads.segment_settings(N, dt=dt, band=100 if dt > 4 else 666, fftpad=1, nifo=len(dets))
    arr, keep = workloads.segment_detectors(N, 3, dets=dets, dt=dt)
    rng = np.random.default_rng(N)
    for pos in keep[1::2]:
        p = pos.reshape(N, 3)
        if shifts == "jumps":
            p[1:] += rng.uniform(-60, 60, (N - 1, 3)) * (rng.random((N - 1, 1)) < 0.2)
        elif shifts == "outside":
            p[N // 3:N // 2] += [5.0 * N, -4.0 * N, 6.0 * N]
            p[-40:] -= [60.0, 60.0, 60.0]
    ref, got = (Context(s, arr, len(dets), precision=q).prelude(1, 3, -2) for q in (1, 0))
    for r, g in zip(ref[:2], got[:2]):
        top = np.abs(r).max(axis=1, keepdims=True)
        assert (top > 0).all() and (shifts != "outside" or (r == 0).any())
        assert np.array_equal(r == 0, g == 0)
        assert np.max(np.abs(g - r) / top) <= 1e-5
    np.testing.assert_allclose(got[2:], ref[2:], rtol=1e-6)   # aa, bb: FP32 squares, FP64 sums
