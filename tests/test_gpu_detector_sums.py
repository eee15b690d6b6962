"""aa and bb of the FP32 forms (k_resample's extra block: four warps share the
detectors and their partial sums) for one to eight detectors and for fewer
partial sums than lanes, against the all-FP64 form.  Tolerance: the antenna
factors' FP32 roundings, about ten of 6e-8 and twice that in the squares, summed
in FP64: 2e-6."""
import numpy as np
import pytest

from polgraw_gb300 import workloads
from polgraw_gb300.lib import Context


@pytest.mark.gpu
@pytest.mark.parametrize("N", [100, 4096, 43082])
@pytest.mark.parametrize("nifo", [1, 2, 3, 4, 5, 8])
def test_sums(N, nifo, gpu_ok):
    dets = ("H1", "L1", "V1", "L1", "H1", "V1", "V1", "L1")[:nifo]
    dt = 8.0 if N < 30000 else 2.0
    s = workloads.segment_settings(max(N, 3000), dt=dt, band=100 if dt > 4 else 666, fftpad=1, nifo=nifo)
    s.N = N
    arr, keep = workloads.segment_detectors(N, 3, dets=dets, dt=dt)
    for k in range(nifo):
        arr[k].sig2 *= 1 + k  # a detector's own weight
    ref, got = (Context(s, arr, nifo, precision=q).prelude(1, 3, -2)[2:] for q in (1, 0))
    np.testing.assert_allclose(got, ref, rtol=2e-6)
