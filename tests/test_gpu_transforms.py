"""The FP32 passes (csrc/pa_pair.cuh) at every transform length, number of
detectors and filling of the transform by data, against the all-FP64 form of
the same library (whose kernels are others, and pinned to the oracle by
test_gpu_parity.py): the normalised F-statistic of one spindown over all bins.

Tolerance, per bin, against F + 2 (2 is the mean of the normalised F): the
transform's rounding is about 6e-8 sqrt(log2 L) <= 2.7e-7 of the rms of X, the
hardware sine and cosine add at most 3.6e-7 per term; F errs by twice that of X
where X is of its rms, so by about 1e-6 of F + 2, and ten standard deviations
cover 2^19 bins: 1e-5."""
import numpy as np
import pytest

from polgraw_gb300 import workloads
from polgraw_gb300.lib import PHASE_NAMES, Context, Opts

CASES = [
    # N, fftpad, dt, detectors, what of the passes
    (3000, 1, 8.0, ("H1", "L1")),           # 2^12: one-stage rows
    (3001, 2, 8.0, ("H1",)),                # 2^13: rows 8 x 4
    (10771, 1, 8.0, ("H1", "L1")),          # 2^14: rows 8 x 8
    (20001, 1, 8.0, ("H1", "L1", "V1")),    # 2^15: rows 16 x 8
    (40003, 1, 2.0, ("H1", "L1")),          # 2^16: rows 16 x 16, three quarters
    (60001, 1, 2.0, ("H1", "L1", "V1")),    # four quarters
    (43082, 2, 2.0, ("H1", "L1")),          # 2^17: rows 8 x 8 x 8, two quarters
    (86164, 1, 2.0, ("H1",)),               # three quarters
    (98304, 1, 2.0, ("H1", "L1")),          # three quarters, full
    (98305, 1, 2.0, ("H1", "L1", "V1")),    # four quarters by one sample
    (131072, 1, 2.0, ("H1", "L1")),         # no zeros at all
    (86164, 1, 2.0, ("H1", "L1", "V1", "H1")),  # four detectors: no loads ahead
    (40000, 4, 2.0, ("H1", "L1")),          # 2^18: rows 16 x 8 x 8, less than a quarter
    (131073, 1, 2.0, ("H1",)),              # two quarters by one sample: three
    (258492, 2, 2.0, ("H1", "L1")),         # 2^19: rows 16 x 16 x 8
    (270001, 2, 2.0, ("H1", "L1", "V1")),   # 2^20: rows 16 x 16 x 16
]


def setup(N, fftpad, dt, dets):
    s = workloads.segment_settings(N, dt=dt, band=666 if dt < 4 else 100, fftpad=fftpad, nifo=len(dets))
    arr, keep = workloads.segment_detectors(N, 3, dets=dets, dt=dt)
    return s, arr, keep


def compare(s, arr, nifo, phase, ss=7):
    o = Opts(20.0, 0, 0, 1)
    F = [Context(s, arr, nifo, precision=p, phase_mode=PHASE_NAMES[phase]).fstat(1, 3, -2, ss, o) for p in (1, 0)]
    assert np.isfinite(F[0]).all() and abs(F[0].mean() - 2) < 0.2
    return float(np.max(np.abs(F[1] - F[0]) / (F[0] + 2)))


@pytest.mark.gpu
@pytest.mark.parametrize("N,fftpad,dt,dets", CASES)
def test_fixed_phase(N, fftpad, dt, dets, gpu_ok):
    s, arr, keep = setup(N, fftpad, dt, dets)
    assert compare(s, arr, len(dets), "fixed") <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("phase", ["f64", "ff"])
@pytest.mark.parametrize("N,fftpad,dt,dets", [CASES[2], CASES[6], CASES[9], CASES[11]])
def test_other_phases(N, fftpad, dt, dets, phase, gpu_ok):
    s, arr, keep = setup(N, fftpad, dt, dets)
    assert compare(s, arr, len(dets), phase) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("N,fftpad", [(10771, 1), (86164, 1), (43082, 2)])
def test_bins_above_half(N, fftpad, gpu_ok):
    """F wanted beyond half the transform: the last stage forms all its outputs."""
    dt = 8.0 if N < 20000 else 2.0
    s, arr, keep = setup(N, fftpad, dt, ("H1", "L1"))
    s.nmax = 3 * s.nfftf // 4
    o = Opts(20.0, 0, 0, 1)
    F = [Context(s, arr, 2, precision=p).fstat(1, 3, -2, 5, o) for p in (1, 0)]
    assert len(F[0]) == s.nmax - s.nmin
    assert np.max(np.abs(F[1] - F[0]) / (F[0] + 2)) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("nspin", [1, 2, 3, 33, 65])
def test_odd_batches(nspin, gpu_ok):
    """Launches of odd numbers of spindowns (a CTA of pass A takes two): each
    spindown's candidates as from a search of that spindown alone."""
    s, arr, keep = setup(10771, 1, 8.0, ("H1", "L1"))
    from polgraw_gb300.lib import Range
    ctx = Context(s, arr, 2)
    o = Opts(8.0, 0, 0, 1)

    def search(a, b):
        r = Range()
        r.spndr[0], r.spndr[1], r.sst = a, b, a
        return ctx.search_batch([(1, 3, -2)], o, r)

    rec, idx, n = search(0, nspin - 1)
    assert n == nspin and len(rec) > 0
    parts = [search(k, k) for k in range(nspin)]
    assert sum(len(p[0]) for p in parts) == len(rec)
    assert np.array_equal(np.concatenate([p[1]["ii"] for p in parts]), idx["ii"])
    # (the phase terms of a sky point are formed relative to its first
    # spindown: F agrees to the rounding of the angle, not to the bit)
    F = np.concatenate([p[1]["F"] for p in parts])
    assert np.max(np.abs(F - idx["F"]) / idx["F"]) <= 1e-5
