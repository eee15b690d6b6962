"""The mixed form of the followup's sums (csrc/pa_followup_f32.cuh) against the
FP64 form where its chunks, groups of points and its choice of the phase change:
data shorter than a chunk and one sample past one, one point to a group of
points and one more, a detector path that is not smooth (the FP64 phase per
sample), data too short for the adjoint's moments.

Tolerances.  F: the sine and cosine err by 5e-8, the angle's FP32 rounding by
9e-8 and FP32 sums of a chunk by a few 1e-7 of their terms, so X by about 1e-6
of its rms and F by 2e-6 of F + 2; 1e-5 allows five times that.  Gradient (where
its sums over samples are in FP64; FP32 sums that cancel have no such bound away
from a signal, and test_gpu_followup.py holds them at one): 2e-3 of the largest
component in units of the widths, as the mixed gradient is held to elsewhere."""
import math

import numpy as np
import pytest

from polgraw_gb300 import synth, workloads
from polgraw_gb300.lib import Followup, Settings, make_detectors

DETS = ("H1", "L1", "V1")


def setup(N, dt, nifo, jitter=0.0, seed=3):
    rng = np.random.default_rng(seed)
    xs, ps, s2, sph, cph, am = [], [], [], [], [], []
    for d in DETS[:nifo]:
        pos, phir, _ = synth.detssb(d, N, dt)
        xs.append(rng.standard_normal(N))
        ps.append(pos + jitter * rng.standard_normal(3 * N))
        s2.append(1.0)
        sph.append(math.sin(phir))
        cph.append(math.cos(phir))
        am.append(synth.rogcvir(synth.SITES[d]["ephi"], synth.SITES[d]["egam"]))
    s = Settings()
    s.N = N
    s.oms = 2 * math.pi * synth.fpo_default(666 if dt < 4 else 100, dt) * dt
    s.omr = synth.C_OMEGA_R * dt
    return (s,) + make_detectors(xs, ps, s2, sph, cph, am)


def points(n, N, seed=4):
    rng = np.random.default_rng(seed)
    return np.stack([rng.uniform(0.2, 2.9, n), rng.uniform(-2e-8, 2e-8, n) * (8e4 / N), rng.uniform(-1.2, 1.2, n),
                     rng.uniform(0, 6.2, n)], axis=1)


CASES = [
    # N, dt, detectors, points, jitter of the path
    (1, 2.0, 1, 2, 0.0),
    (2, 2.0, 2, 1, 0.0),
    (700, 2.0, 1, 3, 0.0),         # the adjoint's FP64 sums
    (1024, 2.0, 2, 31, 0.0),
    (1025, 2.0, 2, 32, 0.0),       # a chunk of one sample
    (10771, 8.0, 3, 33, 0.0),
    (43082, 2.0, 2, 65, 0.0),
    (86164, 2.0, 3, 5, 0.0),
    (10771, 8.0, 2, 9, 1e-3),      # FP64 phase per sample
]


@pytest.mark.gpu
@pytest.mark.parametrize("N,dt,nifo,n,jitter", CASES)
def test_mixed_against_fp64(N, dt, nifo, n, jitter, gpu_ok):
    s, dets, keep = setup(N, dt, nifo, jitter)
    p = points(n, N)
    mixed, exact = (Followup(s, dets, nifo, precision=q) for q in (0, 1))
    a, b = mixed.fstatnet(p), exact.fstatnet(p)
    F = -b[:, 5]
    if N >= 700:  # below, A and B of a detector can vanish
        assert np.max(np.abs(a[:, 5] - b[:, 5]) / (F + 2)) <= 1e-5
        assert np.array_equal(a[:, 6:10], p)
        seed = np.linspace(0.5, 2.0, n)
        Fa, ga = mixed.fstatnet_grad(p, seed)
        Fb, gb = exact.fstatnet_grad(p, seed)
        assert np.array_equal(Fa, -a[:, 5])
        w = np.array([workloads.peak_widths(s, dets, nifo, q[2], q[3]) for q in p])
        d, m = np.abs((ga - gb) * w), np.max(np.abs(gb * w), axis=1)
        assert np.isfinite(ga).all()
        if jitter:
            assert np.all(d <= 2e-3 * m[:, None])


@pytest.mark.gpu
def test_mixed_points_do_not_depend_on_the_group(gpu_ok):
    """A point beside one that takes the other phase gives the same bits."""
    s, dets, keep = setup(10771, 8.0, 2)
    p = points(7, 10771)
    far = p.copy()
    far[::2, 0] = 1e5  # beyond the fast phase's range
    fu = Followup(s, dets, 2)
    alone = np.concatenate([fu.fstatnet(q) for q in far])
    assert np.array_equal(fu.fstatnet(far), alone, equal_nan=True)
    assert np.array_equal(fu.fstatnet(p)[1::2], alone[1::2], equal_nan=True)
    F, g = fu.fstatnet_grad(far)
    each = [fu.fstatnet_grad(q) for q in far]
    assert np.array_equal(g, np.concatenate([e[1] for e in each]))
