"""The followup's gradient in the mixed form (csrc/pa_followup_f32.cuh), in each
form of its phase -- fast (FP32 rests), rough (integer rests), slow (FP64 a
sample) -- and where they meet, against the FP64 form; and the points of a list
(the ascent's) against the same points alone.

Tolerance of the gradient, in units of the peak's widths, against the largest
component: a sample's term errs by 5e-7 (the angle's rounding 9e-8 twice, sine
and cosine 5e-8, seeds and products six of 6e-8), the FP32 sums of a lane by
1e-6, so a component by 1.5e-6 of its own scale over noise, sqrt(sum g^2 h^2);
the largest of the (about two independent) components is below a thirtieth of
that scale once in a thousand points: 1e-4 allows twice that.  F: 1e-5 of F + 2
as in test_gpu_followup_sums.py."""
import math

import numpy as np
import pytest

from polgraw_gb300 import workloads
from polgraw_gb300.lib import Followup
from test_gpu_followup_sums import points, setup

CASES = [
    # N, dt, detectors, frequency (0: as the data's band), points, path
    (700, 2.0, 1, 0, 3, "smooth"),
    (1024, 2.0, 2, 0, 17, "smooth"),        # fast
    (1024, 8.0, 2, 0, 17, "smooth"),        # fast, adjoint rough (short data)
    (1025, 8.0, 2, 0, 16, "smooth"),        # a chunk of one sample
    (10771, 8.0, 3, 0, 33, "smooth"),       # fast
    (10771, 8.0, 2, 100, 33, "smooth"),     # rough
    (10771, 8.0, 1, 1500, 31, "smooth"),    # rough, 0.04 turns
    (10771, 8.0, 2, 0, 9, "rough"),         # rough, a turn
    (10771, 8.0, 2, 0, 9, "jump"),          # one chunk slow
    (5000, 8.0, 2, 0, 5, "wild"),           # slow
    (43082, 4.0, 3, 1000, 7, "smooth"),     # rough
    (86164, 2.0, 3, 0, 5, "smooth"),        # fast
]


def make(N, dt, nifo, freq, path):
    s, dets, keep = setup(N, dt, nifo)
    if freq:
        s.oms = 2 * math.pi * freq * dt
    rng = np.random.default_rng(11)
    for pos in keep[1::2]:
        p = pos.reshape(N, 3)
        if path == "rough":
            p += 1e-3 * rng.standard_normal((N, 3))
        elif path == "wild":
            p += 2.0 * rng.standard_normal((N, 3))
        elif path == "jump":
            p[N // 3:] += [40.0, -30.0, 20.0]
    return s, dets, keep


@pytest.mark.gpu
@pytest.mark.parametrize("N,dt,nifo,freq,n,path", CASES)
def test_gradient_against_fp64(N, dt, nifo, freq, n, path, gpu_ok):
    s, dets, keep = make(N, dt, nifo, freq, path)
    p = points(n, N)
    seed = np.linspace(0.5, 2.0, n)
    (Fa, ga), (Fb, gb) = (Followup(s, dets, nifo, precision=q).fstatnet_grad(p, seed) for q in (0, 1))
    assert np.max(np.abs(Fa - Fb) / (Fb + 2)) <= 1e-5
    w = np.array([workloads.peak_widths(s, dets, nifo, q[2], q[3]) for q in p])
    d, m = np.abs((ga - gb) * w), np.max(np.abs(gb * w), axis=1)
    assert np.all(d <= 1e-4 * m[:, None])


@pytest.mark.gpu
def test_forms_side_by_side(gpu_ok):
    """Fast, rough and slow points in one warp give the bits that each gives alone."""
    s, dets, keep = make(10771, 8.0, 2, 0, "smooth")
    p = points(19, 10771)
    p[1::3, 0] = 1e4    # rough
    p[2::3, 0] = 1e9    # slow
    fu = Followup(s, dets, 2)
    out, (F, g) = fu.fstatnet(p), fu.fstatnet_grad(p)
    for k, q in enumerate(p):
        assert np.array_equal(fu.fstatnet(q)[0], out[k], equal_nan=True)
        Fk, gk = fu.fstatnet_grad(q)
        assert Fk[0] == F[k] and np.array_equal(gk[0], g[k])


@pytest.mark.gpu
@pytest.mark.parametrize("freq,path", [(0, "smooth"), (200, "smooth"), (0, "jump")])
def test_ascent_of_a_list(freq, path, gpu_ok):
    """Points that leave an ascent at different steps (the others go on as a
    list) end where each of them ends alone, and with the F of that place."""
    N = 10771
    s, dets, keep = make(N, 8.0, 2, freq, path)
    p = points(21, N)
    scale = np.mean([workloads.peak_widths(s, dets, 2, q[2], q[3]) for q in p], axis=0)
    fu = Followup(s, dets, 2)
    end, out, its = fu.ascent(p, scale, max_iter=25)
    assert len(set(its)) > 1 and np.all(-out[:, 5] >= -fu.fstatnet(p)[:, 5])
    assert np.array_equal(fu.fstatnet(end), out, equal_nan=True)
    for k in range(len(p)):
        e, o, i = fu.ascent(p[k], scale, max_iter=25)
        assert np.array_equal(e[0], end[k]) and np.array_equal(o[0], out[k], equal_nan=True) and i[0] == its[k]
