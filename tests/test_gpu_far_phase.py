"""FP64-phase form (PA_PHASE_F64): the spindown phase as turns in the low word
of an fma, and products beyond its 2^19 turns, against the all-FP64 form.
Spindown steps that keep all products below 2^19 turns, cross it within the
data, and pass it almost everywhere; tolerance as in test_gpu_transforms.py
(1e-5 of F + 2): the FP64 phases of both err by 1e7 rad x 2e-16."""
import math

import pytest

from test_gpu_transforms import compare, setup


@pytest.mark.gpu
@pytest.mark.parametrize("N,fftpad,dt,dets", [(10771, 1, 8.0, ("H1",)), (20001, 1, 8.0, ("H1", "L1", "V1")),
                                              (43082, 2, 2.0, ("H1", "L1")), (86164, 1, 2.0, ("H1", "L1", "V1", "H1"))])
@pytest.mark.parametrize("turns", [0.9, 1.7, -40.0])
def test_far_products(N, fftpad, dt, dets, turns, gpu_ok):
    s, arr, keep = setup(N, fftpad, dt, dets)
    s.M[5] = turns * 2 ** 19 * 2 * math.pi / (7 * float(N) ** 2)
    # (four detectors over 2^14 fill no second block of bins: the mean is not 2)
    assert compare(s, arr, len(dets), "f64", ss=7) <= 1e-5
