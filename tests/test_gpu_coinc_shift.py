"""Cell shifts of any size (a digit each from the program, any int through the
C-ABI): the FP32 sum of a cell's fractions holds the half shift too, whose
rounding is part of the margin.  Against the CPU oracle; all outputs equal."""
import math

import numpy as np
import pytest

from test_gpu_coinc_tiles import N, _cfg, _check


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [1, 9, -2001, 1000001])
def test_shifts(shift, gpu_ok):
    c, s = math.cos(0.3), math.sin(0.3)
    cfg = _cfg(np.array([[c / 8, -s / 16, 0, 0], [s / 8, c / 16, 0, 0], [0, 0, 1e-7, 2e-8], [0, 0, -2e-8, 1e-7]]))
    for k in range(4):
        cfg.shift[k] = shift + 2 * k
    rng = np.random.default_rng(abs(shift))
    n = 60000
    base = np.column_stack([rng.uniform(0.5, 2.5, n), rng.uniform(-1e-9, 1e-9, n), rng.uniform(-1.2, 1.2, n),
                            rng.uniform(0, 6.2, n), rng.uniform(6.1, 9, n)])
    dev = _check(cfg, {f: base - [0, 0, 0, 0, 0.01 * f] for f in (1, 2, 3)})
    assert dev.summary.inband > n and N < 1 << 24
