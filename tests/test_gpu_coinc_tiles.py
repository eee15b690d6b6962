"""The coincidence kernels at the edges of their tiles and number ranges,
against the CPU oracle: record counts around the 2048- and 4096-record tiles,
runs of duplicates across a tile's end, more coincidences than one block scans,
cells exactly on a rounding boundary, and frequencies, spindowns and SNRs that
are zero, subnormal, infinite, NaN or exactly on a cut.  Every output is a
whole number or a value formed in the oracle's order: all must be equal."""
import math

import numpy as np
import pytest

from test_gpu_coinc import _device, _same

pytestmark = pytest.mark.gpu
N, REFR = 86164, 2


def _cfg(v=None, **kw):
    from polgraw_gb300 import lib as L
    if v is None:
        c, s = math.cos(0.3), math.sin(0.3)
        v = np.array([[c / 8, -s / 16, 0, 0], [s / 8, c / 16, 0, 0], [0, 0, 1e-5, 2e-6], [0, 0, -2e-6, 1e-5]])
    a = dict(N=N, oms=2000.0, vedva_m=v, shift=0, scale=1111, refr=REFR, mincoin=3)
    a.update(kw)
    return L.coinc_cfg(**a)


def _check(cfg, recs):
    import pyoracle
    order = sorted(recs)
    dev = _device(cfg, order, recs)
    _same(dev, pyoracle.coinc(cfg, order, [recs[f] for f in order]))
    return dev


@pytest.mark.parametrize("n", [1, 31, 255, 2047, 2048, 2049, 4095, 4096, 4097, 8300])
def test_record_counts(n, gpu_ok):
    from polgraw_gb300 import synth
    recs = synth.coinc_triggers([1, 2, 3, 4], n, N=N, refr=REFR, seed=n, lines=3, sky=8, signals=40)
    assert len(_check(_cfg(), recs).cells)


def test_runs_across_tiles_and_many_groups(gpu_ok):
    rng = np.random.default_rng(1)
    base = np.column_stack([rng.uniform(0.5, 2.5, 40000), rng.choice([0.0, 1e-9, -3e-10], 40000),
                            rng.uniform(-1.2, 1.2, 40000), rng.uniform(0, 6.2, 40000), rng.uniform(6.1, 9, 40000)])
    recs = {f: base + [0, 0, 0, 0, 0.01 * f] for f in (1, 2, 3)}
    for f in recs:   # the frame's shift taken out: the same cells in all frames
        recs[f][:, 0] -= 2 * recs[f][:, 1] * N * (REFR - f)
        recs[f] = np.concatenate([recs[f], np.repeat(recs[f][:3], 1700, axis=0)])
    dev = _check(_cfg(), recs)
    assert dev.summary.ncoin > 32768


def test_cells_on_rounding_boundaries(gpu_ok):
    v = np.diag([2.0 ** -6, 2.0 ** -8, 2.0 ** -20, 2.0 ** -20])
    k = np.arange(600, 5000)
    recs = {f: np.column_stack([k / 2048.0, np.where(k % 3, 0.0, (k % 7) * 2.0 ** -30), 0.0 * k, 0.0 * k, 7.0 + 0 * k])
            for f in (1, 2, 3)}
    dev = _check(_cfg(v, N=1 << 15), recs)
    assert dev.summary.fp64_cells > 0


@pytest.mark.parametrize("large_n", [False, True])
def test_number_ranges(large_n, gpu_ok):
    inf, nan, lo = math.inf, math.nan, math.pi / 2 - 0.4 * math.pi
    hi, up, dn = math.pi / 2 + 0.4 * math.pi, lambda x: np.nextafter(x, 9), lambda x: np.nextafter(x, -9)
    f = [lo, up(lo), dn(lo), hi, dn(hi), up(hi), 0.0, -0.0, inf, -inf, nan, -nan, math.pi, dn(math.pi), 1.5, 1e-310]
    s = [0.0, -0.0, 1e-310, -5e-324, 1e-30, 2.0 ** -74, 2.0 ** -75, 1e-9, -1e-9, inf, -inf, nan]   # (cells beyond an int are undefined in C)
    q = [6.0, up(6.0), dn(6.0), inf, -inf, nan, 7.0, 0.0]
    ang = [0.0, -0.0, 1e-320, 1.0, -1.3, 8.0, up(8.0), 30.0, -100.0]
    rows = [[a, b, 0.3, 0.4, c] for a in f for b in s for c in q]
    rows += [[1.5, 1e-10, a, b, 7.0] for a in ang for b in ang]
    r = np.array(rows)
    n = 1 << 24 if large_n else N
    _check(_cfg(N=n, narrowdown=0.4, mincoin=2), {1: r, 2: r[::-1].copy(), 3: r[5:]})
