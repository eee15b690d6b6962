"""A batch launched in parts (the first sky point directly, then captured
parts) gives what the sky points give one by one: batch lengths at the edges
of the parts, sky points without work among them, one and two lanes."""
import numpy as np
import pytest

from helpers import case_by_name, key_of, make_host
from test_gpu_schedule import _batch, _ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("lanes,sb", [(1, 0), (2, 2)])
def test_parts_equal_single_points(graphs, lanes, sb, tmp_path, gpu_ok):
    host, _ = make_host(case_by_name("h1l1_gaps_veto"), str(tmp_path))
    ctx = _ctx(host)
    base = list(host.sky_points())
    OUTSIDE = (base[0][0], 100000, 100000)
    F = ctx.fstat(*base[0], 0, host.opts())
    one = {p: _batch(ctx, host, [p]) for p in base + [OUTSIDE]}
    assert len(one[OUTSIDE][0]) == 0
    ctx.set_graphs(graphs)
    if sb:
        ctx.set_schedule(sb, ctx.schedule()[1])
    ctx.set_lanes(lanes)
    for n, gaps in [(1, ()), (1, (0,)), (2, (0,)), (3, (1, 2)), (4, ()), (8, (3, 4, 5, 6)), (9, (0, 1, 2, 8))]:
        pts = [OUTSIDE if i in gaps else base[i % len(base)] for i in range(n)]
        rec, idx, fnum = _batch(ctx, host, pts)
        want = [one[p] for p in pts]
        assert np.array_equal(rec, np.concatenate([w[0] for w in want]))
        assert len(key_of(idx)) == len(rec) and fnum == sum(w[2] for w in want)
    assert np.array_equal(F, ctx.fstat(*base[0], 0, host.opts()))   # after captured work on the same slots
