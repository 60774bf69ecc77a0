"""The grid searches where their rules change: every number of lanes a query,
sets just above the line between all pairs and the grid (and the all-pairs scan
behind a grid that was built and not used), and that the line lies where the grid
does not cost more than the scan it replaces."""
import ctypes as C
import statistics

import numpy as np
import pytest

from test_gpu_far_points import curve, with_far
from test_gpu_grid_search import KINDS, clouds, exhaustive

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("eps", [0.0, 1e-4, 0.02])
def test_radius_above_the_line(gpu, kind, eps):
    from hiten_gb300.connections import GpuSectionMatcher
    rng = np.random.default_rng(len(kind))
    q, r = clouds(kind, 12001, rng), clouds(kind, 11403, rng)
    q[:50] = r[100:150]
    c = float(np.nanmax(np.abs(np.where(np.isfinite(np.r_[q, r]), np.r_[q, r], 0.0))))
    cnt, idx, d2 = GpuSectionMatcher().radius_best(q, r, eps, c)
    ec, ei, ed = exhaustive(q, r, eps, False)
    assert np.array_equal(cnt, ec) and np.array_equal(idx, ei) and np.array_equal(d2, ed)


@pytest.mark.parametrize("n", [40001, 50000, 90001, 180001])
@pytest.mark.parametrize("kind", ["curve", "hundred", "lattice"])
def test_lanes_a_query(gpu, n, kind):
    """Sampled queries (the far points among them) against all points."""
    from hiten_gb300.connections import GpuSectionMatcher
    rng = np.random.default_rng(n)
    p = with_far(curve(n, rng), kind, rng)
    r = with_far(curve(4201, rng), kind, rng)
    c = float(np.abs(np.r_[p, r]).max())
    at = np.unique(np.r_[0, n - 1, rng.integers(0, n, 150), np.argsort(np.abs(p).max(1))[-50:]])
    m = GpuSectionMatcher()
    near = m.nearest(p, c)
    dx, dy = p[at, :1] - p[None, :, 0], p[at, 1:] - p[None, :, 1]
    d2 = dx * dx + dy * dy
    d2[np.arange(len(at)), at] = np.inf
    assert np.array_equal(near[at], np.argmin(d2, axis=1))
    cnt, idx, best = m.radius_best(p, r, 1e-3, c)
    ec, ei, ed = exhaustive(p[at], r, 1e-3, False)
    assert np.array_equal(cnt[at], ec) and np.array_equal(idx[at], ei) and np.array_equal(best[at], ed)


def device_ms(n, nearest):
    import torch
    from hiten_gb300 import _lib
    L = _lib.load()
    rng = np.random.default_rng(5)
    p, q = (with_far(curve(n, rng), "hundred", rng) for _ in range(2))
    d = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    x, y, qx, qy = d(p[:, 0]), d(p[:, 1]), d(q[:, 0]), d(q[:, 1])
    i32 = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2)]
    bd = torch.empty(n, dtype=torch.float64, device="cuda")
    ws = torch.empty(int(L.hg_points_workspace_bytes(n)), dtype=torch.uint8, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    ms = []
    for k in range(12):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(400000)
        a.record()
        if nearest:
            rc = L.hg_nearest_neighbor(n, ptr(x), ptr(y), 1.0, ptr(i32[0]), ptr(ws), ws.numel(), st)
        else:
            rc = L.hg_radius_best(n, ptr(qx), ptr(qy), n, ptr(x), ptr(y), 1e-4, 1.0, ptr(i32[0]), ptr(i32[1]),
                                  ptr(bd), ptr(ws), ws.numel(), st)
        b.record()
        torch.cuda.synchronize()
        assert rc == 0
        if k >= 3:
            ms.append(a.elapsed_time(b))
    return statistics.median(ms)


@pytest.mark.parametrize("nearest", [True, False])
@pytest.mark.parametrize("below,above", [(8100, 8300), (11500, 11700)])
def test_the_line_costs_nothing(gpu, nearest, below, above):
    """Points strewn around the curve widen the grid's cells: above 2^26 pairs
    8300 of them took 2.1 (radius) and 3.9 times (nearest) the all-pairs scan."""
    assert device_ms(above, nearest) < 1.5 * device_ms(below, nearest)
