"""The connection searches through the grid (sets of more than 2^26 pairs):
counts, nearest partners and nearest neighbours equal the exhaustive binary64
search with the lowest index winning ties -- curves, uniform clouds, crowded
cells, one far outlier, repeated points, collinear and identical points, radii
from zero to the whole extent, and coordinates that are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def clouds(kind, n, rng):
    s = rng.uniform(0, 1, n)
    if kind == "curve":
        return np.c_[0.1 * np.cos(6 * s) + rng.normal(0, 1e-4, n), 0.3 * np.sin(6 * s) + rng.normal(0, 1e-4, n)]
    if kind == "uniform":
        return rng.uniform(-1, 1, (n, 2))
    if kind == "crowded":
        return np.where(rng.uniform(size=(n, 1)) < 0.9, rng.normal(0.5, 1e-6, (n, 2)), rng.uniform(-1, 1, (n, 2)))
    if kind == "outlier":
        p = rng.normal(0.7, 1e-3, (n, 2))
        p[n // 2] = (-50.0, 80.0)
        return p
    if kind == "repeated":
        return rng.integers(0, 60, (n, 2)) / 64.0
    if kind == "collinear":
        return np.c_[s, np.full(n, 0.25)]
    if kind == "identical":
        return np.full((n, 2), 0.3)
    p = rng.uniform(-1, 1, (n, 2))
    p[rng.integers(0, n, 9), 0] = np.nan
    p[rng.integers(0, n, 9), 1] = np.inf
    return p


def exhaustive(q, r, eps, self_search):
    cnt, idx, best = [], [], []
    with np.errstate(all="ignore"):
        for k in range(0, len(q), 512):
            dx = q[k:k + 512, :1] - r[None, :, 0]
            dy = q[k:k + 512, 1:] - r[None, :, 1]
            d2 = dx * dx + dy * dy
            if self_search:
                d2[np.arange(d2.shape[0]), np.arange(k, k + d2.shape[0])] = np.inf
            ok = d2 <= eps * eps if eps is not None else d2 < 1e300
            d2 = np.where(ok, d2, np.inf)
            j = np.argmin(d2, axis=1)
            cnt.append(ok.sum(1))
            idx.append(np.where(ok.any(1), j, -1))
            best.append(np.where(ok.any(1), d2[np.arange(len(j)), j], 0.0))
    return np.concatenate(cnt), np.concatenate(idx), np.concatenate(best)


KINDS = ["curve", "uniform", "crowded", "outlier", "repeated", "collinear", "identical", "nonfinite"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("eps", [0.0, 1e-4, 0.02, 5.0])
def test_radius_search(gpu, kind, eps):
    from hiten_gb300.connections import GpuSectionMatcher
    rng = np.random.default_rng(len(kind))
    q, r = clouds(kind, 9001, rng), clouds(kind, 8193, rng)
    q[:50] = r[100:150]
    c = float(np.nanmax(np.abs(np.where(np.isfinite(np.r_[q, r]), np.r_[q, r], 0.0))))
    cnt, idx, d2 = GpuSectionMatcher().radius_best(q, r, eps, c)
    ec, ei, ed = exhaustive(q, r, eps, False)
    assert np.array_equal(cnt, ec) and np.array_equal(idx, ei) and np.array_equal(d2, ed)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [8193, 9000])
def test_nearest_search(gpu, kind, n):
    from hiten_gb300.connections import GpuSectionMatcher
    p = clouds(kind, n, np.random.default_rng(n))
    c = float(np.nanmax(np.abs(np.where(np.isfinite(p), p, 0.0))))
    out = GpuSectionMatcher().nearest(p, c)
    assert np.array_equal(out, exhaustive(p, p, None, True)[1])
