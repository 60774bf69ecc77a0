"""The grid searches at scales where FP32 screens decide little or nothing:
coordinates below, near and beyond FP32's range, and sets whose extent is below
FP32's spacing at their distance from the origin -- the exhaustive binary64
results all the same."""
import numpy as np
import pytest

from test_gpu_far_points import curve, with_far
from test_gpu_grid_search import exhaustive

pytestmark = pytest.mark.gpu

SCALES = [1e-140, 1e-60, 1e-40, 1e-30, 1e-19, 1e18, 1e30, 1e38, 1e60, 1e140]


@pytest.mark.parametrize("kind", ["none", "hundred", "lattice", "pairs"])
@pytest.mark.parametrize("scale,offset", [(s, 0.0) for s in SCALES] + [(1.0, 1e3), (1e-4, 1.0), (1e-9, 1.0)])
def test_nearest(gpu, kind, scale, offset):
    from hiten_gb300.connections import GpuSectionMatcher
    rng = np.random.default_rng(3)
    p = scale * with_far(curve(8203, rng), kind, rng) + offset
    near = GpuSectionMatcher().nearest(p, float(np.abs(p).max()))
    assert np.array_equal(near, exhaustive(p, p, None, True)[1])


@pytest.mark.parametrize("scale,offset", [(s, 0.0) for s in SCALES] + [(1.0, 1e3), (1e-4, 1.0), (1e-9, 1.0)])
def test_radius(gpu, scale, offset):
    from hiten_gb300.connections import GpuSectionMatcher
    rng = np.random.default_rng(4)
    q, r = (scale * with_far(curve(n, rng), "hundred", rng) + offset for n in (12001, 11403))
    c = float(np.abs(np.r_[q, r]).max())
    cnt, idx, d2 = GpuSectionMatcher().radius_best(q, r, 1e-3 * scale, c)
    ec, ei, ed = exhaustive(q, r, 1e-3 * scale, False)
    assert np.array_equal(cnt, ec) and np.array_equal(idx, ei) and np.array_equal(d2, ed)
