"""The section kernel's queued crossings: samples that cross the plane almost
every segment (several crossings of one lane wait together and queues fill
inside a segment), refinements around the scan's chunks of 32 points, sample
counts around the loader's batches of 8, on-surface and repeated samples, ends
that underflow FP32, non-monotone times, and small hit caps -- every hit equals
the sequential oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,refine", [(2, 50), (3, 1), (8, 30), (9, 31), (10, 32), (16, 62), (17, 63), (18, 64), (40, 130),
                                      (41, 50)])
@pytest.mark.parametrize("interp,direction,max_hits", [("linear", 0, 64), ("cubic", 0, 3), ("cubic", -1, 64),
                                                       ("cubic", 1, 1), ("linear", 1, 9)])
def test_hits_equal_the_sequential_oracle(gpu, oracle, m, refine, interp, direction, max_hits):
    from hiten_gb300 import synodic
    n = 70
    rng = np.random.default_rng(m * 1000 + refine)
    S = rng.normal(0.0, 1.0, (m, n, 6))
    S[:, ::5, 1] *= 1e-3                           # near the plane
    S[:, 1::7, 1] = np.abs(S[:, 1::7, 1]) + 0.05   # mostly one side, cubic undershoot
    S[rng.integers(0, m, 40), rng.integers(0, n, 40), 1] = 0.0
    S[:, 3::11, 1] *= 1e-40
    if m > 3:
        S[1::4, 2::9, 1] = S[0::4, 2::9, 1][: len(range(1, m, 4))]
    t = np.sort(rng.uniform(0.0, 5.0, (m, n)), axis=0)
    if m > 5:
        t[4, 6::13] = t[3, 6::13]                  # repeated node
    ht, hy, nh = synodic.detect(t, S, section_axis="y", plane_coords=("x", "vx"), direction=direction,
                                segment_refine=refine, interp=interp, max_hits=max_hits)
    ht, hy, nh = ht.cpu().numpy(), hy.cpu().numpy(), nh.cpu().numpy()
    oracle.set_mode(oracle.MODE_DEVICE)
    with np.errstate(all="ignore"):
        for i in range(n):
            rt, ry = oracle.section_detect(t[:, i], S[:, i], 1, 0.0, direction, (0, 3), segment_refine=refine,
                                           cubic=interp == "cubic", max_hits=max_hits)
            assert nh[i] == len(rt)
            assert np.array_equal(ht[i, :nh[i]], rt, equal_nan=True)
            assert np.array_equal(hy[i, :nh[i]], ry, equal_nan=True)
    oracle.set_mode(oracle.MODE_PYTHON)
    assert nh.sum() > 0 or m == 2
