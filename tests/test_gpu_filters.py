"""Trajectory filters over chunks of samples: the values of the sequential
evaluation (one running minimum and maximum per trajectory) bit for bit, at
the edges of blocks (64 trajectories) and chunks (16 samples), with
non-finite samples anywhere."""
import numpy as np
import pytest

from hiten_gb300.workloads import MU_EM

pytestmark = pytest.mark.gpu


def reference(S, mu):
    """manifold.py:412-432 and energy.py:26-74 sample by sample in numpy binary64."""
    mu1 = 1.0 - mu
    with np.errstate(all="ignore"):
        x, y, z, vx, vy, vz = (S[:, :, c] for c in range(6))
        yy, zz = y * y, z * z
        d1 = np.sqrt(((x + mu) * (x + mu) + yy) + zz)
        b = (x - 1.0) + mu
        d2 = np.sqrt((b * b + yy) + zz)
        f = x - mu1
        r2 = np.sqrt((f * f + yy) + zz)
        C = ((x * x + yy) + 2.0 * (mu1 / d1 + mu / r2)) - ((vx * vx + vy * vy) + vz * vz)
        m1, m2, e = d1[0].copy(), d2[0].copy(), np.zeros(S.shape[1])
        a0 = np.abs(C[0])
        for q in range(1, S.shape[0]):
            m1 = np.where(d1[q] < m1, d1[q], m1)
            m2 = np.where(d2[q] < m2, d2[q], m2)
            d = np.abs(C[q] - C[0])
            rel = np.where(a0 > 1e-14, d / a0, d)
            e = np.where(rel > e, rel, e)
    return m1, m2, e


@pytest.mark.parametrize("n,m", [(1, 1), (1, 16), (1, 17), (63, 33), (64, 1000), (65, 31), (129, 4713), (2000, 5),
                                 (120000, 20)])
@pytest.mark.parametrize("special", [False, True])
def test_filters_equal_the_sequential_scan(gpu, n, m, special):
    import torch

    from hiten_gb300 import manifold
    rng = np.random.default_rng(n * 7919 + m)
    S = rng.normal(0.0, 0.5, (m, n, 6)) + np.array([0.85, 0, 0, 0, 0, 0])
    if special:
        k = max(1, n // 5)
        for v in (np.nan, np.inf, -np.inf, 1e200, 0.0):
            S[rng.integers(0, m, k), rng.integers(0, n, k), rng.integers(0, 6, k)] = v
        S[0, rng.integers(0, n, k), rng.integers(0, 6, k)] = np.nan
        S[0, rng.integers(0, n, k), 0] = -MU_EM
    got = manifold.trajectory_filters(torch.as_tensor(S, device="cuda"), MU_EM)
    for g, w in zip(got, reference(S, MU_EM)):
        assert np.array_equal(g.cpu().numpy(), w, equal_nan=True)
