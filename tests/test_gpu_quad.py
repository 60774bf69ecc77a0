"""Four-warp DOP853 of the 42-dim system (a state warp and three warps of
third-columns per five trajectories): bit-identical to the CPU oracle, state
and STM, at batch sizes that split a group's third-columns over the three
warps in every way, with spans of their own, samples and flips."""
import numpy as np
import pytest

from hiten_gb300 import _lib
from hiten_gb300 import workloads as W

pytestmark = pytest.mark.gpu
MU = W.MU_EM


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 13, 761])
@pytest.mark.parametrize("fwd,flip", [(1, None), (-1, (36, 42)), (-1, (10, 40))])
def test_quad_dop853_matches_oracle(gpu, oracle, n, fwd, flip):
    y0 = W.stm_fixed_batch(n, seed=17)
    tf = np.linspace(0.3, 1.2, n)
    with gpu.tuning(lanes_d42=18):
        res = gpu.propagate_dop853(y0, 0.0, tf, MU, rtol=1e-11, atol=1e-11, fwd=fwd, flip=flip, n_samples=9)
    with gpu.tuning(lanes_d42=7):
        one = gpu.propagate_dop853(y0, 0.0, tf, MU, rtol=1e-11, atol=1e-11, fwd=fwd, flip=flip, n_samples=9)
    for a in ("y_end", "t_end", "n_accept", "n_reject", "status", "samples"):
        assert np.array_equal(getattr(res, a).cpu().numpy(), getattr(one, a).cpu().numpy()), a
    assert np.all(res.status.cpu().numpy() == _lib.HG_OK)
    oracle.set_mode(oracle.MODE_DEVICE)
    try:
        for i in np.unique([0, n // 2, n - 1]):
            ref, na, nr, st = oracle.dop853_dense(y0[i], np.linspace(0.0, tf[i], 9), MU, rtol=1e-11, atol=1e-11,
                                                  fwd=fwd, flip=flip)
            assert st == 0 and int(res.n_accept[i]) == na and int(res.n_reject[i]) == nr
            assert np.array_equal(res.samples.cpu().numpy()[:, i], ref)
    finally:
        oracle.set_mode(oracle.MODE_PYTHON)
