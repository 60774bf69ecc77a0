"""6-dim fixed-step propagation in the layouts its batch size selects (six,
two and one lane per trajectory): every row equals the oracle's bit for bit,
at the edges of a warp's trajectories (5, 16, 32) and of the layouts' ranges,
odd output strides and both directions."""
import numpy as np
import pytest

from hiten_gb300.workloads import MU_EM, stm_fixed_batch
from oracle import hgo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4, 5, 6, 159, 161, 9001, 9008, 30001, 30016])
@pytest.mark.parametrize("order,fwd,every", [(4, 1, 1), (6, -1, 3), (8, -1, 2), (8, 1, 7)])
def test_fixed_step_rows_match_oracle(gpu, n, order, fwd, every):
    hgo.set_mode(hgo.MODE_DEVICE)
    y = stm_fixed_batch(n, seed=n)[:, 36:].copy()
    t = np.cumsum(np.r_[0.0, np.linspace(0.5e-2, 2e-2, 7)])
    rows, status = gpu.propagate_fixed(y, t, MU_EM, order=order, out_every=every, fwd=fwd, return_status=True)
    ref, _ = hgo.fixed_rk_batch(order, y, t, MU_EM, out_every=every, fwd=fwd)
    assert np.array_equal(rows.cpu().numpy(), ref.transpose(1, 0, 2))
    assert not status.any()


@pytest.mark.parametrize("n", [7, 9001])
def test_fixed_step_flags_nonfinite_states(gpu, n):
    y = stm_fixed_batch(n, seed=1)[:, 36:].copy()
    bad = [0, n // 2, n - 1]
    y[bad, 3] = np.nan
    _, status = gpu.propagate_fixed(y, np.linspace(0.0, 0.1, 4), MU_EM, order=4, return_status=True)
    want = np.zeros(n, bool)
    want[bad] = True
    assert np.array_equal(status.cpu().numpy() != 0, want)
