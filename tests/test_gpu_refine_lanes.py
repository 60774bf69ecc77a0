"""Deferred refinement of 6-dim crossings on six lanes (two halvings a pass, up
to 40 crossings of capacity per SM) and on one lane: the same bits, at the line
between the two, with tolerances that end the bisection on either halving of a
pass or not at all."""
import numpy as np
import pytest
import torch

from hiten_gb300 import workloads as W

pytestmark = pytest.mark.gpu
MU = W.MU_EM
FIELDS = ("hit_t", "hit_y", "n_hits", "t_end", "y_end", "status", "n_accept")


@pytest.fixture(scope="module")
def line(gpu):
    return 40 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("xtol,gtol", [(1e-12, 1e-12), (1e-3, 1e-30), (2e-3, 1e-30), (1e-9, 1e-5), (0.0, 0.0)])
@pytest.mark.parametrize("fwd,direction", [(1, 0), (-1, 0), (1, 1), (1, -1)])
def test_six_lanes_equal_one_lane(gpu, line, xtol, gtol, fwd, direction):
    ev = gpu.EventSpec(index=1, offset=0.0, direction=direction, max_hits=1, xtol=xtol, gtol=gtol)
    y0 = W.section_states(line + 1, seed=4)

    def run(y):
        return gpu.propagate_dop853(y, 0.0, 2.0, MU, rtol=1e-11, atol=1e-11, fwd=fwd, flip=(0, 6), event=ev)

    one = run(y0)  # one lane: a capacity of line + 1 crossings
    assert int(one.n_hits.sum()) > 0
    for n in (1, 4, 5, 6, 31, line):
        six = run(y0[:n])
        for f in FIELDS:
            a, b = getattr(six, f), getattr(one, f)[:n]
            if f in ("hit_t", "hit_y"):
                a, b = a[six.n_hits > 0], b[six.n_hits > 0]
            assert torch.equal(a, b), (n, f)


@pytest.mark.parametrize("n", [1, 7, 190])
def test_six_lanes_many_hits_match_oracle(gpu, oracle, n):
    y0 = W.section_states(n, seed=9)
    ev = gpu.EventSpec(index=1, offset=0.0, direction=-1, max_hits=8)
    res = gpu.propagate_dop853(y0, 0.0, 10.0, MU, rtol=1e-11, atol=1e-11, event=ev)
    oracle.set_mode(oracle.MODE_DEVICE)
    try:
        ref = oracle.dop853_event_batch(y0, 0.0, 10.0, MU, 1, 0.0, -1, 8, rtol=1e-11, atol=1e-11, max_step=1e4)
    finally:
        oracle.set_mode(oracle.MODE_PYTHON)
    hits = res.n_hits.cpu().numpy()
    assert np.array_equal(hits, ref["n_hits"])
    for i, k in enumerate(hits):
        assert np.array_equal(res.hit_t[i, :k].cpu().numpy(), ref["hit_t"][i, :k])
        assert np.array_equal(res.hit_y[i, :k].cpu().numpy(), ref["hit_y"][i, :k])
