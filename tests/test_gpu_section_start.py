"""Section detection of trajectories that start on the surface: the sequential
oracle's hits at small caps; where one crossing is wanted the one at the start
spares the scan."""
import statistics

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def samples(m, n, start, rng):
    S = rng.normal(0.0, 1.0, (m, n, 6))
    S[:, :, 1] = 0.5 + np.abs(S[:, :, 1])
    if start == "on":
        S[0, :, 1] = 0.0
    elif start == "some on":
        S[0, ::3, 1] = 0.0
        S[m // 2, ::5, 1] = -1.0
    elif start == "resting":
        S[:m // 2 + 1, ::2, 1] = 1e-9 * rng.normal(size=(m // 2 + 1, (n + 1) // 2))
    return S


@pytest.mark.parametrize("start", ["on", "some on", "resting"])
@pytest.mark.parametrize("interp", ["linear", "cubic"])
@pytest.mark.parametrize("direction", [0, 1, -1])
@pytest.mark.parametrize("max_hits", [1, 2, 5])
def test_hits_equal_the_sequential_oracle(gpu, oracle, start, interp, direction, max_hits):
    from hiten_gb300 import synodic
    n, m = 45, 12
    S = samples(m, n, start, np.random.default_rng(max_hits))
    t = np.linspace(0.0, 2.0, m)
    ht, hy, nh = (a.cpu().numpy() for a in synodic.detect(t, S, section_axis="y", plane_coords=("x", "vx"),
                                                          direction=direction, interp=interp, max_hits=max_hits))
    oracle.set_mode(oracle.MODE_DEVICE)
    for i in range(n):
        rt, ry = oracle.section_detect(t, S[:, i], 1, 0.0, direction, (0, 3), segment_refine=50,
                                       cubic=interp == "cubic", max_hits=max_hits)
        assert nh[i] == len(rt)
        assert np.array_equal(ht[i, :nh[i]], rt) and np.array_equal(hy[i, :nh[i]], ry)
    oracle.set_mode(oracle.MODE_PYTHON)


@pytest.mark.parametrize("interp", ["linear", "cubic"])
def test_one_crossing_at_the_start_spares_the_scan(gpu, interp):
    """With 20000 sub-intervals a segment, 32 trajectories whose start is the one
    crossing wanted take no longer than 32 without a crossing."""
    import torch
    from hiten_gb300 import synodic
    t = torch.linspace(0.0, 1.0, 3, dtype=torch.float64, device="cuda")

    def ms(start):
        S = torch.as_tensor(samples(3, 32, start, np.random.default_rng(0)), device="cuda")
        out = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            synodic.detect(t, S, section_axis="y", plane_coords=("x", "vx"), direction=None, segment_refine=20000,
                           interp=interp, max_hits=1)
            b.record()
            torch.cuda.synchronize()
            out.append(a.elapsed_time(b))
        return statistics.median(out[2:])

    assert ms("on") < 2.0 * ms("off")
