"""Small 6-dim DOP853 batches, one trajectory per warp (five six-lane groups
sharing the stage sums and the dense samples): the results of the six-lane
layout bit for bit -- sample counts around the groups' stride of five, several
samples inside one step, the last sample only, events with several hits, spans
of zero, and a segmented run that pauses and resumes."""
import numpy as np
import pytest

from hiten_gb300.workloads import MU_EM, section_states, stm_fixed_batch

pytestmark = pytest.mark.gpu


def same(a, b):
    for k, v in vars(a).items():
        w = getattr(b, k)
        assert (v is None) == (w is None), k
        if v is not None:
            assert np.array_equal(v.cpu().numpy(), w.cpu().numpy(), equal_nan=True), k


@pytest.mark.parametrize("n,m,last", [(1, 2, False), (1, 6, False), (3, 37, False), (2, 1001, False), (7, 500, True),
                                      (900, 11, False)])
@pytest.mark.parametrize("fwd", [1, -1])
def test_samples_equal_the_six_lane_layout(gpu, n, m, last, fwd):
    y = stm_fixed_batch(n, seed=m)[:, 36:].copy()
    tmax = np.linspace(0.4, 2.0, n)
    tmax[-1] = 0.0 if n > 2 else tmax[-1]
    kw = dict(rtol=1e-11, atol=1e-11, max_steps=400, fwd=fwd, n_samples=m, sample_last_only=last)
    wide = gpu.propagate_dop853(y, 0.0, tmax, MU_EM, **kw)
    with gpu.tuning(lanes_d6=6):
        six = gpu.propagate_dop853(y, 0.0, tmax, MU_EM, **kw)
    same(wide, six)


@pytest.mark.parametrize("n,hits", [(1, 1), (5, 8), (901, 3)])
@pytest.mark.parametrize("segmented", [False, True])
def test_events_equal_the_six_lane_layout(gpu, n, hits, segmented):
    y = section_states(n, seed=hits)
    ev = gpu.EventSpec(index=1, offset=0.0, direction=-1, max_hits=hits)
    kw = dict(rtol=1e-11, atol=1e-11, event=ev, segmented=segmented, seg_steps=7, max_segments=3)
    wide = gpu.propagate_dop853(y, 0.0, 8.0, MU_EM, **kw)
    with gpu.tuning(lanes_d6=6):
        six = gpu.propagate_dop853(y, 0.0, 8.0, MU_EM, **kw)
    same(wide, six)
