"""The layout rules of hg_internal.h around their changeovers, compiled as host
C++: where a trajectory gets a warp (the sizes of test_gpu_wide_layout.py among
them), six, two lanes or one; where 42-dim runs go from groups of three or four
warps to pairs; and bench.py's copy of the rule, which names the layout of the
timed launch."""
import os
import subprocess

import pytest

import bench
from conftest import REPO


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("lanes") / "lanes_rule")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I" + os.path.join(REPO, "hiten_gb300", "csrc"),
                           "-I" + os.path.join(REPO, "include"),
                           os.path.join(REPO, "tests", "native", "lanes_rule.cpp"), "-o", exe])

    def run(ns, sms=152, cap=3.0):
        out = subprocess.check_output([exe, str(sms), str(cap)] + [str(n) for n in ns]).decode().split()
        return [tuple(map(int, out[3 * k + 1:3 * k + 3])) for k in range(len(ns))]
    return run


def test_a_warp_per_trajectory_where_the_wide_layout_is_tested(rule):
    assert [g for g, _ in rule([1, 2, 3, 5, 7, 900, 901])] == [30] * 7


def test_lanes_never_grow_with_the_batch(rule):
    ns = sorted({int(1.03 ** k) for k in range(1, 420)})
    got = rule(ns)
    d6 = [g for g, _ in got]
    assert d6 == sorted(d6, reverse=True) and set(d6) == {30, 6, 2, 1}
    # 18 up to three groups of five trajectories an SM
    assert [g for _, g in rule([1, 760, 2280, 2281, 4096])] == [18, 18, 18, 12, 12]
    assert [g for _, g in got] == [18 if n <= 2280 else 12 for n in ns]


@pytest.mark.parametrize("sms,cap", [(152, 3.0), (148, 3.0), (152, 4.0)])
def test_bench_names_the_layout_of_the_rule(rule, sms, cap):
    ns = [1, 100, 900, 1100, 1300, 4000, 6000, 7296, 9728, 16384, 19456, 25000, 29184, 48640, 65536]
    got = [6 if g == 30 else g for g, _ in rule(ns, sms, cap)]
    assert got == [bench.sched_lanes(n, cap * sms, sms) for n in ns]
