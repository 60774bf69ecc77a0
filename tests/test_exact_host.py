"""The kernels' square roots and quotients on the integer pipes
(csrc/hg_exact.cuh), compiled as host C++ with FP32 estimates at the ends of
their admitted error, are IEEE's wherever they do not hand the value back; and
they hand back few."""
import os
import platform
import subprocess

import pytest

from conftest import REPO


@pytest.mark.parametrize("seed", [1, 2])
def test_integer_sqrt_and_quotient_match_ieee(tmp_path, seed):
    exe = str(tmp_path / "exact_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                           "-I" + os.path.join(REPO, "hiten_gb300", "csrc"),
                           os.path.join(REPO, "tests", "native", "exact_check.cpp"), "-o", exe])
    n, wrong, rq, rqo, rs, rso = map(int, subprocess.check_output([exe, "4000000", str(seed)]).decode().split())
    assert n == 4000000 and wrong == 0
    # handed back: |fr| within 2^-13 (quotient), 4e-4 (root) of a half, two sides each
    assert rq > 100000 and rq - rqo < 1.5 * 2 * 2.0 ** -13 * rq + 50
    assert rs > 100000 and rs - rso < 1.5 * 2 * 4e-4 * rs + 50


def test_integer_powers_match_quad(tmp_path):
    """The step-size controller's powers on the integer pipes
    (csrc/hg_powint.cuh) are the correctly rounded ones wherever they do not
    hand the value back (one in 340: six of the 2048 patterns below the
    rounded bits)."""
    exe = str(tmp_path / "powint_check")
    cmd = ["g++", "-O2", "-std=gnu++17", "-ffp-contract=off", "-I" + os.path.join(REPO, "hiten_gb300", "csrc"),
           os.path.join(REPO, "tests", "native", "powint_check.cpp"), "-o", exe]
    if platform.machine() not in ("aarch64", "arm64"):
        cmd.append("-lquadmath")
    subprocess.check_call(cmd)
    n, wrong, rnd, ok, rts, rok = map(int, subprocess.check_output([exe, "200000"]).decode().split())
    assert n > 1_000_000 and wrong == 0
    assert rnd > 1_000_000 and rnd - ok < 1.5 * 6 / 2048 * rnd
    # x^1.5 hands back 8 of 2048 patterns, x^2.5 twelve
    assert rts == 400_000 and rts - rok < 1.5 * 10 / 2048 * rts
