"""The kernels' square roots and quotients on the integer pipes
(csrc/hg_exact.cuh), compiled as host C++ with FP32 estimates at the ends of
their admitted error, are IEEE's wherever they do not hand the value back; and
they hand back few."""
import os
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
