"""The section kernel's FP32 segment skip (csrc/hg_section_skip.cuh), compiled
as host C++, never skips a segment in which the reference's binary64 Hermite
form changes sign at a scanned point, and skips most segments away from the
plane."""
import os
import subprocess

from conftest import REPO


def test_fp32_skip_is_certain(tmp_path):
    exe = str(tmp_path / "section_skip_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                           "-I" + os.path.join(REPO, "hiten_gb300", "csrc"),
                           os.path.join(REPO, "tests", "native", "section_skip_check.cpp"), "-o", exe])
    n, clear, wrong = map(int, subprocess.check_output([exe, "2000000"]).decode().split())
    assert n == 2000000 and wrong == 0
    assert clear > 0.2 * n
