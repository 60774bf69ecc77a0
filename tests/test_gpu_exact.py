"""Square roots and quotients of csrc/hg_exact.cuh on the device (the
hardware's FP32 estimates, the FP64 sequences behind them) give the bits of
IEEE sqrt and division and of the hg_div_rn sequence."""
import os
import subprocess

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu


def test_exact_device_forms(gpu, tmp_path):
    exe = str(tmp_path / "exact_check")
    subprocess.check_call(["nvcc", "-std=c++17", "-gencode=arch=compute_103a,code=sm_103a", "-O3", "--fmad=false",
                           "-I" + os.path.join(REPO, "hiten_gb300", "csrc"),
                           os.path.join(REPO, "tests", "native", "exact_check.cu"), "-o", exe])
    n, wrong, err = subprocess.check_output([exe, str(1 << 28)], timeout=300).decode().split()
    assert err == "cudaSuccess" and int(n) == 1 << 28
    assert int(wrong) == 0, f"{wrong} results differ from IEEE arithmetic"
