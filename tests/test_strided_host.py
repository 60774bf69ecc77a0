"""The connection searches' index arithmetic (csrc/hg_strided.cuh) up to
2^31 - 1 items: every loop stays inside its count, takes each of its items once
and ends; whole blocks cover a count.  Compiled as host C++."""
import os
import re
import subprocess

from conftest import REPO

CSRC = os.path.join(REPO, "hiten_gb300", "csrc")


def test_indexes_up_to_the_largest_count(tmp_path):
    exe = str(tmp_path / "strided_check")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover", "-I" + CSRC,
                           os.path.join(REPO, "tests", "native", "strided_check.cpp"), "-o", exe])
    loops, wrong = map(int, subprocess.check_output([exe]).decode().split())
    assert loops == 13 * (2 + 15) and wrong == 0


def test_connection_kernels_index_through_it():
    """No thread index of the connection kernels is formed in 32 bits."""
    src = open(os.path.join(CSRC, "hg_connect.cu")).read()
    assert not re.findall(r"int \w+ = blockIdx\.x \* blockDim\.x", src)
