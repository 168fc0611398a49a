"""The bound of the kernels' mbarrier waits (tests/native/bounded_wait.cu): by
time, not only by polls, each of which may suspend for microseconds."""
import os
import subprocess

import pytest

from tests.test_tma_geometry_cpu import ROOT, _nvcc

SRC = os.path.join(ROOT, "tests", "native", "bounded_wait.cu")


def test_a_wait_ends_by_the_clock(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "bounded_wait")
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "-gencode",
                           "arch=compute_100a,code=sm_100a", "--extended-lambda", "-I",
                           os.path.join(ROOT, "include"), SRC, "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "ok"
