"""Destroying a handle does not wait for another handle's state copy
(tests/native/state_io_close.cu)."""
import os
import subprocess

import pytest

from tests.test_tma_geometry_cpu import ROOT, _nvcc

SRC = os.path.join(ROOT, "tests", "native", "state_io_close.cu")


def test_close_beside_a_copy(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "state_io_close")
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-I",
                           os.path.join(ROOT, "include"), SRC, "-o", exe, "-lpthread"])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "ok"
