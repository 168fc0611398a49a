"""DAMPING's set-up where memory is short (tests/native/damping_fallback.cu): a box
whose velocities fit one at a time is not refused because three at a time do
not."""
import os
import subprocess

import pytest

from tests.test_tma_geometry_cpu import ROOT, _nvcc

SRC = os.path.join(ROOT, "tests", "native", "damping_fallback.cu")


def test_one_field_at_a_time_where_three_do_not_fit(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "damping_fallback")
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-I",
                           os.path.join(ROOT, "include"), SRC, "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "ok"
