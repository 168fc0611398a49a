"""The parities of the MHD stage blocks' layer barriers over a batch's work-list,
modelled on the CPU with the kernels' own rule (tests/native/mhd_phase_model.cu):
items with tensor copies and without them, in any order and of any layer count,
must leave every wait at the phase the barrier is in."""
import os
import subprocess

import pytest

from tests.test_tma_geometry_cpu import ROOT, _nvcc

SRC = os.path.join(ROOT, "tests", "native", "mhd_phase_model.cu")


def test_mixed_items_keep_the_barrier_parity(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "mhd_phase_model")
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-I",
                           os.path.join(ROOT, "include"), SRC, "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok ") and int(r.stdout.split()[1]) > 100_000
