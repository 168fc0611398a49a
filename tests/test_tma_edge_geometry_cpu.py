"""The edge tiles' TMA halo boxes of the MHD stage, checked on the CPU: a host
program (tests/native/tma_edge_geometry.cu, compiled by nvcc against the
kernels' own header) checks every tile of every grid width the tensor copies
serve: aligned box start, stencil windows inside the box, flux columns that
cover them."""
import os
import subprocess

import pytest

from tests.test_tma_geometry_cpu import ROOT, _nvcc

SRC = os.path.join(ROOT, "tests", "native", "tma_edge_geometry.cu")


def test_edge_boxes_are_aligned_and_cover_the_stencils(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "tma_edge_geometry")
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-I",
                           os.path.join(ROOT, "include"), SRC, "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok ") and int(r.stdout.split()[1]) > 10_000
