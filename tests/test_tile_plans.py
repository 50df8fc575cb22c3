"""Tile plans of the block kernels on the host: ``tests/native/tile_plan_check.cu`` is compiled by nvcc
as host code and checks the memo of the extents and the cells that the blocks of a cell range cover."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_tile_plans(tmp_path):
    exe = str(tmp_path / "tile_plan_check")
    subprocess.run(["nvcc", "-std=c++17", "--expt-relaxed-constexpr", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-x",
                    "cu", os.path.join(HERE, "native", "tile_plan_check.cu"), "-o", exe], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
