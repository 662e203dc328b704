"""Entry positions near the largest nnz (2^31 - 1), walked on the host with the helpers that the
kernels use: every entry once, none past the end, no step that wraps."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_positions_up_to_the_largest_nnz(tmp_path):
    exe = str(tmp_path / "positions")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-o", exe,
                    os.path.join(HERE, "position_driver.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[:2000]
