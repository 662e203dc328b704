"""The cache of matrix memory (csrc/block_cache.cuh) on a stand-in for CUDA, without a GPU:
contexts that are reset, several devices, memory that runs short, matrices freed twice."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("block_cache") / "driver")
    cmd = ["g++", "-std=c++17", "-O1", "-Wall", "-o", exe, os.path.join(HERE, "block_cache_driver.cpp"), "-lpthread"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
    return exe


@pytest.mark.parametrize("what", ["reuse", "reset", "devices", "twice", "waits", "room"])
def test_block_cache(driver, what):
    res = subprocess.run([driver, what], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout[-2000:]
