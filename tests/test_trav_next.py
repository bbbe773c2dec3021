"""The eight lanes of a cooperative group choose the same next node, and leave the same stack, in whatever
order the lanes of the warp happen to run between two barriers (lmgpu_dev.cuh, on the host)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "lightmetrica-v3_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    exe = str(tmp_path_factory.mktemp("trav_next") / "check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-I", CSRC, "-I", os.path.join(CUDA, "include"), "-o", exe,
                    os.path.join(HERE, "trav_next_check.cpp")], check=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_group_agrees_in_any_order(checker, seed):
    r = subprocess.run([checker, str(seed)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
