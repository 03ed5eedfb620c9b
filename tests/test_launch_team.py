"""A solve whose team of blocks the device cannot place (fewer SMs for the process or stream) goes on with the
next team, or with the captured kernels: csrc/teams.h against a fake of the launch that returns the
errors, on the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
MAIN = os.path.join(HERE, "sanitize", "launch_team_main.cpp")
CUDA = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))


def test_refused_launches(tmp_path):
    gxx = shutil.which("g++") or "/usr/bin/g++"
    if not os.path.exists(gxx) or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")):
        pytest.skip("g++ or the CUDA headers not available")
    exe = str(tmp_path / "launch_team")
    r = subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(CUDA, "include"), MAIN, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
