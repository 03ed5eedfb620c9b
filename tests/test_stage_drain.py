"""The end of the layer kernel's pipeline after a timeout (csrc/stage_drain.cuh), on the host: whichever tiles its two
producers stopped at, every barrier phase that copies were issued for ends."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_stop(tmp_path):
    gxx = shutil.which("g++") or "/usr/bin/g++"
    if not os.path.exists(gxx):
        pytest.skip("g++ not available")
    exe = str(tmp_path / "stage_drain")
    r = subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", os.path.join(HERE, "sanitize", "stage_drain_main.cpp"),
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
