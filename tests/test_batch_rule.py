"""The choice between the two batch kernels (csrc/batch_rule.h), on the host: a launch shape is refused only where
the kernel that takes every batch does not fit."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_rule(tmp_path):
    gxx = shutil.which("g++") or "/usr/bin/g++"
    if not os.path.exists(gxx):
        pytest.skip("g++ not available")
    exe = str(tmp_path / "batch_rule")
    r = subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", os.path.join(HERE, "sanitize", "batch_rule_main.cpp"),
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
