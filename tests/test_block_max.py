"""The block-wide maximum that sizes the streaming solve's stages (csrc/block_max.cuh), run by host threads
under ThreadSanitizer with thread 0 the last to arrive: its first store must not race with, or erase, the
others' maxima."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
MAIN = os.path.join(HERE, "sanitize", "block_max_main.cpp")


@pytest.mark.parametrize("flags", [[], ["-fsanitize=thread"]])
def test_late_first_thread(tmp_path, flags):
    gxx = shutil.which("g++") or "/usr/bin/g++"
    if not os.path.exists(gxx):
        pytest.skip("g++ not available")
    exe = str(tmp_path / "block_max")
    r = subprocess.run([gxx, "-std=c++20", "-O1", "-g", "-pthread", *flags, MAIN, "-o", exe], capture_output=True, text=True)
    if r.returncode != 0 and "tsan" in r.stderr.lower():
        pytest.skip("sanitizer runtime not available: " + r.stderr.strip()[-200:])
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120,
                       env=dict(os.environ, TSAN_OPTIONS="halt_on_error=1"))
    if "unexpected memory mapping" in r.stderr:
        pytest.skip("ThreadSanitizer does not run under this kernel's address layout")
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr[-2000:])
