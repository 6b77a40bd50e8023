"""The warp's taps are read as aligned words, never past the end of the frame
that the caller gave, whose allocation may end there: tests/tap_words_check.cpp compiles the kernel's load on the host
and watches it."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "image360_b200", "csrc")


def test_tap_loads_stay_inside_the_frame(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "tap_words_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", CSRC, "-o", exe, os.path.join(HERE, "tap_words_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
