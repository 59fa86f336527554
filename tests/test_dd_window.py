"""The channels that the distance-driven grad's tiles stage (csrc/dd_window.h),
built for the host: pieces read staged channels only, and cover every position
of a tile, for all footprints (pixels up to 60 channels wide)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_window(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "dd_window_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "cpp", "dd_window_check.cc")], check=True)
    cases, bad = map(int, subprocess.run([exe], capture_output=True, check=True).stdout.split())
    assert cases > 100000 and bad == 0
