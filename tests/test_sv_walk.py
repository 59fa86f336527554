"""The single-view backprojector's channel addresses (csrc/sv_walk.h), built for
the host with signed overflow trapping."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_addresses(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "sv_walk_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", "-o", exe, os.path.join(HERE, "cpp", "sv_walk_check.cc")], check=True)
    cases, bad = map(int, subprocess.run([exe], capture_output=True, check=True).stdout.split())
    assert cases > 100000 and bad == 0
