"""Build numbers of the device's linked lists do not come round (fd_build.h)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")


def test_numbers_do_not_come_round(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "fundem_b200", "csrc"),
                           os.path.join(ROOT, "tests", "apps", "build_clock_check.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split("\n")
    for line in out[:2]:
        kind, clean, without = line.split()
        assert clean == "1", line            # with the clock no cell holds an object that is not in it
        assert int(without) > 0, line        # without it some do
    assert out[2] == "limit 1" and out[3] == "resets 1 most 1"
