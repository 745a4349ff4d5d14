"""The integer-pipe double-to-float conversion equals the IEEE conversion."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_against_the_host_conversion(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "float_rn_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", str(exe), os.path.join(HERE, "csrc", "float_rn_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
