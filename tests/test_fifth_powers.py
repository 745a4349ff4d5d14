"""The linear-spring law's powers of the impact velocity, x^0.2 and x^0.4, and
the grouped roots and quotients, against the host's arithmetic."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_against_the_host(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "fifth_powers_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "csrc", "fifth_powers_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
