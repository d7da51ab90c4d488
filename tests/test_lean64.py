"""Host check of csrc/lean64.cuh: the correctly rounded roots, reciprocals, quotients and
products of the FP64 loops and the Morton grid cell, against the plain operators."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_lean64_matches_the_operators(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "lean64_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "native", "lean64_check.cpp")], check=True)
    r = subprocess.run([str(exe), "1000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert " wrong 0 " in r.stdout
