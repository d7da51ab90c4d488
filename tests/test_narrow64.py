"""Host check of csrc/split64.cuh's narrow64 and widen32 against the plain conversions, and of
the share of roots, reciprocals and quotients of csrc/lean64.cuh that fail their proof."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_conversions_and_proofs(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "narrow64_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "native", "narrow64_check.cpp")], check=True)
    r = subprocess.run([str(exe), "4000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert " wrong 0 " in r.stdout
