"""The pair arithmetic of mantaray_gb300/csrc/split.cuh, compiled for the host,
against long double over depths 0.01 m to 8 km and wavenumbers 1e-3 to 3
rad/m: the FP64 anchor within 16 units of 2^-53, the pairs' derivatives within
2^-42, the refraction factor within 2^-42 (1 + kh)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_split_arithmetic(tmp_path):
    exe = str(tmp_path / "split_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "split_check.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    checked, anchor, pair, f = out.stdout.split()
    assert out.returncode == 0 and int(checked) > 200_000, out.stdout
    assert float(anchor) <= 1 and float(pair) <= 1 and float(f) <= 1, out.stdout
