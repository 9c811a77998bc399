"""The pair arithmetic of mantaray_gb300/csrc/split.cuh, compiled for the host,
against long double over depths 0.01 m to 8 km and wavenumbers 1e-3 to 3
rad/m: the FP64 anchor within 16 units of 2^-53, the pairs' derivatives within
2^-42, the refraction factor within 2^-42 (1 + kh).  And dispersion.cuh: |k|
within 12 units of 2^-53 of the dispersion relation's root, cosine and sine
within 4."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _run(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, name + ".cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout
    return [float(v) for v in out.stdout.split()]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_split_arithmetic(tmp_path):
    checked, anchor, pair, f = _run(tmp_path, "split_check")
    assert checked > 200_000 and anchor <= 1 and pair <= 1 and f <= 1, (anchor, pair, f)


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_dispersion(tmp_path):
    checked, k, trig = _run(tmp_path, "dispersion_check")
    assert checked > 150_000 and k <= 1 and trig <= 1, (k, trig)
