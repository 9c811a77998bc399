"""How much memory a field handle's records may take (csrc/handles.h)."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_records_fit(tmp_path):
    exe = str(tmp_path / "records_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(CUDA, "include"), "-o", exe,
                    os.path.join(HERE, "records_check.cpp"), "-L", os.path.join(CUDA, "lib64"),
                    "-lcudart"], check=True)
    assert subprocess.run([exe]).returncode == 0
