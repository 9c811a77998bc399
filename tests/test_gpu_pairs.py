"""The packed pair arithmetic of csrc/split.cuh on the device, where a product
that was contracted into the sum after it would leave 2^-25 of its size: sums
and differences of products within 2^-43 (a product drops 2^-45 to 2^-46, the
low halves of a sum 2^-46), with and without the product of the low halves."""

import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("define", [[], ["-DMR_SPLIT_LOW_PRODUCT"]])
def test_products_are_not_contracted(tmp_path, define):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "pairs_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-fmad=false", *define, "-o", exe, os.path.join(HERE, "pairs_check.cu")],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0
    worst = [float(v) for v in out.stdout.split()]
    assert len(worst) == 8 and max(worst) <= 1.0, worst
