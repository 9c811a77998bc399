"""Two host units of csrc/split.cuh, with and without the product of the low
halves, in one program: each keeps its own form."""

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mantaray_gb300",
                    "csrc")

UNIT = """
#include "{csrc}/split.cuh"
float {name}(float h, float l) {{
  return mr::sqr(mr::F2{{h, l}}).l + mr::mul(mr::F2{{h, l}}, mr::F2{{h, l}}).l;
}}
"""
MAIN = """
#include <stdio.h>
float with_low(float, float), without_low(float, float);
int main() { printf("%a %a\\n", with_low(1.0f, 0x1p-20f), without_low(1.0f, 0x1p-20f)); }
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("order", [[0, 1], [1, 0]])
def test_forms_of_the_product_link(tmp_path, order):
    objects = []
    for name, define in (("with_low", ["-DMR_SPLIT_LOW_PRODUCT"]), ("without_low", [])):
        src, obj = tmp_path / (name + ".cpp"), tmp_path / (name + ".o")
        src.write_text(UNIT.format(csrc=CSRC, name=name))
        subprocess.run(["g++", "-O0", "-std=c++17", "-ffp-contract=off", *define, "-c", "-o",
                        str(obj), str(src)], check=True)
        objects.append(str(obj))
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "forms")
    subprocess.run(["g++", "-o", exe, str(tmp_path / "main.cpp"), *[objects[i] for i in order]],
                   check=True)
    a, b = (float.fromhex(v) for v in subprocess.run([exe], capture_output=True,
                                                     text=True).stdout.split())
    # (1 + 2^-20)^2 has 2^-40 in the product of the low halves
    assert b == 2 * 2.0 ** -19 and a == 2 * (2.0 ** -19 + 2.0 ** -40)
