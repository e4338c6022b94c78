"""Units that take another number of limbs a loop body build their passes under
names of their own: one name stands for one function in the whole library, also
if its device code is linked across units."""

import os
import shutil
import subprocess

import pytest

from heu_gb300 import build

HEADERS = ["sq_encrypt.cuh", "sq_mul.cuh", "sq_decrypt.cuh"]
UNIT = """
%s
%s
#include <typeinfo>
const char* lanes_%d() { return typeid(hg::SqLanes<2, 16>).name(); }
int unroll_%d() { return hg::kSqUnroll<2, 16>; }
"""
MAIN = """
#include <cstdio>
const char* lanes_0();
const char* lanes_1();
int unroll_0();
int unroll_1();
int main() { std::printf("%s %s %d %d\\n", lanes_0(), lanes_1(), unroll_0(), unroll_1()); }
"""


def test_units_with_another_unrolling_have_names_of_their_own(tmp_path):
    nvcc = build._nvcc()
    if not (os.path.exists(nvcc) or shutil.which(nvcc)):
        pytest.skip("no nvcc")
    includes = "\n".join('#include "%s"' % h for h in HEADERS)
    for i, define in enumerate(("", "#define HG_SQ_UNROLL 4")):
        (tmp_path / f"u{i}.cu").write_text(UNIT % (define, includes, i, i))
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "names")
    cmd = [nvcc, *build.ARCH, "-std=c++17", "-I", build.CSRC, "-I", build.INCLUDE, "-o", exe]
    subprocess.run(cmd + [str(tmp_path / f) for f in ("u0.cu", "u1.cu", "main.cpp")], check=True, capture_output=True)
    name0, name1, unroll0, unroll1 = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert (unroll0, unroll1) == ("16", "4")
    assert name0 != name1
