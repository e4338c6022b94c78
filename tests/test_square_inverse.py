"""The batch inverse's root modulo n^2 (host code): one inverse modulo n, lifted
once.  Every result recomputed with Python integers; needs only g++."""

import math
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_square_inverse_matches_python_integers(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "square_inverse_test")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-o", exe,
                    os.path.join(HERE, "cpp", "square_inverse_test.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300, check=True).stdout
    cases = [line.split()[1:] for line in out.splitlines() if line.startswith("case")]
    assert len(cases) == 50
    for S, n, x, got in cases:
        n, x, r2 = int(n, 16), int(x, 16), pow(2, 64 * int(S))
        if math.gcd(x, n) != 1:
            assert got == "none"
        else:
            assert int(got, 16) == r2 * pow(x, -1, n * n) % (n * n)
