"""The double-float quotient and the single quotients from a shared reciprocal
(forestfv_public_gb300/csrc/ffv_df.cuh), compiled for the host: the former within 2^-44 of the quotient
in extended precision over the range that the header states (the remainder's double-float subtraction
is good to 2^-46 of the dividend, the second quotient's rounding adds 2^-48), the latter with the
division's bits for every operand."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OUT = os.path.join(ROOT, "tests", "c", "_build")


def test_quotients():
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    os.makedirs(OUT, exist_ok=True)
    exe = os.path.join(OUT, "df_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Wno-unused-function",
                    "-I" + os.path.join(ROOT, "forestfv_public_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "c", "df_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert ", 0 failures" in r.stdout
