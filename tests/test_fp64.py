"""The bit-level FP64 helpers of the reference-exact kernels
(forestfv_public_gb300/csrc/ffv_fp64.cuh), compiled for the host, against the plain FP64
expressions they stand for: identical bits."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OUT = os.path.join(ROOT, "tests", "c", "_build")


def test_helpers_give_the_plain_expressions_bits():
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    os.makedirs(OUT, exist_ok=True)
    exe = os.path.join(OUT, "fp64_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Wno-unused-function",
                    "-I" + os.path.join(ROOT, "forestfv_public_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "c", "fp64_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert ", 0 mismatches" in r.stdout
