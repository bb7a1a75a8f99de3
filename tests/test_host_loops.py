"""The host loops about the sizes where they go from one thread to started threads to the kept
workers (forestfv_public_gb300/csrc/ffv_internal.h), compiled for the host and run as a program."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_element_once(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "loop_sizes")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-pthread",
                    "-I" + os.path.join(ROOT, "forestfv_public_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "c", "loop_sizes.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("0 failures"), r.stdout + r.stderr
