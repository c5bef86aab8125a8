"""The integer sums of the heated FP64 deposits (csrc/tpm_fx.cuh) on the host:
tests/fx_sum_check.cpp compares sums of up to 70000 terms, in two orders, with the
exact sum rounded once."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "triplyperiodic-modified_gb300", "csrc")


def test_fx_sums(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    (tmp_path / "cuda_runtime.h").write_text("#pragma once\n")
    exe = tmp_path / "fx_sum_check"
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(tmp_path),
                           "-I", CSRC, os.path.join(HERE, "fx_sum_check.cpp"), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
