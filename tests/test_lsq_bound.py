"""lsq_decide (csu_b200/csrc/cuda/lsqdd.cuh), the gradient kernel's rounding decision from exact sums and an error
bound, against this host's x87 long double: no component it decides differs by a bit, uniform fields are decided
exactly, and ordinary cells nearly always (on power-of-two spacings exact ties are common and stay undecided)."""
import os
import platform
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(platform.machine() != "x86_64", reason="needs x87 long double")
def test_decided_components_equal_x87(tmp_path):
    exe = str(tmp_path / "lsqsum_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(ROOT, "tests", "native", "lsqsum_check.cpp")], check=True)
    r = subprocess.run([exe, "1000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    f = dict(kv.split("=") for kv in r.stdout.split() if "=" in kv)
    assert f["mismatches"] == "0", r.stdout
    assert float(f["decided5"]) == 1.0, r.stdout
    assert float(f["decided0"]) > 0.95, r.stdout
