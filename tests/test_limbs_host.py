"""The integer coefficients of the exact sums over basis vectors, on the host
(tests/cpp/limb_coefs_check.cpp)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_ritz_coefficients_keep_their_bits(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    csrc = ROOT / "exact_diagonalization_for_fermionic_systems_with_gpu_gb300" / "csrc"
    exe = tmp_path / "limb_coefs_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", str(csrc), str(ROOT / "tests/cpp/limb_coefs_check.cpp"),
                    str(csrc / "ed_limbs.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.count(" ok") == 72
