"""The row-pair matvec's gather schedule, checked on the host against the
tables it is built from (tests/cpp/pair_schedule_check.cpp)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_pair_schedule_covers_tables(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    csrc = ROOT / "exact_diagonalization_for_fermionic_systems_with_gpu_gb300" / "csrc"
    exe = tmp_path / "pair_schedule_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", str(csrc), str(ROOT / "tests/cpp/pair_schedule_check.cpp"),
                    str(csrc / "ed_tables.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.count(" ok") == 14


def test_class_schedule_covers_tables(tmp_path):
    """The complex row engine's class schedule (tests/cpp/class_schedule_check.cpp)."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    csrc = ROOT / "exact_diagonalization_for_fermionic_systems_with_gpu_gb300" / "csrc"
    exe = tmp_path / "class_schedule_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", str(csrc), str(ROOT / "tests/cpp/class_schedule_check.cpp"),
                    str(csrc / "ed_tables.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.count(" ok") == 7
