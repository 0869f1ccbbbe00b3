"""Device allocations of batched Lanczos calls, counted by a stand-in for
cudaMalloc (tests/cpp/count_malloc.c) in a child process: a batch of one and a
batch sent to the mixed-sector kernel build no row-pair tables, and a batch on
the row pairs builds them once, in one allocation."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
PYPATH = os.pathsep.join([str(ROOT)] + ([os.environ["PYTHONPATH"]] if os.environ.get("PYTHONPATH") else []))

CHILD = r"""
import ctypes, os
import exact_diagonalization_for_fermionic_systems_with_gpu_gb300 as ed
from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L

calls = ctypes.CDLL(None).malloc_calls
ops = [ed.Hubbard(ed.H_TBq(9, 4).extend(t), ed.H_TBq(9, 3).extend(t), 2.0)
       for t in (L.chain(9, eps=[0.1 * b * i for i in range(9)]) for b in range(3))]
for op in ops:  # the workspaces
    ed.Lanczos().eigen(op, max_steps=10, mode="fixed")

def made(ops):
    n = calls()
    ed.lanczos_batch(ops, 10, seed=1)
    return calls() - n

os.environ["ED_LZ_BATCH"] = "multi"
multi = made(ops)
del os.environ["ED_LZ_BATCH"]
print(made(ops[:1]), multi, made(ops), made(ops))
"""


def test_batch_builds_the_tables_it_uses(ed, tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    so = tmp_path / "count_malloc.so"
    subprocess.run([cc, "-shared", "-fPIC", "-O1", str(ROOT / "tests/cpp/count_malloc.c"), "-o", str(so), "-ldl"],
                   check=True)
    r = subprocess.run([sys.executable, "-c", CHILD], env=dict(os.environ, PYTHONPATH=PYPATH, LD_PRELOAD=str(so)),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert [int(v) for v in r.stdout.split()] == [0, 0, 1, 0]


CREATE = r"""
import ctypes
import exact_diagonalization_for_fermionic_systems_with_gpu_gb300 as ed
from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L

calls = ctypes.CDLL(None).malloc_calls

def made(t):
    n = calls()
    op = ed.Hubbard(ed.H_TBq(12, 3).extend(t), ed.H_TBq(12, 4).extend(t), 2.0)
    return calls() - n

made(L.chain(12))
many = made(L.lieb12([1.0 + 0.1 * i for i in range(12)]))
two = made(L.chain(12) + [("H", i, (i + 2) % 12, -0.5, 0.0) for i in range(12)])
print(two - many, made(L.kagome12(flux=0.3)) - many)
"""


def test_operator_uploads_the_tables_it_uses(ed, tmp_path):
    """Beyond what every operator has: four segment tables for a few real
    classes, one class schedule for complex ones."""
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    so = tmp_path / "count_malloc.so"
    subprocess.run([cc, "-shared", "-fPIC", "-O1", str(ROOT / "tests/cpp/count_malloc.c"), "-o", str(so), "-ldl"],
                   check=True)
    r = subprocess.run([sys.executable, "-c", CREATE], env=dict(os.environ, PYTHONPATH=PYPATH, LD_PRELOAD=str(so)),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert [int(v) for v in r.stdout.split()] == [4, 1]
