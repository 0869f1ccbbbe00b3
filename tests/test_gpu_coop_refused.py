"""Cooperative launches that the device refuses (a context with part of its SMs):
the calls that make them fall back to kernels that need no resident grid, with
the same bits.  The refusal comes from a stand-in for the runtime's launch
function (tests/cpp/refuse_coop.c) in a child process; nothing is launched."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
PYPATH = os.pathsep.join([str(ROOT)] + ([os.environ["PYTHONPATH"]] if os.environ.get("PYTHONPATH") else []))

CHILD = r"""
import sys
import numpy as np
import torch
import exact_diagonalization_for_fermionic_systems_with_gpu_gb300 as ed
from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L

def op(N, u, d, t, U=2.0):
    return ed.Hubbard(ed.H_TBq(N, u).extend(t), ed.H_TBq(N, d).extend(t), U)

what, out, res = sys.argv[1], sys.argv[2], {}
if what == "apply":
    rand = list(1.0 + 0.3 * np.random.default_rng(2).standard_normal(12))
    two = L.chain(9) + [("H", i, (i + 2) % 9, -0.4, 0.0) for i in range(9)]
    for name, o in (("chain", op(8, 4, 4, L.chain(8))), ("kagome", op(12, 5, 6, L.kagome12())),
                    ("flux", op(12, 3, 4, L.kagome12(flux=0.4))), ("classes", op(9, 4, 5, two)),
                    ("random", op(12, 4, 4, L.lieb12(rand)))):
        rng = np.random.default_rng(3)
        x = rng.standard_normal(o.rows()) + (1j * rng.standard_normal(o.rows()) if o.is_complex else 0.0)
        xd = torch.from_numpy(x).cuda()
        y = torch.empty_like(xd)
        o.Hubbard_mv(xd, y)
        res[name] = y.cpu().numpy()
        res[name + "_host"] = o.matvec(x)
        for form, kw in (("run", {}), ("reorth", {"reorth": True})):
            lz = ed.Lanczos()
            e, v = lz.eigen(o, max_steps=12, mode="fixed", seed=1, **kw)
            res[f"{name}_{form}"] = np.concatenate([[e], lz.a, lz.b])
            res[f"{name}_{form}_v"] = v
else:
    for N, u, d, B in ((9, 4, 3, 2), (10, 5, 5, 8)):
        ops = [op(N, u, d, L.chain(N, eps=list(0.1 * (b + 1) * np.arange(N))), 1.0 + b) for b in range(B)]
        starts = np.random.default_rng(5).standard_normal((B, ops[0].rows()))
        for name, s in (("seed", None), ("user", starts)):
            e, v, a, b = ed.lanczos_batch(ops, 15, seed=4, starts=s)
            for k, r in zip("evab", (e, v, a, b)):
                res[f"{N}_{name}_{k}"] = r
np.savez(out, **res)
"""


def run(tmp_path, what, refuse):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    so = tmp_path / "refuse_coop.so"
    subprocess.run([cc, "-shared", "-fPIC", "-O1", str(ROOT / "tests/cpp/refuse_coop.c"), "-o", str(so), "-ldl"],
                   check=True)
    got = {}
    for form in ("refused", "plain"):
        out = tmp_path / f"{form}.npz"
        env = dict(os.environ, PYTHONPATH=PYPATH, LD_PRELOAD=str(so))
        if form == "refused":
            env["REFUSE_COOP"] = str(refuse)
        r = subprocess.run([sys.executable, "-c", CHILD, what, str(out)], env=env, capture_output=True, text=True)
        assert r.returncode == 0, (form, r.stderr)
        got[form] = np.load(out)
    assert got["refused"].files == got["plain"].files
    for k in got["plain"].files:
        assert np.array_equal(got["refused"][k], got["plain"][k]), k


def test_apply_without_cooperative_launch(ed, tmp_path):
    run(tmp_path, "apply", 1)


def test_batch_without_its_own_grid(ed, tmp_path):
    """The batch kernel's blocks of 1,024 threads refused: k_lz_multi, whose
    blocks are smaller."""
    run(tmp_path, "batch", 1024)
