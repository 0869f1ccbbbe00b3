"""The one-launch FP64 apply (exponent pass, conversion and rows in one
cooperative kernel) against the generic kernels' three launches, bit for bit:
the same exact integer sums from the same fixed-point copy of x."""
import numpy as np
import pytest

from conftest import philox_uniform

pytestmark = pytest.mark.gpu


def apply_cases():
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    r = list(philox_uniform(4, 12, 0.5) + 1.0)
    return [
        # units below and above the grid, odd rows, one row, every row-engine variant
        ("ring4", 4, 2, 2, L.chain(4), 1.0),
        ("ring8", 8, 4, 4, L.chain(8), 4.0),
        ("ring7_odd", 7, 3, 2, L.chain(7), 2.0),
        ("one_row", 9, 0, 4, L.chain(9), 2.0),
        ("one_state", 6, 6, 6, L.chain(6), 2.0),
        ("kagome12_66", 12, 6, 6, L.kagome12(), 8.0),
        ("kagome12_84_odd", 12, 8, 4, L.kagome12(), 8.0),
        ("no_schedule", 10, 5, 5, L.chain(10), 1.0),
        ("lieb12_classes", 12, 5, 6, L.lieb12(r), 4.0),
        ("kagome12_two_classes", 12, 4, 5, [(k, i, j, v * (1.0 if i % 2 else 0.5), p) for k, i, j, v, p in L.kagome12()], 2.0),
        ("flux", 12, 4, 6, L.kagome12(flux=0.3, peierls=True), 4.0),
        ("flux_one_class", 8, 3, 4, [("P", i, (i + 1) % 8, -1.0, 0.0) for i in range(8)], 4.0),
    ]


@pytest.mark.parametrize("case", apply_cases(), ids=lambda c: c[0])
def test_one_launch_apply_matches_generic(ed, monkeypatch, case):
    import torch
    name, N, qu, qd, t, U = case
    ops = {}
    for kind in ("auto", "generic"):
        if kind == "generic":
            monkeypatch.setenv("ED_MATVEC", "generic")
        elif name == "no_schedule":
            monkeypatch.setenv("ED_NO_SCHED", "1")
        ops[kind] = ed.Hubbard(ed.H_TBq(N, qu).extend(t), ed.H_TBq(N, qd).extend(t), U)
        monkeypatch.delenv("ED_MATVEC", raising=False)
        monkeypatch.delenv("ED_NO_SCHED", raising=False)
    n = ops["auto"].rows()
    rng = np.random.default_rng(5)
    dt = torch.complex128 if ops["auto"].is_complex else torch.float64
    for scale in (1.0, 1e-200, 0.0, 3e150):  # a new exponent on every call
        x = rng.standard_normal(n) + (1j * rng.standard_normal(n) if ops["auto"].is_complex else 0.0)
        xd = torch.from_numpy(x * scale).to(dt).cuda()
        ys = []
        for op in ops.values():
            y = torch.empty(n, dtype=dt, device="cuda")
            op.Hubbard_mv(xd, y)
            ys.append(y)
        assert torch.equal(ys[0], ys[1]), scale
    with pytest.raises(Exception):
        bad = np.full(n, np.nan, dtype=np.complex128 if ops["auto"].is_complex else np.float64)
        ops["auto"].matvec(bad)
    good = ops["auto"].matvec(x)
    assert np.array_equal(good, ops["generic"].matvec(x))


def test_one_launch_apply_in_a_graph(ed):
    """Captured once and replayed on new values of x, on a side stream."""
    import torch
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    op = ed.Hubbard(ed.H_TBq(8, 4).extend(L.chain(8)), ed.H_TBq(8, 4).extend(L.chain(8)), 4.0)
    x = torch.zeros(op.rows(), dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        op.Hubbard_mv(x, y)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        op.Hubbard_mv(x, y)
    for seed in range(3):
        v = np.random.default_rng(seed).standard_normal(op.rows()) * 10.0 ** seed
        x.copy_(torch.from_numpy(v))
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), op.matvec(v))


@pytest.mark.parametrize("case", ["lieb_random", "kagome_random_flux", "kagome_random_odd", "few_classes", "one_up_hop"])
def test_entry_products_match_generic(ed, monkeypatch, case):
    """Tables with a coefficient per bond (a product per entry, in the apply,
    the per-step, the persistent and the mixed batched kernels) and tables
    whose rows hold several entries of a class (class sums), against the
    generic kernel bit for bit."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    r = list(philox_uniform(14, 12, 0.5) + 1.0)
    N, qu, qd, t = 12, 5, 4, L.lieb12(r)
    if case == "kagome_random_flux":
        qu, qd, t = 3, 4, L.kagome12(r, flux=0.4)
    elif case == "kagome_random_odd":
        qu, qd, t = 2, 8, L.kagome12(r)
    elif case == "few_classes":  # five amplitudes on 24 bonds
        t = [(k, i, j, v * (1.0 + 0.25 * (b % 5)), p) for b, (k, i, j, v, p) in enumerate(L.kagome12())]
    elif case == "one_up_hop":
        qu, qd = 12, 5
    ops = {}
    for kind in ("auto", "generic"):
        if kind == "generic":
            monkeypatch.setenv("ED_MATVEC", "generic")
        ops[kind] = ed.Hubbard(ed.H_TBq(N, qu).extend(t), ed.H_TBq(N, qd).extend(t), 4.0)
        monkeypatch.delenv("ED_MATVEC", raising=False)
    n = ops["auto"].rows()
    x = np.random.default_rng(8).standard_normal(n)
    x = x + 1j * x[::-1] if ops["auto"].is_complex else x
    assert np.array_equal(ops["auto"].matvec(x), ops["generic"].matvec(x))
    runs = []
    for kind, form in (("generic", "0"), ("auto", "0"), ("auto", "1")):
        monkeypatch.setenv("ED_LZ_FUSED", form)
        lz = ed.Lanczos()
        e, v = lz.eigen(ops[kind], max_steps=25, mode="fixed", seed=6)
        runs.append((e, lz.a, lz.b, v))
    monkeypatch.delenv("ED_LZ_FUSED")
    chain = ed.Hubbard(ed.H_TBq(8, 4).extend(L.chain(8)), ed.H_TBq(8, 4).extend(L.chain(8)), 1.0)
    e, vs, al, be = ed.lanczos_multi([chain, ops["auto"]], 25, seed=5)  # run 1 from seed 6
    runs.append((e[1], list(al[1]), list(be[1]), vs[1]))
    for other in runs[1:]:
        assert other[:3] == runs[0][:3]
        assert np.array_equal(other[3], runs[0][3])


@pytest.mark.parametrize("case", ["pairs", "pairs_odd", "real_class", "imaginary", "unequal_spins", "no_down_hops", "one_row"])
def test_complex_class_sums_match_generic(ed, monkeypatch, case):
    """Complex operators of at most four classes (class sums, conjugate classes
    sharing their products) in the apply, per-step, persistent and batched
    kernels against the generic kernel bit for bit."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    import math
    ring = lambda n, v, ph: [("P", i, (i + 1) % n, v, ph) for i in range(n)]  # noqa: E731
    N, qu, qd, U = 9, 4, 3, 2.0
    tu = td = ring(9, -1.0, 0.3) + [("P", i, (i + 2) % 9, 0.5, 0.6) for i in range(9)]
    if case == "pairs_odd":
        N, qu, qd = 7, 3, 2
        tu = td = ring(7, -1.0, 0.3) + [("P", i, (i + 2) % 7, 0.5, 0.6) for i in range(7)]
    elif case == "real_class":
        tu = td = ring(9, -1.0, 0.3) + [("P", 0, 4, 0.7, 0.0)]
    elif case == "imaginary":
        tu = td = ring(9, 1.0, math.pi / 2) + [("P", 0, 4, 0.7, 0.2)]
    elif case == "unequal_spins":
        td = ring(9, -0.25, 0.1)
    elif case == "no_down_hops":
        td = [("N", i, 0, 0.1 * i, 0.0) for i in range(9)]
    elif case == "one_row":
        qu = 9
    ops = {}
    for kind in ("auto", "generic"):
        if kind == "generic":
            monkeypatch.setenv("ED_MATVEC", "generic")
        ops[kind] = ed.Hubbard(ed.H_TBq(N, qu).extend(tu), ed.H_TBq(N, qd).extend(td), U)
        monkeypatch.delenv("ED_MATVEC", raising=False)
    n = ops["auto"].rows()
    rng = np.random.default_rng(8)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    assert np.array_equal(ops["auto"].matvec(x), ops["generic"].matvec(x))
    runs = []
    for kind, form in (("generic", "0"), ("auto", "0"), ("auto", "1")):
        monkeypatch.setenv("ED_LZ_FUSED", form)
        lz = ed.Lanczos()
        e, v = lz.eigen(ops[kind], max_steps=20, mode="fixed", seed=6)
        runs.append((e, lz.a, lz.b, v))
    monkeypatch.delenv("ED_LZ_FUSED")
    chain = ed.Hubbard(ed.H_TBq(8, 4).extend(L.chain(8)), ed.H_TBq(8, 4).extend(L.chain(8)), 1.0)
    e, vs, al, be = ed.lanczos_multi([chain, ops["auto"]], 20, seed=5)  # run 1 from seed 6
    runs.append((e[1], list(al[1]), list(be[1]), vs[1]))
    for other in runs[1:]:
        assert other[:3] == runs[0][:3]
        assert np.array_equal(other[3], runs[0][3])


# the last rows of the unit queue split into two or four column ranges, and
# whole where their ranges would be narrow or more than the grid: apply and
# persistent Lanczos against the generic kernel
@pytest.mark.parametrize("N,qu,qd,flux", [(12, 2, 6, 0.3), (12, 2, 4, 0.3), (12, 6, 6, 0.3), (12, 4, 6, 0.3), (8, 4, 4, 0.2),
                                          (12, 2, 6, 0.0), (13, 2, 4, 0.0), (11, 4, 4, 0.0), (10, 6, 3, 0.0)])
def test_split_rows_match_generic(ed, monkeypatch, N, qu, qd, flux):
    import torch
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    if flux and N == 12:
        t = L.kagome12(flux=flux, peierls=True)
    else:
        t = [("P" if flux else "H", i, (i + 1) % N, -1.0, flux) for i in range(N)]
    up, dn = ed.H_TBq(N, qu).extend(t), ed.H_TBq(N, qd).extend(t)
    ops = [ed.Hubbard(up, dn, 4.0)]
    monkeypatch.setenv("ED_MATVEC", "generic")
    ops.append(ed.Hubbard(up, dn, 4.0))
    monkeypatch.delenv("ED_MATVEC")
    assert [op.matvec_kind for op in ops] == ["rows", "generic"]
    n = ops[0].rows()
    dt = torch.complex128 if flux else torch.float64
    x = torch.from_numpy(np.random.default_rng(8).standard_normal(n)).to(dt).cuda()
    x *= (1.0 - 2.0j) if flux else 1.0
    ys, runs = [], []
    for op in ops:
        y = torch.empty_like(x)
        op.Hubbard_mv(x, y)
        ys.append(y)
        lz = ed.Lanczos()
        e, v = lz.eigen(op, max_steps=12, mode="fixed", seed=2)
        runs.append(((e, lz.a, lz.b, lz.result.min_bits, lz.result.status), v))
        op.close()
    assert torch.equal(ys[0], ys[1])
    assert runs[0][0] == runs[1][0]
    assert np.array_equal(runs[0][1], runs[1][1])
