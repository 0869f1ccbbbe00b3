"""The row-pair matvec (sectors whose tables leave the row engine no shared
memory) against the generic kernel, bit for bit: the same exact integer sums."""
import numpy as np
import pytest

from conftest import philox_uniform

pytestmark = pytest.mark.gpu


def pair_cases():
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    eps = list(philox_uniform(31, 9, 3.0))
    open9 = L.chain(9, periodic=False, eps=eps)
    half = [(k, i, j, v * (0.5 if k == "H" else 1.0), p) for k, i, j, v, p in open9]
    return [
        # even rows, one sign; odd rows; more down columns than a block, fewer than a lane pair
        ("open_even", 9, 4, 4, open9, open9, 2.0),
        ("open_odd_up", 9, 3, 4, L.chain(9), L.chain(9), 1.0),
        ("odd_columns", 7, 3, 4, L.chain(7), L.chain(7), 1.0),
        ("mixed_signs", 10, 5, 5, L.chain(10), L.chain(10), 4.0),
        ("kagome", 12, 2, 5, L.kagome12(), L.kagome12(), 8.0),
        ("half_hop", 9, 4, 5, half, half, 2.0),
        ("two_hops", 9, 4, 5, open9, half, 2.0),
        ("two_hops_odd", 7, 2, 3, [t for t in half if t[1] < 6 and t[2] < 6], L.chain(7), 2.0),
        ("no_down_hops", 9, 4, 4, open9, [("N", i, 0, eps[i], 0.0) for i in range(9)], 2.0),
        ("no_up_hops", 9, 0, 4, open9, open9, 2.0),
        ("one_column", 9, 4, 9, open9, open9, 2.0),
        ("two_columns", 2, 1, 1, L.chain(2, periodic=False), L.chain(2, periodic=False), 3.0),
        ("chain14", 14, 3, 7, L.chain(14, periodic=False), L.chain(14, periodic=False), 1.0),
        ("chain14_odd", 14, 4, 6, L.chain(14), L.chain(14), 1.0),
        ("chain16", 16, 2, 8, L.chain(16), L.chain(16), 1.0),
    ]


@pytest.mark.parametrize("case", pair_cases(), ids=lambda c: c[0])
def test_pair_matvec_matches_generic(ed, monkeypatch, case):
    import torch
    _, N, qu, qd, ut, dt, U = case
    ops = {}
    for kind in ("pair", "generic"):
        monkeypatch.setenv("ED_MATVEC", kind)
        ops[kind] = ed.Hubbard(ed.H_TBq(N, qu).extend(ut), ed.H_TBq(N, qd).extend(dt), U)
    monkeypatch.delenv("ED_MATVEC")
    n = ops["pair"].rows()
    x = torch.from_numpy(np.random.default_rng(3).standard_normal(n + 1)).cuda()
    ys = {}
    for k, op in ops.items():
        y = torch.full((n + 2,), 7.0, dtype=torch.float64, device="cuda")
        op.Hubbard_mv(x[1:], y[1:n + 1])  # from and to odd doubles
        z = torch.empty(n, dtype=torch.float64, device="cuda")
        op.Hubbard_mv(x[:n].clone(), z)
        assert float(y[0]) == 7.0 and float(y[n + 1]) == 7.0
        ys[k] = (y.cpu().numpy(), z.cpu().numpy())
    assert np.array_equal(ys["pair"][0], ys["generic"][0])
    assert np.array_equal(ys["pair"][1], ys["generic"][1])
    runs = {}
    for k, op in ops.items():
        lz = ed.Lanczos()
        e, v = lz.eigen(op, max_steps=min(20, n), mode="fixed", seed=4)
        runs[k] = (e, lz.a, lz.b, lz.result.min_bits, lz.result.status), v
        op.close()
    assert runs["pair"][0] == runs["generic"][0]
    assert np.array_equal(runs["pair"][1], runs["generic"][1])


# several row pairs a block: fewer 64-column units than computing warps, a
# remainder of units carried from pair to pair, and rows too long for two
# pairs in shared memory (even and odd)
@pytest.mark.parametrize("N,qu,qd", [(12, 6, 2), (13, 6, 4), (14, 6, 7), (15, 4, 6), (16, 4, 8), (23, 3, 4)])
def test_pair_matvec_many_pairs_a_block(ed, monkeypatch, N, qu, qd):
    import torch
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    terms = L.chain(N, periodic=N % 2 == 1)
    ops = {}
    for kind in ("pair", "generic"):
        monkeypatch.setenv("ED_MATVEC", kind)
        ops[kind] = ed.Hubbard(ed.H_TBq(N, qu).extend(terms), ed.H_TBq(N, qd).extend(terms), 2.0)
    n = ops["pair"].rows()
    x = torch.from_numpy(np.random.default_rng(6).standard_normal(n)).cuda()
    ys, runs = {}, {}
    for k, op in ops.items():
        y = torch.empty(n, dtype=torch.float64, device="cuda")
        op.Hubbard_mv(x, y)
        ys[k] = y
        lz = ed.Lanczos()
        e, v = lz.eigen(op, max_steps=5, mode="fixed", seed=2)
        runs[k] = (e, lz.a, lz.b, lz.result.min_bits, lz.result.status), v
    assert torch.equal(ys["pair"], ys["generic"])
    assert runs["pair"][0] == runs["generic"][0]
    assert np.array_equal(runs["pair"][1], runs["generic"][1])
    for op in ops.values():
        op.close()


# sectors that have row-engine tables too: the row-pair kernel by size; the
# persistent row kernel (forced) and the generic one give the same bits
@pytest.mark.parametrize("N,qu,qd", [(13, 5, 6), (13, 6, 7), (14, 5, 5), (15, 5, 4), (16, 6, 3)])
def test_pair_chosen_by_size(ed, monkeypatch, N, qu, qd):
    import torch
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    terms = L.chain(N, eps=list(philox_uniform(5, N, 2.0)))
    up, dn = ed.H_TBq(N, qu).extend(terms), ed.H_TBq(N, qd).extend(terms)
    op = ed.Hubbard(up, dn, 2.0)
    monkeypatch.setenv("ED_MATVEC", "generic")
    ref = ed.Hubbard(up, dn, 2.0)
    monkeypatch.delenv("ED_MATVEC")
    assert op.matvec_kind == "rows" and ref.matvec_kind == "generic"
    x = torch.from_numpy(np.random.default_rng(7).standard_normal(op.rows())).cuda()
    ys = [torch.empty_like(x) for _ in range(2)]
    op.Hubbard_mv(x, ys[0])
    ref.Hubbard_mv(x, ys[1])
    assert torch.equal(ys[0], ys[1])
    runs = []
    for o, fused in ((op, None), (op, "1"), (ref, None)):  # two launches a step; one; two
        if fused:
            monkeypatch.setenv("ED_LZ_FUSED", fused)
        lz = ed.Lanczos()
        e, v = lz.eigen(o, max_steps=6, mode="fixed", seed=3)
        monkeypatch.delenv("ED_LZ_FUSED", raising=False)
        assert lz.result.launches >= 12 if fused is None else lz.result.launches < 12
        runs.append(((e, lz.a, lz.b, lz.result.min_bits, lz.result.status), v))
    for r in runs[1:]:
        assert r[0] == runs[0][0]
        assert np.array_equal(r[1], runs[0][1])
    op.close()
    ref.close()


def test_operators_say_whether_they_run_row_pairs(ed, monkeypatch):
    """row_pairs: true for every operator the tests above force onto the pairs (so
    that they compare two kernels) and for those the size rule sends there, false
    for the generic kernel, small, complex, multi-class and two-pass ones."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    def op(N, qu, qd, ut, dt=None):
        return ed.Hubbard(ed.H_TBq(N, qu).extend(ut), ed.H_TBq(N, qd).extend(ut if dt is None else dt), 2.0)
    forced = [c[1:6] for c in pair_cases()] + [(N, qu, qd, L.chain(N, periodic=N % 2 == 1), None) for N, qu, qd in
                                               ((12, 6, 2), (13, 6, 4), (14, 6, 7), (15, 4, 6), (16, 4, 8), (23, 3, 4))]
    for N, qu, qd, ut, dt in forced:
        for kind in ("pair", "generic"):
            monkeypatch.setenv("ED_MATVEC", kind)
            o = op(N, qu, qd, ut, dt)
            assert o.row_pairs == (kind == "pair"), (N, qu, qd, kind)
            o.close()
    monkeypatch.delenv("ED_MATVEC")
    by_size = [(13, 5, 6), (13, 6, 7), (14, 5, 5), (15, 5, 4), (16, 6, 3), (14, 3, 7), (16, 2, 8)]
    others = [(12, 6, 6, L.kagome12()), (12, 6, 6, L.kagome12(flux=0.2)), (13, 5, 6, L.chain(13) + [("H", 0, 2, -0.5, 0.0)]),
              (18, 1, 9, L.lieb18())]
    for N, qu, qd, t in [(*k, L.chain(k[0])) for k in by_size] + others:
        o = op(N, qu, qd, t)
        assert o.row_pairs == ((N, qu, qd) in by_size and len(t) == N), (N, qu, qd, o.matvec_kind)
        o.close()
