"""GPU Lanczos (device recurrence, device tridiagonal eigensolve, Ritz
vector) against the oracle and the golden energies.

Tolerances: E0 to 1e-10 relative (the reference's stop test targets
0.01*sqrt(eps)); Ritz vectors through their residual |Hv - E0 v| and the
entanglement entropy to 1e-8.
"""
import numpy as np
import pytest

from conftest import philox_uniform, rel_err

pytestmark = pytest.mark.gpu


def op_for(ed, N, qu, qd, terms_u, terms_d, U):
    return ed.Hubbard(ed.H_TBq(N, qu).extend(terms_u), ed.H_TBq(N, qd).extend(terms_d), U)


def test_chain8_fixed100_reorth(ed, orc, golden_energies):
    """Plain small config: L=8 PBC, 4+4, U=4, 100 steps with full
    reorthogonalisation, start vector Philox(seed 0); E0 and the half-chain
    entanglement entropy of the Ritz vector."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    g = golden_energies["chain8_pbc_q44_U4"]
    op = op_for(ed, 8, 4, 4, L.chain(8), L.chain(8), 4.0)
    lz = ed.Lanczos(op.dimUP, op.dimDN)
    e0, v = lz.eigen(op, max_steps=100, mode="fixed", reorth=True, seed=0)
    assert abs(e0 - g["E0"]) < 1e-10 * abs(g["E0"]), e0 - g["E0"]
    assert abs(np.linalg.norm(v) - 1.0) < 1e-12
    r = op.matvec(v) - e0 * v
    assert np.linalg.norm(r) < 1e-7
    s_vn, s_ref = orc.entanglement_entropy(v, 8, 4, 4, [0, 1, 2, 3])
    assert abs(s_vn - g["EE_vN_A0123"]) < 1e-8
    assert abs(s_ref - g["EE_ref_A0123"]) < 1e-8 * abs(g["EE_ref_A0123"])


def test_reference_mode_matches_oracle(ed, orc, golden_energies):
    """Same start vector, the reference stop test (every 10 steps,
    tolconv = 0.01 sqrt(eps)): the same number of steps, T to 1e-10 and E0."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    op = op_for(ed, 8, 4, 4, L.chain(8), L.chain(8), 4.0)
    t = orc.Tables(8, 4, L.chain(8))
    f = philox_uniform(235, op.rows())
    e_o, a_o, b_o, v_o = orc.lanczos(t, t, 4.0, f, 1000, mode="reference")
    lz = ed.Lanczos(op.dimUP, op.dimDN)
    e0, v = lz.eigen(op, f=f, max_steps=1000, mode="reference")
    assert lz.result.converged == 1
    assert len(lz.a) == len(a_o)
    k = min(30, len(a_o))
    assert np.max(np.abs(np.array(lz.a[:k]) - a_o[:k])) < 1e-10
    assert np.max(np.abs(np.array(lz.b[:k]) - b_o[:k])) < 1e-10
    assert abs(e0 - e_o) < 1e-10 * abs(e_o)
    assert abs(abs(v @ v_o) - 1.0) < 1e-8


def test_reference_mode_kagome12_one_launch(ed, golden_energies, monkeypatch):
    """The reference stop test on Kagome12 6+6, U=8: the persistent kernel
    runs every step in one launch while the host tests T every ten steps on
    the mirrored alpha and beta, and the launch stops a few steps after the
    test passes.  Against the per-step kernels, which stop at the test's
    step with a host round trip every ten steps: the same step count, alpha,
    beta and E0 bit for bit; the golden E0 to 1e-10; six kernel launches in
    all (start vector three, one persistent, Ritz sum two)."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    g = golden_energies["kagome12_q66_U8"]["E0"]
    op = op_for(ed, 12, 6, 6, L.kagome12(), L.kagome12(), 8.0)
    lz = ed.Lanczos()
    e0, v = lz.eigen(op, max_steps=1000, mode="reference", seed=4)
    assert lz.result.converged == 1 and lz.result.steps % 10 == 0
    assert lz.result.launches == 6, lz.result.launches
    assert lz.result.n_matvec >= lz.result.steps
    assert abs(e0 - g) < 1e-10 * abs(g)
    monkeypatch.setenv("ED_LZ_FUSED", "0")
    lz2 = ed.Lanczos()
    e2, v2 = lz2.eigen(op, max_steps=1000, mode="reference", seed=4)
    assert lz2.result.steps == lz.result.steps and lz2.result.n_matvec == lz2.result.steps
    assert lz2.a == lz.a and lz2.b == lz.b and e2 == e0
    assert np.array_equal(v2, v)


def test_kagome12_300_steps(ed, golden_energies):
    """Kagome 12-site, 6+6, U=8, 300 fixed steps: E0 to 1e-10 and the Ritz vector."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    g = golden_energies["kagome12_q66_U8"]
    op = op_for(ed, 12, 6, 6, L.kagome12(), L.kagome12(), 8.0)
    lz = ed.Lanczos(op.dimUP, op.dimDN)
    e0, v = lz.eigen(op, max_steps=300, mode="fixed", seed=0)
    assert abs(e0 - g["E0"]) < 1e-10 * abs(g["E0"]), e0 - g["E0"]
    assert np.linalg.norm(op.matvec(v) - e0 * v) < 1e-6
    assert lz.result.min_bits >= 44


@pytest.mark.parametrize("sector", [(6, 6), (7, 5), (8, 4)])
def test_mbl_chain12_sectors(ed, orc, golden_energies, sector):
    """MBL chain L=12, W=6, U=1, three sectors.  Fixed 300 steps: E0 and both
    entropies to 1e-8.  The reference stop test (mode='reference') stops once
    the residual is ~1e-9 |H|, which bounds the Ritz vector's accuracy: the
    reference formula -sum s ln s amplifies errors of tiny singular values
    (d/ds = ln s + 1), so there it is held to 1e-7."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    qu, qd = sector
    g = golden_energies[f"chain12_open_W6_seed100_q{qu}{qd}_U1"]
    terms = L.chain(12, periodic=False, eps=g["eps"])
    op = op_for(ed, 12, qu, qd, terms, terms, 1.0)
    e0, v = ed.Lanczos(op.dimUP, op.dimDN).eigen(op, max_steps=300, mode="fixed", seed=3)
    assert abs(e0 - g["E0"]) < 1e-10 * abs(g["E0"])
    s_vn, s_ref = orc.entanglement_entropy(v, 12, qu, qd, list(range(6)))
    assert abs(s_vn - g["EE_vN_A0to5"]) < 1e-8
    assert abs(s_ref - g["EE_ref_A0to5"]) < 1e-8 * max(1.0, abs(g["EE_ref_A0to5"]))
    e0, v = ed.Lanczos(op.dimUP, op.dimDN).eigen(op, max_steps=1000, mode="reference", seed=3)
    assert abs(e0 - g["E0"]) < 1e-10 * abs(g["E0"])
    s_vn, s_ref = orc.entanglement_entropy(v, 12, qu, qd, list(range(6)))
    assert abs(s_vn - g["EE_vN_A0to5"]) < 1e-8
    assert abs(s_ref - g["EE_ref_A0to5"]) < 1e-7 * max(1.0, abs(g["EE_ref_A0to5"]))


def test_lieb12(ed, golden_energies):
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    g = golden_energies["lieb12_q66_U4"]
    op = op_for(ed, 12, 6, 6, L.lieb12(), L.lieb12(), 4.0)
    e0, _ = ed.Lanczos().eigen(op, max_steps=1000, mode="reference", ritz="none", seed=1)
    assert abs(e0 - g["E0"]) < 1e-10 * abs(g["E0"])


def test_atomic_limit_diagonal_operator(ed, orc, golden_energies):
    """No hopping (a diagonal H with a degenerate ground level): 120 steps
    reach the closed-form E0; at 60 steps the (unconverged) E0 equals the
    oracle's Lanczos on the same start vector."""
    g = golden_energies["atomic8_q32_U3"]
    eps = g["eps"]
    terms = [("N", i, 0, eps[i], 0.0) for i in range(8)]
    op = op_for(ed, 8, 3, 2, terms, terms, 3.0)
    e0, _ = ed.Lanczos().eigen(op, max_steps=120, mode="fixed", ritz="none", seed=2)
    assert abs(e0 - g["E0"]) < 1e-10 * max(1.0, abs(g["E0"]))
    e60, _ = ed.Lanczos().eigen(op, max_steps=60, mode="fixed", ritz="none", seed=2)
    f = philox_uniform(2, op.rows())
    e60_o = orc.lanczos(orc.Tables(8, 3, terms), orc.Tables(8, 2, terms), 3.0, f, 60, mode="fixed",
                        want_evec=False)[0]
    assert abs(e60 - e60_o) < 1e-10 * abs(e60_o)


def test_complex_peierls_lanczos(ed, orc):
    """Complex (twisted) operator: E0 from the device Lanczos equals scipy."""
    import scipy.sparse.linalg as sla
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    terms = L.kagome12(flux=0.4)
    op = op_for(ed, 12, 5, 4, terms, terms, 4.0)
    H = orc.hamiltonian(12, 5, 4, terms, terms, 4.0)
    w = sla.eigsh(H, k=1, which="SA", tol=1e-13)[0][0]
    e0, v = ed.Lanczos().eigen(op, max_steps=1000, mode="reference", seed=5)
    assert abs(e0 - w) < 1e-10 * abs(w)
    assert np.linalg.norm(H @ v - e0 * v) < 1e-6


def test_start_vector_user_vs_random_same(ed):
    """ED_START_RANDOM(seed) is exactly the Philox vector a caller would pass."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    op = op_for(ed, 8, 4, 4, L.chain(8), L.chain(8), 4.0)
    lz1, lz2 = ed.Lanczos(), ed.Lanczos()
    e1, _ = lz1.eigen(op, max_steps=40, mode="fixed", ritz="none", seed=9)
    e2, _ = lz2.eigen(op, f=philox_uniform(9, op.rows()), max_steps=40, mode="fixed", ritz="none")
    assert lz1.a == lz2.a and lz1.b == lz2.b and e1 == e2


def test_lanczos_profile_and_launch_count(ed):
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L, _capi
    import ctypes as C
    op = op_for(ed, 12, 6, 6, L.kagome12(), L.kagome12(), 8.0)
    lib = _capi.load()
    cfg = _capi.ed_lanczos_cfg(max_steps=50, mode=1, reorth=0, ritz=1, start=0, profile=1, seed=0)
    res = _capi.ed_lanczos_result()
    v = np.empty(op.rows())
    assert lib.ed_lanczos_run(op.handle, C.byref(cfg), None, 0, C.c_void_p(v.ctypes.data), 0, None, None,
                              C.byref(res), None) == 0
    assert res.n_matvec == 50 and res.matvec_ms > 0 and res.axpy_ms > 0
    assert res.launches == 3 + 2 * 50 + 2


def fused_cases():
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    eps12 = list(philox_uniform(100, 12, 6.0))
    return [
        ("kagome12_66_U8_fixed300_ritz", 12, 6, 6, L.kagome12(), L.kagome12(), 8.0, "fixed", 300, "stored"),
        ("kagome12_66_U8_reference", 12, 6, 6, L.kagome12(), L.kagome12(), 8.0, "reference", 1000, "stored"),
        ("kagome12_54_flux_complex", 12, 5, 4, L.kagome12(flux=0.3), L.kagome12(flux=0.3), 4.0, "fixed", 80,
         "stored"),
        ("kagome12_55_Kx_2classes", 12, 5, 5, L.kagome12_kinetic_x(), L.kagome12_kinetic_x(), 1.0, "fixed", 60,
         "none"),
        ("chain12_open_W6_66_three_slots", 12, 6, 6, L.chain(12, periodic=False, eps=eps12),
         L.chain(12, periodic=False, eps=eps12), 1.0, "fixed", 120, "none"),
        ("chain2_11_breakdown", 2, 1, 1, L.chain(2, periodic=False), L.chain(2, periodic=False), 3.0, "fixed", 12,
         "stored"),
    ]


@pytest.mark.parametrize("case", fused_cases(), ids=lambda c: c[0])
def test_persistent_kernel_matches_per_step_kernels(ed, monkeypatch, case):
    """The persistent Lanczos kernel (all steps in one cooperative launch)
    and the per-step kernels (a matvec and an axpy launch per step) perform
    the same exact integer reductions and the same scalar arithmetic: alpha,
    beta, E0 and the Ritz vector agree bit for bit, also past a breakdown and
    with the three-slot (no stored basis) recurrence."""
    name, N, qu, qd, tu, td, U, mode, steps, ritz = case
    op = op_for(ed, N, qu, qd, tu, td, U)
    runs = {}
    for fused in ("1", "0"):
        monkeypatch.setenv("ED_LZ_FUSED", fused)
        lz = ed.Lanczos()
        e0, v = lz.eigen(op, max_steps=steps, mode=mode, ritz=ritz, seed=3)
        runs[fused] = (lz.a, lz.b, e0, v, lz.result.steps, lz.result.launches)
    monkeypatch.delenv("ED_LZ_FUSED")
    f, p = runs["1"], runs["0"]
    assert f[0] == p[0] and f[1] == p[1] and f[2] == p[2] and f[4] == p[4]
    if ritz != "none":
        assert np.array_equal(f[3], p[3])
    assert f[5] < p[5]  # the persistent path launched fewer kernels


def test_persistent_kernel_launch_count(ed):
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L, _capi
    import ctypes as C
    op = op_for(ed, 12, 6, 6, L.kagome12(), L.kagome12(), 8.0)
    lib = _capi.load()
    cfg = _capi.ed_lanczos_cfg(max_steps=50, mode=1, reorth=0, ritz=1, start=0, profile=0, seed=0)
    res = _capi.ed_lanczos_result()
    v = np.empty(op.rows())
    assert lib.ed_lanczos_run(op.handle, C.byref(cfg), None, 0, C.c_void_p(v.ctypes.data), 0, None, None,
                              C.byref(res), None) == 0
    # random, emax, start; one persistent launch; Ritz sum and scale (the
    # tridiagonal eigensolve runs on the host)
    assert res.launches == 3 + 1 + 2


@pytest.mark.parametrize("case", ["kagome12_fixed", "chain8_reference", "chain12_fixed_per_step"])
def test_ritz_recompute_matches_stored(ed, monkeypatch, case):
    """ED_RITZ_RECOMPUTE (the reference's second Lanczos pass, three working
    vectors) regenerates the same Lanczos vectors bit for bit, so its Ritz
    vector equals the stored-basis sum up to the FP64 accumulation of the
    second pass (1e-12 normwise), with identical T and E0."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    if case == "kagome12_fixed":
        op, steps, mode = op_for(ed, 12, 6, 6, L.kagome12(), L.kagome12(), 8.0), 300, "fixed"
    elif case == "chain8_reference":
        op, steps, mode = op_for(ed, 8, 4, 4, L.chain(8), L.chain(8), 4.0), 1000, "reference"
    else:
        eps = list(philox_uniform(100, 12, 6.0))
        t = L.chain(12, periodic=False, eps=eps)
        op, steps, mode = op_for(ed, 12, 6, 6, t, t, 1.0), 200, "fixed"
        monkeypatch.setenv("ED_LZ_FUSED", "0")
    l1, l2 = ed.Lanczos(), ed.Lanczos()
    e1, v1 = l1.eigen(op, max_steps=steps, mode=mode, ritz="stored", seed=2)
    e2, v2 = l2.eigen(op, max_steps=steps, mode=mode, ritz="recompute", seed=2)
    assert e1 == e2 and l1.a == l2.a and l1.b == l2.b
    assert np.linalg.norm(v1 - v2) < 1e-12
    assert abs(np.linalg.norm(v2) - 1.0) < 1e-13


@pytest.mark.parametrize("ritz", ["stored", "recompute"])
def test_two_pass_matvec_lanczos_ritz_vector(ed, monkeypatch, ritz):
    """The two-pass matvec runs Lanczos in a permuted down order; start and
    Ritz vectors are permuted on the way in and out, so T, E0 and the Ritz
    vector equal the generic kernel's (the vector to its last bits: only the
    order of the FP64 norm sum differs)."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    runs = {}
    for kind in ("striped", "generic"):
        monkeypatch.setenv("ED_MATVEC", kind)
        op = op_for(ed, 12, 6, 6, L.kagome12(), L.kagome12(), 8.0)
        lz = ed.Lanczos()
        e0, v = lz.eigen(op, max_steps=150, mode="fixed", ritz=ritz, seed=5)
        runs[kind] = (lz.a, lz.b, e0, v)
        op.close()
    monkeypatch.delenv("ED_MATVEC")
    s, g = runs["striped"], runs["generic"]
    assert s[0] == g[0] and s[1] == g[1] and s[2] == g[2]
    assert np.max(np.abs(s[3] - g[3])) < 1e-15


def test_lanczos_batch_matches_single_runs(ed):
    """ed_lanczos_batch: four disorder realisations of the open L=12 (6,6)
    sector in one persistent launch give, run by run, the alpha, beta, E0 and
    Ritz vector of the run's own ed_lanczos_run bit for bit; a batch of one
    equals a single run too."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import sweeps
    ops = []
    for r in range(4):
        eu, edn = sweeps.mbl_disorder(r, 12, 6.0)
        ops.append(ed.Hubbard(ed.H_TBq(12, 6).extend(sweeps.mbl_chain_terms(eu)),
                              ed.H_TBq(12, 6).extend(sweeps.mbl_chain_terms(edn)), 1.0 + 0.5 * r))
    steps = 60
    for group in (ops, ops[2:3]):
        base = 7 if len(group) > 1 else 9
        e0, ev, al, be = ed.lanczos_batch(group, steps, seed=base)
        for b, op in enumerate(group):
            lz = ed.Lanczos()
            e, v = lz.eigen(op, max_steps=steps, mode="fixed", seed=base + b)
            assert e0[b] == e
            assert np.array_equal(al[b], np.array(lz.a)) and np.array_equal(be[b], np.array(lz.b))
            assert np.array_equal(ev[b], v)


def test_lanczos_batch_of_different_tables_runs_each_as_alone(ed):
    """Operators with different hopping tables (open and periodic chain)
    share a launch in the general batch kernel; each run equals its own."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    a = ed.Hubbard(ed.H_TBq(12, 6).extend(L.chain(12, periodic=False)), ed.H_TBq(12, 6).extend(L.chain(12, periodic=False)), 1.0)
    b = ed.Hubbard(ed.H_TBq(12, 6).extend(L.chain(12)), ed.H_TBq(12, 6).extend(L.chain(12)), 1.0)
    e0, ev, al, be = ed.lanczos_batch([a, b], 40, seed=5)
    for k, op in enumerate((a, b)):
        lz = ed.Lanczos()
        e, v = lz.eigen(op, max_steps=40, mode="fixed", seed=5 + k)
        assert e0[k] == e and np.array_equal(al[k], np.array(lz.a)) and np.array_equal(ev[k], v)


@pytest.mark.parametrize("case", ["chain12_66", "kagome12_flux"])
def test_autotune_keeps_results(ed, case):
    """ed_op_autotune times the per-step and persistent kernels (three queue
    weights, two and one CTAs per SM) and applies the fastest; the Lanczos
    coefficients afterwards are the same bit for bit, and set_tuning carries
    the choice to a second operator of the same shape."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L, sweeps
    if case == "chain12_66":
        eu, edn = sweeps.mbl_disorder(0, 12, 6.0)
        make = lambda: ed.Hubbard(ed.H_TBq(12, 6).extend(sweeps.mbl_chain_terms(eu)),
                                  ed.H_TBq(12, 6).extend(sweeps.mbl_chain_terms(edn)), 1.0)
    else:
        t = L.kagome12(flux=0.3)
        make = lambda: ed.Hubbard(ed.H_TBq(12, 6).extend(t), ed.H_TBq(12, 6).extend(t), 4.0)
    op = make()
    lz0 = ed.Lanczos()
    lz0.eigen(op, max_steps=40, mode="fixed", ritz="none", seed=3)
    info = op.autotune(steps=20)
    assert info["per_step_us"] > 0 and all(v > 0 for v in info["persistent_us"])
    # the rows-per-CTA axis: one CTA per SM timed too where the plan has two,
    # and the choice is the fastest of all
    cands = [info["per_step_us"]] + info["persistent_us"] + ([info["one_cta_us"]] if info["one_cta_us"] > 0 else [])
    assert info["candidates"] == len(cands)
    assert info["us_per_step"] == min(cands)
    assert info["ctas_per_sm"] in (1, 2) if info["persistent"] else info["ctas_per_sm"] == 0
    lz1 = ed.Lanczos()
    lz1.eigen(op, max_steps=40, mode="fixed", ritz="none", seed=3)
    assert lz1.a == lz0.a and lz1.b == lz0.b
    op2 = make()
    op2.set_tuning(info["result"])
    lz2 = ed.Lanczos()
    lz2.eigen(op2, max_steps=40, mode="fixed", ritz="none", seed=3)
    assert lz2.a == lz0.a and lz2.b == lz0.b


def test_reorth_coefficients_match_oracle(ed, orc):
    """Full reorthogonalisation with the Gram-Schmidt coefficients formed on
    the device: the first 40 alpha and beta of the L=8 (3,5) chain track the
    oracle's reorthogonalised FP64 recurrence to 1e-11 (later coefficients
    of any two implementations drift apart once Ritz values converge: each
    step amplifies rounding differences), E0 agrees with the oracle's to
    1e-12, and repeated runs are bit-identical."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    op = op_for(ed, 8, 3, 5, L.chain(8), L.chain(8), 2.0)
    f = philox_uniform(7, op.rows())
    runs = []
    for _ in range(2):
        lz = ed.Lanczos()
        e0, _ = lz.eigen(op, f=f, max_steps=100, mode="fixed", reorth=True, ritz="none")
        runs.append((e0, list(lz.a), list(lz.b)))
    assert runs[0] == runs[1]
    tu, td = orc.Tables(8, 3, L.chain(8)), orc.Tables(8, 5, L.chain(8))
    e_o, a_o, b_o, _ = orc.lanczos(tu, td, 2.0, f, 100, mode="fixed", reorth=True, want_evec=False)
    a, b = np.array(runs[0][1]), np.array(runs[0][2])
    assert np.max(np.abs(a[:40] - np.asarray(a_o)[:40])) < 1e-11 * np.max(np.abs(a_o))
    assert np.max(np.abs(b[1:40] - np.asarray(b_o)[1:40])) < 1e-11 * np.max(np.abs(b_o))
    assert abs(runs[0][0] - e_o) < 1e-12 * abs(e_o)


def test_grid_barrier_timeout_is_reported_and_operator_recovers(ed, golden_energies, monkeypatch):
    """The persistent kernel's bounded grid-barrier wait, made to run out on
    purpose: ED_GRID_WAIT="1000000,1" gives every barrier a 1 ms limit and
    makes it wait for one arrival more than the grid has, an arrival that
    never comes.  Every CTA gives up at its first barrier (no bulk copy is in
    flight there) and ed_lanczos_run returns ED_ERR_TIMEOUT; the next run on
    the same operator, without the knob, returns the golden E0."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import _capi, lattices as L
    op = op_for(ed, 12, 6, 6, L.kagome12(), L.kagome12(), 8.0)
    monkeypatch.setenv("ED_GRID_WAIT", "1000000,1")
    with pytest.raises(_capi.EdError) as ei:
        ed.Lanczos().eigen(op, max_steps=30, mode="fixed", ritz="none", seed=0)
    assert ei.value.status == _capi.ED_ERR_TIMEOUT
    monkeypatch.delenv("ED_GRID_WAIT")
    lz = ed.Lanczos()
    e0, v = lz.eigen(op, max_steps=300, mode="fixed", seed=0)
    assert lz.result.launches <= 8  # the persistent path, not the per-step kernels
    g = golden_energies["kagome12_q66_U8"]["E0"]
    assert abs(e0 - g) < 1e-10 * abs(g)
    assert np.linalg.norm(op.matvec(v) - e0 * v) < 1e-6


def test_autotune_two_pass_chunk_keeps_results(ed):
    """The two-pass matvec's pass-D window (the tuner's chunk axis) on the
    small Lieb18 case (4+9, 48,620 down columns): both chunks timed, and the
    Lanczos coefficients under the chosen one equal the untuned run's."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    t = L.lieb18()
    op = ed.Hubbard(ed.H_TBq(18, 4).extend(t), ed.H_TBq(18, 9).extend(t), 4.0)
    assert op.matvec_kind == "two_pass"
    lz0 = ed.Lanczos()
    lz0.eigen(op, max_steps=6, mode="fixed", ritz="none", seed=2)
    info = op.autotune(steps=3)
    assert info["chunk"] > 0 and all(v > 0 for v in info["chunk_us"])
    lz1 = ed.Lanczos()
    lz1.eigen(op, max_steps=6, mode="fixed", ritz="none", seed=2)
    assert lz1.a == lz0.a and lz1.b == lz0.b
    op.close()


@pytest.mark.parametrize("steps", [1, 2, 15, 16, 17, 33])
@pytest.mark.parametrize("qu,qd", [(3, 2), (3, 4), (0, 3)])
def test_ritz_sum_lengths(ed, qu, qd, steps):
    """The stored-basis Ritz sum (exact, carried every 16 terms) at term
    counts around the carry interval, for odd and even row counts, against the
    second-pass sum, which adds the same vectors one at a time in FP64: at
    most one rounding of 2^-53 a term apart, 1e-14 in norm."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    from conftest import philox_uniform
    t = L.chain(7, eps=list(philox_uniform(9, 7, 1.5)))
    op = ed.Hubbard(ed.H_TBq(7, qu).extend(t), ed.H_TBq(7, qd).extend(t), 3.0)
    if steps > op.rows() // 3:
        pytest.skip("more steps than the sector's Krylov space")
    e1, v1 = ed.Lanczos().eigen(op, max_steps=steps, mode="fixed", ritz="stored", seed=4)
    e2, v2 = ed.Lanczos().eigen(op, max_steps=steps, mode="fixed", ritz="recompute", seed=4)
    assert e1 == e2
    assert np.linalg.norm(v1 - v2) < 1e-14
    op.close()


@pytest.mark.parametrize("case", ["tiny", "odd", "odd_long", "complex", "multi_class", "wide", "wider", "one_row", "reference"])
def test_reorth_one_launch_matches_per_step(ed, monkeypatch, case):
    """A reorthogonalised run in one cooperative launch gives the per-step
    kernels' T, E0, Ritz vector and bookkeeping bit for bit: odd and even
    sectors, complex and multi-class operators, the basis in shared memory or
    not (long runs, wide ranges), a range wider than the block, one row, and
    the stop test's launches of ten steps."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    N, qu, qd, t, steps, mode = 8, 4, 4, L.chain(8), 40, "fixed"
    if case == "tiny":
        N, qu, qd, t, steps = 4, 2, 2, L.chain(4), 8
    elif case in ("odd", "odd_long"):
        N, qu, qd, t = 7, 3, 2, L.chain(7, eps=list(philox_uniform(6, 7, 1.0)))
        steps = 33 if case == "odd" else 400
    elif case == "complex":
        N, qu, qd, t = 12, 2, 3, L.kagome12(flux=0.4)
    elif case == "multi_class":
        N, qu, qd, t = 12, 3, 2, L.lieb12(list(philox_uniform(8, 12, 0.5) + 1.0))
    elif case == "wide":
        N, qu, qd, t, steps = 10, 5, 5, L.chain(10), 70
    elif case == "wider":
        N, qu, qd, t, steps = 11, 5, 5, L.chain(11), 25
    elif case == "one_row":
        N, qu, qd, t = 9, 0, 4, L.chain(9, eps=list(philox_uniform(2, 9, 1.0)))
    else:
        steps, mode = 200, "reference"
    got = {}
    for form in ("launch", "steps"):
        monkeypatch.setenv("ED_LZ_FUSED", "0") if form == "steps" else monkeypatch.delenv("ED_LZ_FUSED", raising=False)
        op = op_for(ed, N, qu, qd, t, t, 4.0)
        lz = ed.Lanczos()
        e0, v = lz.eigen(op, max_steps=steps, mode=mode, ritz="stored", reorth=True, seed=5)
        r = lz.result
        got[form] = (e0, lz.a, lz.b, r.steps, r.status, r.min_bits, r.converged, r.residual), v, r.launches
        op.close()
    assert got["launch"][0] == got["steps"][0]
    assert np.array_equal(got["launch"][1], got["steps"][1])
    assert got["launch"][2] < got["steps"][2]


# batches on the row pairs: one to sixteen buffers' worth of units a pair, odd up
# and down counts, signs of either kind and mixed, unequal hopping of the spins, one
# pair, vectors above and below a pass of the grid, more items than CTAs or fewer
@pytest.mark.parametrize("N,qu,qd,B,ring,t_dn", [(8, 4, 4, 2, True, -1.0), (9, 4, 2, 8, False, -1.0), (7, 3, 4, 3, True, -1.0),
                                                 (10, 5, 5, 7, False, 1.0), (11, 5, 5, 3, True, -0.7), (6, 0, 3, 2, True, -1.0),
                                                 (6, 1, 6, 2, True, -1.0), (12, 6, 5, 2, True, -1.0)])
def test_lanczos_batch_sectors(ed, N, qu, qd, B, ring, t_dn):
    from conftest import philox_uniform
    ops = []
    for r in range(B):
        eps = philox_uniform(40 + r, 2 * N, 2.0)
        bonds = [(i, (i + 1) % N) for i in range(N if ring else N - 1)]
        tu = [("H", i, j, -1.0, 0.0) for i, j in bonds] + [("N", i, 0, eps[i], 0.0) for i in range(N)]
        td = [("H", i, j, t_dn, 0.0) for i, j in bonds] + [("N", i, 0, eps[N + i], 0.0) for i in range(N)]
        ops.append(ed.Hubbard(ed.H_TBq(N, qu).extend(tu), ed.H_TBq(N, qd).extend(td), 1.0 + 0.25 * r))
    steps = min(15, ops[0].rows())
    e0, ev, al, be = ed.lanczos_batch(ops, steps, seed=3)
    for b, op in enumerate(ops):
        lz = ed.Lanczos()
        e, v = lz.eigen(op, max_steps=steps, mode="fixed", seed=3 + b)
        n = len(lz.a)
        assert e0[b] == e
        assert np.array_equal(al[b][:n], np.array(lz.a)) and np.array_equal(be[b][:n + 1], np.array(lz.b)[:n + 1])
        assert np.array_equal(ev[b], v)
        op.close()


@pytest.mark.parametrize("steps", [127, 128, 129, 257])
@pytest.mark.parametrize("N,qu,qd,near", [(10, 4, 3, False), (11, 3, 3, False), (10, 4, 3, True), (11, 3, 3, True)])
def test_ritz_sum_long(ed, N, qu, qd, near, steps):
    """The stored-basis Ritz sum past its carry interval (128 terms), even and
    odd row counts, against the second-pass sum; near: a start vector 1e-5 from
    the ground state, whose coefficients fall so fast that a segment ends inside
    a batch of vectors.  Each sum is off by a rounding of 2^-53 a term and two
    of the normalisation at most."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    t = L.chain(N, eps=list(philox_uniform(9, N, 1.5)))
    op = op_for(ed, N, qu, qd, t, t, 3.0)
    f = None
    if near:
        _, f = ed.Lanczos().eigen(op, max_steps=100, mode="fixed", reorth=True, seed=2)
        f = f + 1e-5 * ed.Lanczos().random_vector(op.rows(), 3)
    e1, v1 = ed.Lanczos().eigen(op, f, max_steps=steps, mode="fixed", ritz="stored", seed=4)
    e2, v2 = ed.Lanczos().eigen(op, f, max_steps=steps, mode="fixed", ritz="recompute", seed=4)
    assert e1 == e2
    assert np.linalg.norm(v1 - v2) < 2 * (steps + 2) * 2.0**-53
    op.close()


@pytest.mark.parametrize("case", ["one_class", "complex", "classes", "reference"])
def test_reorth_goes_over_to_per_step(ed, monkeypatch, case):
    """Reorthogonalised runs of large sectors: the first steps in one launch, the
    others by the per-step kernels (nine launches a step), with the bits of a
    run that takes those from the start; the stop test on both sides."""
    from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L
    N, qu, qd, steps, mode, per_step = 12, 6, 6, 125, "fixed", 8  # 853,776 values: 117 steps in one launch
    t = L.chain(12, eps=list(philox_uniform(6, 12, 1.0)))
    if case == "complex":
        t, qu, qd, steps, per_step = L.kagome12(flux=0.4), 3, 5, 40, 12  # 348,480 values: 28
    elif case == "classes":
        t, qu, qd, steps, per_step = L.lieb12(list(philox_uniform(8, 12, 0.5) + 1.0)), 4, 4, 50, 10  # 245,025 values: 40
    elif case == "reference":
        t, qu, qd, steps, mode, per_step = L.kagome12(flux=0.4), 3, 5, 100, "reference", 30
    got = {}
    for form in ("default", "steps"):
        monkeypatch.setenv("ED_LZ_FUSED", "0") if form == "steps" else monkeypatch.delenv("ED_LZ_FUSED", raising=False)
        op = op_for(ed, N, qu, qd, t, t, 4.0)
        lz = ed.Lanczos()
        e0, v = lz.eigen(op, max_steps=steps, mode=mode, ritz="stored", reorth=True, seed=5)
        r = lz.result
        got[form] = (e0, lz.a, lz.b, r.steps, r.status, r.min_bits, r.converged, r.residual), v, r.launches
        op.close()
    assert got["default"][0] == got["steps"][0]
    assert np.array_equal(got["default"][1], got["steps"][1])
    assert 9 * per_step <= got["default"][2] < got["steps"][2]
