"""Performance cases: what a user of this package has it compute, through its
public entry points, from single operator applications on a few thousand
states to Lanczos runs on vectors far beyond the L2 cache.

Kinds of case
  apply     y = H x on device vectors (``Hubbard.Hubbard_mv``), real and complex
  solve     ground state by fixed-step Lanczos with its Ritz vector (``Lanczos.eigen``)
  disorder  one batch of a disorder sweep: Lanczos of several samples, their
            entanglement entropies and site densities
  flux      one twist of a flux sweep: complex ground state and the first and
            second derivative of E0
  excited   several lowest eigenpairs of a random-hopping cluster and S^2 of each
  evolve    a quench: psi(t) at many times from one Krylov space

``exact`` gives the same quantities from plain FP64 torch and numpy code that
shares nothing with the package.
"""
import math

import numpy as np
import torch

from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import evolution, hubbard, observables, spectra
from exact_diagonalization_for_fermionic_systems_with_gpu_gb300 import lattices as L


def _case(name, kind, lattice, n_sites, n_up, n_dn, U, **kw):
    return dict(name=name, kind=kind, lattice=lattice, n_sites=n_sites, n_up=n_up, n_dn=n_dn, U=U, **kw)


def listed():
    return [
        # the inner call of a user's own iteration on the smallest cluster of the examples: launch latency
        _case("apply_chain8", "apply", "ring", 8, 4, 4, 4.0),
        # the reference's headline operator, vectors inside L2
        _case("apply_kagome12", "apply", "kagome", 12, 6, 6, 8.0),
        # the twisted (Peierls) operator of the flux sweep
        _case("apply_flux_kagome12", "apply", "kagome_flux", 12, 6, 6, 4.0),
        # the reference's 16-site chain with disorder: 1.3 GB vectors
        _case("apply_chain16", "apply", "chain", 16, 8, 8, 1.0),
        # the smallest ground state, fully reorthogonalised: many tiny dependent steps
        _case("solve_chain8_reorth", "solve", "ring", 8, 4, 4, 4.0, steps=100, ritz="stored", reorth=True),
        # the headline ground state
        _case("solve_kagome12", "solve", "kagome", 12, 6, 6, 8.0, steps=300, ritz="stored", reorth=False),
        # a ground state whose vectors and Krylov basis are larger than L2
        _case("solve_chain14", "solve", "chain", 14, 7, 7, 1.0, steps=100, ritz="stored", reorth=False),
        # the 18-site Lieb cluster (down rows beyond shared memory), the Ritz vector by a second recurrence
        _case("solve_lieb18", "solve", "lieb18", 18, 4, 9, 4.0, steps=40, ritz="recompute", reorth=False),
        # eight samples of the disorder sweep's (7, 5) sector
        _case("disorder_chain12", "disorder", "chain", 12, 7, 5, 1.0, steps=300, samples=8),
        # one twist of the flux sweep
        _case("flux_kagome12", "flux", "kagome_flux", 12, 6, 6, 4.0, steps=300, response_steps=100),
        # four levels of the random-hopping Lieb cluster with their total spin
        _case("excited_lieb12", "excited", "lieb_random", 12, 6, 6, 4.0, nev=4),
        # a complex state of the 12-site chain at sixteen times
        _case("evolve_chain12", "evolve", "chain", 12, 6, 6, 1.0, steps=140, times=16, t_max=2.0),
    ]


#: no drawn sector is larger than the largest listed one
_MAX_ROWS = math.comb(16, 8) ** 2


def _sector(rng, n, spread, max_rows):
    """(N_up, N_dn) near half filling, odd and unequal ones among them."""
    while True:
        qu = min(n - 1, max(1, n // 2 + rng.randint(-spread, spread)))
        qd = min(n - 1, max(1, n // 2 + rng.randint(-spread, spread)))
        if math.comb(n, qu) * math.comb(n, qd) <= max_rows:
            return qu, qd


def draw(rng):
    kind = rng.choice(["apply", "apply", "solve", "solve", "disorder", "flux", "excited", "evolve"])
    U = rng.choice([1.0, 2.0, 4.0, 8.0]) + rng.randint(0, 9) / 10.0
    if kind == "apply":
        lat = rng.choice(["ring", "chain", "chain", "kagome", "kagome_flux", "lieb_random"])
        n = rng.randint(6, 16) if lat in ("ring", "chain") else 12  # rows grow by a factor of about 15 per two sites
        qu, qd = _sector(rng, n, 2, _MAX_ROWS)
        return _draw(kind, lat, n, qu, qd, U)
    if kind == "solve":
        pick = rng.randint(0, 5)
        if pick == 0:
            n = rng.randint(7, 9)
            qu, qd = _sector(rng, n, 1, 20000)
            return _draw(kind, "ring", n, qu, qd, U, steps=rng.randint(40, 80), ritz="stored", reorth=True)
        if pick == 1:
            return _draw(kind, "lieb18", 18, rng.randint(2, 4), rng.choice([8, 9, 10]), U, steps=rng.randint(15, 40),
                         ritz="recompute", reorth=False)
        if pick == 2:
            qu, qd = _sector(rng, 12, 2, _MAX_ROWS)
            return _draw(kind, "kagome", 12, qu, qd, U, steps=rng.randint(100, 300), ritz="stored", reorth=False)
        n = rng.randint(9, 15)
        qu, qd = _sector(rng, n, 2, math.comb(14, 7) ** 2 * 2)
        return _draw(kind, "chain", n, qu, qd, U, steps=rng.randint(30, 100), ritz="stored", reorth=False)
    if kind == "disorder":
        n = rng.randint(10, 12)
        qu, qd = _sector(rng, n, 2, math.comb(12, 6) * math.comb(12, 5))
        return _draw(kind, "chain", n, qu, qd, U, steps=rng.randint(150, 300), samples=rng.randint(2, 8))
    if kind == "flux":
        qu, qd = _sector(rng, 12, 1, _MAX_ROWS)
        return _draw(kind, "kagome_flux", 12, qu, qd, U, steps=rng.randint(250, 300),
                     response_steps=rng.randint(50, 100))
    if kind == "excited":
        qu, qd = _sector(rng, 12, 1, _MAX_ROWS)
        return _draw(kind, "lieb_random", 12, qu, qd, U, nev=rng.randint(2, 5))
    n = rng.randint(10, 13)
    qu, qd = _sector(rng, n, 1, math.comb(12, 6) ** 2 * 2)
    t_max = rng.choice([0.5, 1.0, 2.0])  # the Krylov space has to reach t_max times half the spectral width
    return _draw(kind, "chain", n, qu, qd, U, steps=40 + int(50 * t_max) + rng.randint(0, 20),
                 times=rng.randint(3, 16), t_max=t_max)


def _draw(*a, **kw):
    c = _case(None, *a, **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------- models --
def _terms(case, rng, derivative=0, phi=None):
    """(up terms, down terms) of the case's lattice; rng gives the disorder."""
    lat, n = case["lattice"], case["n_sites"]
    if lat == "ring":
        t = L.chain(n)
        return t, t
    if lat == "chain":  # on-site disorder W * uniform(-1, 1), drawn for each spin
        w = 6.0
        return (L.chain(n, periodic=False, eps=w * rng.uniform(-1, 1, n)),
                L.chain(n, periodic=False, eps=w * rng.uniform(-1, 1, n)))
    if lat == "kagome":
        t = L.kagome12()
    elif lat == "kagome_flux":
        d1, d2 = L.kagome12_flux_derivatives(phi)
        t = (L.kagome12(flux=phi, peierls=True), d1, d2)[derivative]
    elif lat == "lieb_random":
        t = L.lieb12(list(rng.uniform(0.5, 1.5, 12)))
    else:
        t = L.lieb18()
    return t, t


def _model(case, seed, sample=0, derivative=0):
    """Term lists of one sample, the same for prepare and exact."""
    rng = np.random.default_rng([seed, sample])
    phi = float(rng.uniform(0.2, 0.5))
    return _terms(case, rng, derivative, phi)


def _op(case, terms, U=None):
    n = case["n_sites"]
    up = hubbard.H_TBq(n, case["n_up"]).extend(terms[0])
    dn = hubbard.H_TBq(n, case["n_dn"]).extend(terms[1])
    return hubbard.Hubbard(up, dn, case["U"] if U is None else U)


def _vector(rows, seed, cplx):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.complex128 if cplx else torch.float64
    x = torch.randn(rows, dtype=dt, device="cuda", generator=g)
    return x / torch.linalg.vector_norm(x)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "disorder":
        ops = [_op(case, _model(case, seed, b)) for b in range(case["samples"])]
        evecs = torch.empty((len(ops), ops[0].rows()), dtype=torch.float64, device="cuda")
        return {"case": case, "seed": seed, "ops": ops, "evecs": evecs}
    op = _op(case, _model(case, seed))
    state = {"case": case, "seed": seed, "op": op}
    dt = torch.complex128 if op.is_complex else torch.float64
    if kind == "apply":
        state["x"] = _vector(op.rows(), seed, op.is_complex)
        state["y"] = torch.empty(op.rows(), dtype=dt, device="cuda")
    elif kind in ("solve", "flux"):
        state["evec"] = torch.empty(op.rows(), dtype=dt, device="cuda")
    if kind == "flux":
        state["d1"] = _op(case, _model(case, seed, derivative=1), 0.0)
        state["d2"] = _op(case, _model(case, seed, derivative=2), 0.0)
    if kind == "evolve":
        state["psi"] = _vector(op.rows(), seed, True)
    return state


def _half(case):
    return range(case["n_sites"] // 2)


def run(state):
    case, seed, kind = state["case"], state["seed"], state["case"]["kind"]
    if kind == "disorder":
        ops, evecs = state["ops"], state["evecs"]
        e0, _, _, _ = hubbard.lanczos_batch(ops, case["steps"], seed=seed, evec_out=evecs)
        svn, sref = observables.entanglement_entropy_batch(ops[0], evecs, _half(case))
        dens = [observables.site_densities(op, evecs[b]) for b, op in enumerate(ops)]
        return {"e0": e0, "evecs": evecs, "s_vn": svn, "s_ref": sref, "densities": np.array(dens)}
    op = state["op"]
    if kind == "apply":
        op.Hubbard_mv(state["x"], state["y"])
        return {"y": state["y"]}
    if kind == "solve":
        e0, evec = hubbard.Lanczos(op.dimUP, op.dimDN).eigen(
            op, max_steps=case["steps"], mode="fixed", ritz=case["ritz"], reorth=case["reorth"], seed=seed,
            evec_out=state["evec"])
        return {"e0": e0, "evec": evec}
    if kind == "flux":
        e0, psi = hubbard.Lanczos(op.dimUP, op.dimDN).eigen(op, max_steps=case["steps"], mode="fixed", ritz="stored",
                                                            seed=seed, evec_out=state["evec"])
        d1, d2 = observables.response(op, state["d1"], state["d2"], psi, e0, steps=case["response_steps"])
        return {"e0": e0, "evec": psi, "d1": d1, "d2": d2}
    if kind == "excited":
        w, v, _ = spectra.eigs_lowest(op, case["nev"], seed=seed)
        s2 = [observables.s2_expect(op, v[k])[1] for k in range(case["nev"])]
        return {"evals": w, "evecs": v, "s2": np.array(s2)}
    psi = evolution.krylov_evolve(op, state["psi"], _times(case), max_steps=case["steps"])
    return {"psi": psi}


def _times(case):
    return [case["t_max"] * (k + 1) / case["times"] for k in range(case["times"])]


# ------------------------------------------------------------------ work --
_BONDS = {"kagome": 24, "kagome_flux": 24, "lieb_random": 16, "lieb18": 24}


def work(case):
    """Bytes and operations one pass cannot do without: every input read and
    every output written once; for a Krylov method each step reads its two
    vectors, writes one and applies H, and the result reads the basis once."""
    n, qu, qd = case["n_sites"], case["n_up"], case["n_dn"]
    rows = math.comb(n, qu) * math.comb(n, qd)
    w = 2 if case["lattice"] == "kagome_flux" else 1
    bonds = _BONDS.get(case["lattice"], n if case["lattice"] == "ring" else n - 1)
    hops = sum(2.0 * bonds * q * (n - q) / (n * (n - 1)) for q in (qu, qd))
    mv = 2.0 * rows * (hops + 1) * (4 if w == 2 else 1)
    vec = 8.0 * rows * w
    kind = case["kind"]
    if kind == "apply":
        return {"bytes": 2 * vec, "flops": mv}
    steps = case.get("steps", 0)
    if kind == "solve":
        passes = 2 if case["ritz"] == "recompute" else 1
        ortho = 4.0 * rows * steps * steps if case["reorth"] else 0.0
        return {"bytes": passes * steps * 3 * vec + (steps * vec if passes == 1 else 0) + vec,
                "flops": passes * steps * (mv + 10.0 * rows) + 2.0 * rows * steps + ortho}
    if kind == "flux":
        total = steps + case["response_steps"]
        return {"bytes": total * 3 * vec + steps * vec + vec, "flops": total * (mv + 20.0 * rows * w) + 4.0 * rows * steps}
    if kind == "disorder":
        one = steps * (mv + 10.0 * rows) + 2.0 * rows * steps
        svd = sum(_svd_flops(case))
        return {"bytes": case["samples"] * (4 * steps + 3) * vec, "flops": case["samples"] * (one + svd)}
    if kind == "excited":
        ncv = 4 * (case["nev"] + 1)  # one cycle at the least
        return {"bytes": ncv * 3 * vec + case["nev"] * 2 * vec, "flops": ncv * (mv + 4.0 * rows * ncv)}
    t = case["times"]
    return {"bytes": 2 * (4 * steps * vec) + (t + 1) * 2 * vec,
            "flops": 2 * (steps * (mv + 10.0 * rows) + 4.0 * rows * steps * t)}


def _blocks(n, qu, qd):
    """(ku, kd, rows, columns) of the entanglement blocks of the first n // 2 sites."""
    a = n // 2
    b = n - a
    for ku in range(max(0, qu - b), min(a, qu) + 1):
        for kd in range(max(0, qd - b), min(a, qd) + 1):
            yield (ku, kd, math.comb(a, ku) * math.comb(a, kd), math.comb(b, qu - ku) * math.comb(b, qd - kd))


def _svd_flops(case):
    for _, _, r, c in _blocks(case["n_sites"], case["n_up"], case["n_dn"]):
        m, k = max(r, c), min(r, c)
        yield 4.0 * m * k * k - 4.0 * k ** 3 / 3.0


# ----------------------------------------------------------------- exact --
def _basis(n, q):
    words = np.arange(1 << n, dtype=np.int64)
    count = np.zeros_like(words)
    for i in range(n):
        count += (words >> i) & 1
    return words[count == q]


def _between(words, i, j):
    lo, hi = min(i, j), max(i, j)
    par = np.zeros_like(words)
    for k in range(lo + 1, hi):
        par ^= (words >> k) & 1
    return 1.0 - 2.0 * par


class _Exact:
    """H of one sector as two sparse one-spin matrices and a diagonal, on the GPU in 64 bits."""

    def __init__(self, case, terms, U):
        n = case["n_sites"]
        self.cplx = case["lattice"] == "kagome_flux"
        self.dt = torch.complex128 if self.cplx else torch.float64
        self.up, eu, self.wu = self._spin(n, case["n_up"], terms[0])
        self.dn, ed, self.wd = self._spin(n, case["n_dn"], terms[1])
        self.nu, self.nd = len(self.wu), len(self.wd)
        wu, wd = torch.from_numpy(self.wu).cuda(), torch.from_numpy(self.wd).cuda()
        diag = torch.from_numpy(eu).cuda()[:, None] + torch.from_numpy(ed).cuda()[None, :]
        for i in range(n):
            diag += U * (((wu >> i) & 1)[:, None] * ((wd >> i) & 1)[None, :])
        self.diag = diag

    def _spin(self, n, q, terms):
        words = _basis(n, q)
        where = np.full(1 << n, -1, dtype=np.int64)
        where[words] = np.arange(len(words))
        diag = np.zeros(len(words))
        rows, cols, vals = [], [], []
        for kind, i, j, v, ph in terms:
            if kind == "N":
                diag += v * ((words >> i) & 1)
                continue
            full = np.nonzero((((words >> i) & 1) == 1) & (((words >> j) & 1) == 0))[0]  # i -> j
            to = where[words[full] ^ ((1 << i) | (1 << j))]
            amp = v * _between(words[full], i, j) * np.exp(1j * (ph if kind == "P" else 0.0))
            rows += [to, full]
            cols += [full, to]
            vals += [amp, amp.conj()]
        r, c, a = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
        a = a if self.cplx else a.real
        m = torch.sparse_coo_tensor(np.stack([r, c]), torch.from_numpy(np.ascontiguousarray(a)),
                                    (len(words), len(words))).coalesce()
        return m.to_sparse_csr().cuda(), diag, words

    def __call__(self, x):
        x = x.reshape(self.nu, self.nd)
        y = self.diag * x
        y += self.up @ x
        y += (self.dn @ x.t().contiguous()).t()
        return y.reshape(-1)


def _start(rows, seed, cplx):
    """uniform(-1, 1) from numpy's Philox counter keyed by seed."""
    bits = np.random.Philox(key=[seed, 0]).random_raw(rows * (2 if cplx else 1))
    f = ((bits >> np.uint64(12)) | np.uint64(0x3FF0000000000000)).view(np.float64) * 2.0 - 3.0
    x = torch.from_numpy(f.view(np.complex128) if cplx else f).cuda()
    return x / torch.linalg.vector_norm(x)


def _tri(alpha, beta):
    k = len(alpha)
    return np.diag(alpha) + np.diag(beta[1:k], 1) + np.diag(beta[1:k], -1)


def _lanczos(H, x, steps, keep=True):
    """alpha, beta (beta[0] = |x|) and the basis; orthogonalised in full where the basis is kept."""
    beta, alpha = [float(torch.linalg.vector_norm(x))], []
    V = torch.zeros((steps, x.numel()), dtype=x.dtype, device=x.device) if keep else None
    v, prev = x / beta[0], None
    for k in range(steps):
        if keep:
            V[k] = v
        w = H(v)
        alpha.append(float(torch.vdot(v, w).real))
        w -= alpha[-1] * v
        if prev is not None:
            w -= beta[-1] * prev
        if keep:
            for _ in range(2):
                w -= (V[: k + 1].conj() @ w) @ V[: k + 1]
        beta.append(float(torch.linalg.vector_norm(w)))
        if beta[-1] < 1e-12:
            break
        prev, v = v, w / beta[-1]
    return np.array(alpha), np.array(beta), V


def _ground(H, x, steps, keep=True):
    a, b, V = _lanczos(H, x, steps, keep)
    w, z = np.linalg.eigh(_tri(a, b))
    z = z[:, 0]
    z = z if z[np.argmax(np.abs(z))] > 0 else -z
    if not keep:
        return float(w[0]), None
    psi = torch.from_numpy(z).to(V.dtype).cuda() @ V[: len(z)]
    return float(w[0]), psi / torch.linalg.vector_norm(psi)


def _entropies(case, H, psi):
    """(S_vN, sum -s ln s) of the first n // 2 sites, block by block."""
    n, a = case["n_sites"], case["n_sites"] // 2
    M = psi.reshape(H.nu, H.nd).cpu().numpy()

    def split(words):
        pa, pb = words & ((1 << a) - 1), words >> a
        cnt = np.array([bin(int(w)).count("1") for w in pa])
        return cnt, pa, pb

    cu, au, bu = split(H.wu)
    cd, ad, bd = split(H.wd)
    s_vn = s_ref = 0.0
    for ku, kd, _, _ in _blocks(n, case["n_up"], case["n_dn"]):
        iu, idn = np.nonzero(cu == ku)[0], np.nonzero(cd == kd)[0]
        ua, ra = np.unique(au[iu], return_inverse=True)
        ub, rb = np.unique(bu[iu], return_inverse=True)
        da, sa = np.unique(ad[idn], return_inverse=True)
        db, sb = np.unique(bd[idn], return_inverse=True)
        block = np.zeros((len(ua), len(da), len(ub), len(db)))
        block[ra[:, None], sa[None, :], rb[:, None], sb[None, :]] = M[np.ix_(iu, idn)]
        s = np.linalg.svd(block.reshape(len(ua) * len(da), -1), compute_uv=False)
        s = s[s > 0]
        s_ref -= float(np.sum(s * np.log(s)))
        q = s * s
        q = q[q > 0]
        s_vn -= float(np.sum(q * np.log(q)))
    return s_vn, s_ref


def _densities(case, H, psi):
    n = case["n_sites"]
    p = (psi.abs() ** 2).reshape(H.nu, H.nd)
    up = np.array([((H.wu >> i) & 1) for i in range(n)], dtype=np.float64)
    dn = np.array([((H.wd >> i) & 1) for i in range(n)], dtype=np.float64)
    U, D = torch.from_numpy(up).cuda(), torch.from_numpy(dn).cuda()
    return np.array([(U @ p.sum(1)).cpu().numpy(), (D @ p.sum(0)).cpu().numpy(),
                     ((U @ p) * D).sum(1).cpu().numpy()])


def _s2(case, H, psi):
    """S^2 = ((N_up - N_dn) / 2)^2 + (|S+ psi|^2 + |S- psi|^2) / 2."""
    n, qu, qd = case["n_sites"], case["n_up"], case["n_dn"]
    M = psi.reshape(H.nu, H.nd).cpu().numpy()

    def flip(src, dst, rs, rd, ws, wd):
        # sum_i c+_(i, dst) c_(i, src) on M with rs, rd the target bases
        out = np.zeros((len(rs), len(rd)))
        for i in range(n):
            s = np.nonzero((ws >> i) & 1)[0]
            d = np.nonzero(((wd >> i) & 1) == 0)[0]
            ss = _between(ws[s], -1, i)
            sd = _between(wd[d], -1, i)
            ts = np.searchsorted(rs, ws[s] ^ (1 << i))
            td = np.searchsorted(rd, wd[d] | (1 << i))
            block = M[np.ix_(s, d)] if src == "up" else M[np.ix_(d, s)].T
            out[np.ix_(ts, td)] += ss[:, None] * sd[None, :] * block
        return float(np.sum(out * out))

    total = 0.0
    if qd > 0 and qu < n:  # S+
        total += flip("dn", "up", _basis(n, qd - 1), _basis(n, qu + 1), H.wd, H.wu)
    if qu > 0 and qd < n:  # S-
        total += flip("up", "dn", _basis(n, qu - 1), _basis(n, qd + 1), H.wu, H.wd)
    return 0.25 * (qu - qd) ** 2 + 0.5 * total


def _lowest(H, x, nev):
    """The nev lowest eigenpairs: Lanczos with the whole basis kept, until they have settled."""
    last = None
    for steps in (120, 200, 320):
        a, b, V = _lanczos(H, x, steps)
        w, z = np.linalg.eigh(_tri(a, b))
        if last is not None and np.max(np.abs(w[:nev] - last)) < 1e-12 * abs(w[0]):
            break
        last = w[:nev]
    vecs = torch.from_numpy(np.ascontiguousarray(z[:, :nev].T)).cuda() @ V[: len(w)]
    return w[:nev], vecs


def _expm(H, psi, times):
    """exp(-i H t) psi by Taylor steps of dt |H| <= 2."""
    bound = float(H.diag.abs().max()) + 30.0
    out, t = [], 0.0
    for t1 in times:
        m = max(1, math.ceil((t1 - t) * bound / 2.0))
        dt = (t1 - t) / m
        for _ in range(m):
            term = psi
            acc = psi.clone()
            for k in range(1, 40):
                hr = torch.complex(H(term.real.contiguous()), H(term.imag.contiguous()))
                term = hr * (-1j * dt / k)
                acc += term
                if k % 6 == 0 and float(torch.linalg.vector_norm(term)) < 1e-17:
                    break
            psi = acc
        t = t1
        out.append(psi)
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "disorder":
        e0, svn, sref, dens = [], [], [], []
        for b in range(case["samples"]):
            H = _Exact(case, _model(case, seed, b), case["U"])
            e, psi = _ground(H, _start(H.nu * H.nd, seed + b, False), case["steps"])
            s = _entropies(case, H, psi)
            e0.append(e)
            svn.append(s[0])
            sref.append(s[1])
            dens.append(_densities(case, H, psi))
        return {"e0": np.array(e0), "evecs": None, "s_vn": np.array(svn), "s_ref": np.array(sref),
                "densities": np.array(dens)}
    H = _Exact(case, _model(case, seed), case["U"])
    rows = H.nu * H.nd
    if kind == "apply":
        return {"y": H(_vector(rows, seed, H.cplx))}
    if kind == "solve":
        keep = rows * case["steps"] <= 1 << 31
        e0, psi = _ground(H, _start(rows, seed, False), case["steps"], keep)
        return {"e0": e0, "evec": psi if case["reorth"] else None}
    if kind == "flux":
        e0, psi = _ground(H, _start(rows, seed, True), case["steps"])
        dH = _Exact(case, _model(case, seed, derivative=1), 0.0)
        d2H = _Exact(case, _model(case, seed, derivative=2), 0.0)
        phi = dH(psi)
        d1 = torch.vdot(psi, phi)
        a, b, _ = _lanczos(H, phi - d1 * psi, case["response_steps"])
        g = 1.0 / (e0 - a[-1])
        for k in range(len(a) - 2, -1, -1):
            g = 1.0 / (e0 - a[k] - g * b[k + 1] ** 2)
        d2 = float(torch.vdot(psi, d2H(psi)).real) + 2.0 * b[0] ** 2 * g
        return {"e0": e0, "evec": None, "d1": float(d1.real), "d2": d2}
    if kind == "excited":
        w, v = _lowest(H, _start(rows, seed, False), case["nev"])
        return {"evals": w, "evecs": None, "s2": np.array([_s2(case, H, v[k]) for k in range(case["nev"])])}
    return {"psi": _expm(H, _vector(rows, seed, True), _times(case))}
