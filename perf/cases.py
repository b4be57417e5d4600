"""Performance cases of the CSF-FCI engine: the calls that a CASCI/CASSCF
program or a user of the batched solver makes, each through a public entry
point, with the inputs such a program has in hand.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, solver object and what a program keeps
    run(state)          one pass; returns its outputs
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   the outputs of run() in plain torch/numpy, 64 bits

Kinds of case (the key "kind"):

    sigma      FCISolver.contract_2e: one H.c on a determinant vector
    rdm        make_rdm12 / make_rdm12s / trans_rdm12 / trans_rdm12s / make_rdm1
    transform  CSFTransformer.vec_csf2det followed by vec_det2csf
    diagonal   make_hdiag, then make_hdiag_csf over it
    solve      FCISolver.kernel plus make_rdm12 of every root, host in and out
    batch      BatchedCSFSolver.kernel on many uneven problems
    gradient   csf_fci_energy, forward and backward, with a kept solver
"""
import itertools
from math import comb

import numpy as np
import torch

import pyscf_forge_b200 as b200
from pyscf_forge_b200 import autograd, batched
from pyscf_forge_b200.csf_fci.csfstring import CSFTransformer, count_all_csfs

# Davidson settings of the repository's own solves
SOLVER = dict(conv_tol=1e-10, max_cycle=400, max_space=30)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest sigma: a few hundred determinants, latency only
        dict(name="sigma6", kind="sigma", norb=6, na=3, nb=3, eta=1, host=False, spin_h1=False),
        # an odd-electron vector from host memory, spin-dependent h1 (UHF-like
        # orbitals): numpy in and out, as a CPU program calls it
        dict(name="sigma11_host", kind="sigma", norb=11, na=6, nb=5, eta=0, host=True, spin_h1=True),
        # the ordinary CAS(12,12) singlet sigma, device resident
        dict(name="sigma12", kind="sigma", norb=12, na=6, nb=6, eta=1, host=False, spin_h1=False),
        # an odd orbital count with unequal electron numbers
        dict(name="sigma13_odd", kind="sigma", norb=13, na=7, nb=6, eta=0, host=False, spin_h1=False),
        # the largest: CAS(16,16) singlet, the headline vector
        dict(name="sigma16", kind="sigma", norb=16, na=8, nb=8, eta=1, host=False, spin_h1=False),
        # density matrices of a CAS(14,14) singlet (every CASSCF macro-iteration)
        dict(name="rdm14", kind="rdm", call="make_rdm12", norb=14, na=7, nb=7, eta=1),
        # spin-resolved transition densities between two doublets (property
        # integrals, state interaction)
        dict(name="trans_rdm11s", kind="rdm", call="trans_rdm12s", norb=11, na=6, nb=5, eta=0),
        # CSF -> determinants -> CSF of a block of two triplet vectors, as
        # each Davidson iteration does
        dict(name="transform14", kind="transform", norb=14, na=7, nb=7, smult=3, nvec=2),
        # the determinant and CSF diagonals that start every solve
        dict(name="diagonal14", kind="diagonal", norb=14, na=7, nb=7, smult=3),
        # a whole small solve with its densities (active space of eight)
        dict(name="solve8", kind="solve", norb=8, na=4, nb=4, smult=1, nroots=1),
        # many uneven problems at once, singlets to quintets, one to four roots
        dict(name="batch20", kind="batch", nprob=20, first=1000, norb_lo=6, norb_hi=11),
        # three-state energy and its gradient with respect to the integrals
        dict(name="gradient12", kind="gradient", norb=12, na=6, nb=6, smult=1, nroots=3),
    ]


def _electrons(rng, norb):
    """Electron numbers around half filling, odd totals as often as even."""
    tot = max(2, min(2 * norb - 2, norb + rng.randint(-2, 2)))
    na = (tot + 1) // 2
    if rng.random() < 0.25 and na + 1 <= norb and tot - na > 1:
        na += 1
    return na, tot - na


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "rdm", "rdm", "transform", "diagonal", "solve", "batch", "gradient"])
    if kind == "sigma":
        norb = rng.randint(5, 15)
        na, nb = _electrons(rng, norb)
        eta = rng.choice([0, 1, -1]) if na == nb else 0
        return dict(kind=kind, norb=norb, na=na, nb=nb, eta=eta, host=norb <= 12 and rng.random() < 0.4,
                    spin_h1=na != nb and rng.random() < 0.4)
    if kind == "rdm":
        norb = rng.randint(5, 14)
        na, nb = _electrons(rng, norb)
        call = rng.choice(["make_rdm12", "make_rdm12", "make_rdm12s", "trans_rdm12", "trans_rdm12s", "make_rdm1"])
        return dict(kind=kind, call=call, norb=norb, na=na, nb=nb, eta=rng.choice([0, 1, -1]) if na == nb else 0)
    if kind in ("transform", "diagonal"):
        norb = rng.randint(6, 14)
        na, nb = _electrons(rng, norb)
        c = dict(kind=kind, norb=norb, na=na, nb=nb, smult=na - nb + 1 + 2 * rng.randint(0, 1))
        if kind == "transform":
            c["nvec"] = rng.randint(1, 4)
        return c
    if kind in ("solve", "gradient"):
        norb = rng.randint(6, 10)
        na, nb = _electrons(rng, norb)
        smult = na - nb + 1 + 2 * rng.randint(0, 1)
        return dict(kind=kind, norb=norb, na=na, nb=nb, smult=smult, nroots=rng.randint(1, 3))
    hi = rng.randint(7, 10)
    return dict(kind=kind, nprob=rng.randint(3, 16), first=rng.randint(0, 10000), norb_lo=rng.randint(5, hi),
                norb_hi=hi)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _integrals(norb, seed, spin=False):
    """The repository's seeded integrals: h1 symmetric N(0, 0.3) with a
    rising diagonal, eri from 2 norb Cholesky-like vectors."""
    rng = np.random.default_rng(seed)
    h1 = rng.normal(0.0, 0.3, (norb, norb))
    h1 = 0.5 * (h1 + h1.T)
    np.fill_diagonal(h1, np.linspace(-2.0, 0.5, norb))
    L = rng.normal(0.0, 0.2, (2 * norb, norb, norb))
    L = 0.5 * (L + L.transpose(0, 2, 1))
    eri = 0.5 * np.einsum("xpq,xrs->pqrs", L, L)
    if spin:
        d = rng.normal(0.0, 0.05, (norb, norb))
        h1 = np.stack([h1 + d + d.T, h1 - d - d.T])
    return h1, eri


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _vector(case, seed):
    """Normalised CI matrix (na strings, nb strings), with c = eta c^T where
    the case asks for it."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))
    shape = (comb(case["norb"], case["na"]), comb(case["norb"], case["nb"]))
    c = torch.randn(shape, generator=g, dtype=torch.float64, device=dev)
    if case.get("eta"):
        c = c + case["eta"] * c.T
    return c.div_(torch.linalg.vector_norm(c))


def _csf_vectors(case, seed):
    dev = _device()
    n = count_all_csfs(case["norb"], case["na"], case["nb"], case["smult"])
    g = torch.Generator(device=dev).manual_seed(int(seed))
    x = torch.randn((case["nvec"], n), generator=g, dtype=torch.float64, device=dev)
    return x / torch.linalg.vector_norm(x, dim=1, keepdim=True)


def _solver(case):
    sol = b200.csf_solver(None, smult=case.get("smult", 1))
    for k, v in SOLVER.items():
        setattr(sol, k, v)
    sol.nroots = case.get("nroots", 1)
    if "smult" in case:
        # a program's solver object has its transformer from its first call on
        sol.norb, sol.nelec = case["norb"], (case["na"], case["nb"])
        sol.check_transformer_cache()
    return sol


def _shapes(case):
    """The uneven batch's orbital and electron numbers, spins and roots."""
    return batched.make_uneven_batch(case["nprob"], case["first"], case["norb_lo"], case["norb_hi"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return dict(case=case, problems=[
            batched.Problem(p.norb, p.nelec, p.smult, p.nroots, *_integrals(p.norb, 1000 * int(seed) + i))
            for i, p in enumerate(_shapes(case))])
    norb, nelec = case["norb"], (case["na"], case["nb"])
    st = dict(case=case, norb=norb, nelec=nelec)
    if kind == "transform":
        st["transformer"] = CSFTransformer(norb, nelec[0], nelec[1], case["smult"])
        st["x"] = _csf_vectors(case, seed)
        return st
    st["solver"] = sol = _solver(case)
    h1, eri = _integrals(norb, seed, case.get("spin_h1", False))
    if kind == "sigma":
        st["h2eff"] = sol.absorb_h1e(h1, eri, norb, nelec, 0.5)
        c = _vector(case, seed)
        st["c"] = c.cpu().numpy() if case["host"] else c
    elif kind == "rdm":
        st["vectors"] = [_vector(case, seed)]
        if case["call"].startswith("trans"):
            st["vectors"].append(_vector(case, seed + 500009))
    elif kind == "diagonal":
        st["h1"], st["eri"] = (torch.as_tensor(x, device=_device()) for x in (h1, eri))
    elif kind == "solve":
        st["h1"], st["eri"] = h1, eri
    else:
        st["h1"] = torch.as_tensor(h1, device=_device()).requires_grad_()
        st["eri"] = torch.as_tensor(eri, device=_device()).requires_grad_()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "batch":
        sol = batched.BatchedCSFSolver(**SOLVER)
        res = sol.kernel(st["problems"])
        # all problems' numbers by kind (energies, CI vectors up to their
        # arbitrary sign, densities)
        return dict(e=np.concatenate([e for e, _, _, _ in res]),
                    ci=np.concatenate([np.abs(c).ravel() for _, ci, _, _ in res for c in ci]),
                    dm1=np.concatenate([d1.ravel() for _, _, r, _ in res for d1, _ in r]),
                    dm2=np.concatenate([d2.ravel() for _, _, r, _ in res for _, d2 in r]))
    norb, nelec = st["norb"], st["nelec"]
    if kind == "sigma":
        return st["solver"].contract_2e(st["h2eff"], st["c"], norb, nelec)
    if kind == "rdm":
        return getattr(st["solver"], case["call"])(*st["vectors"], norb, nelec)
    if kind == "transform":
        t = st["transformer"]
        det = t.vec_csf2det(st["x"], normalize=False)
        return dict(det=det, csf=t.vec_det2csf(det, normalize=False))
    if kind == "diagonal":
        sol = st["solver"]
        hd = sol.make_hdiag(st["h1"], st["eri"], norb, nelec)
        return dict(det=hd, csf=sol.make_hdiag_csf(st["h1"], st["eri"], norb, nelec, hdiag_det=hd))
    if kind == "solve":
        sol = st["solver"]
        e, ci = sol.kernel(st["h1"], st["eri"], norb, nelec)
        cis = ci if isinstance(ci, list) else [ci]
        # CI vectors up to their arbitrary sign
        return dict(e=np.atleast_1d(e), ci=[np.abs(c) for c in cis], rdm=[sol.make_rdm12(c, norb, nelec) for c in cis])
    st["h1"].grad = st["eri"].grad = None
    e = autograd.csf_fci_energy(st["h1"], st["eri"], norb, nelec, case["smult"], case["nroots"],
                                solver=st["solver"])
    e.mean().backward()
    return dict(e=e.detach(), h1=st["h1"].grad, eri=st["eri"].grad)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def _sigma_work(norb, na, nb, eta):
    """One sigma: h2e, the vector and the result; two multiplications and
    additions of the pair matrix per determinant, half of them where the
    vector is (anti)symmetric."""
    ndet = comb(norb, na) * comb(norb, nb)
    npair = norb * (norb + 1) // 2
    return dict(bytes=16.0 * ndet + 8.0 * npair * npair, flops=2.0 * npair * npair * ndet * (0.5 if eta else 1.0))


def _rdm_work(norb, na, nb, nvec, second=True, spin=False):
    """The 2-RDM: every unique pair of excitations once per determinant."""
    ndet = comb(norb, na) * comb(norb, nb)
    n2 = norb * norb
    per = (1.0 if nvec == 2 else 0.5) * 2.0 * n2 * n2 * (2.0 if spin else 1.0) if second else 2.0 * n2
    return dict(bytes=8.0 * nvec * ndet + 8.0 * (n2 * n2 * (3 if spin else 1) if second else n2), flops=per * ndet)


def _solve_work(norb, na, nb, smult, nroots, sigmas_per_root=25):
    """A solve is at least some tens of sigmas for each root, then the
    densities."""
    try:
        ncsf = count_all_csfs(norb, na, nb, smult)
    except RuntimeError:
        ncsf = 0
    k = max(1, min(nroots, ncsf or 1))
    n = 1 if ncsf <= 200 else sigmas_per_root
    s = _sigma_work(norb, na, nb, na == nb)
    r = _rdm_work(norb, na, nb, 1)
    return dict(bytes=k * (n * s["bytes"] + r["bytes"]), flops=k * (n * s["flops"] + r["flops"]))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        tot = dict(bytes=0.0, flops=0.0)
        for p in _shapes(case):
            w = _solve_work(p.norb, p.nelec[0], p.nelec[1], p.smult, p.nroots)
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    norb, na, nb = case["norb"], case["na"], case["nb"]
    if kind == "sigma":
        return _sigma_work(norb, na, nb, case["eta"])
    if kind == "rdm":
        call = case["call"]
        return _rdm_work(norb, na, nb, 2 if call.startswith("trans") else 1, call != "make_rdm1", call.endswith("s"))
    if kind in ("solve", "gradient"):
        return _solve_work(norb, na, nb, case["smult"], case["nroots"])
    ndet = comb(norb, na) * comb(norb, nb)
    ncsf = count_all_csfs(norb, na, nb, case["smult"])
    if kind == "transform":
        # each direction reads one vector and writes the other; the
        # determinant order of the configurations is read once each way
        nvec = case["nvec"]
        fl = 0.0
        for npair in range(max(0, na + nb - norb), min(na, nb) + 1):
            ns = na + nb - 2 * npair
            nconf = comb(norb, npair) * comb(norb - npair, ns)
            fl += 4.0 * nvec * nconf * comb(ns, (ns + na - nb) // 2) * _count_csfs(ns, case["smult"])
        return dict(bytes=2.0 * (8.0 * nvec * (ndet + ncsf) + 4.0 * ndet), flops=fl)
    return dict(bytes=8.0 * ndet + 8.0 * ndet + 8.0 * ncsf + 4.0 * ndet, flops=4.0 * ndet + 2.0 * ncsf)


# ---------------------------------------------------------------------------
# the same results in plain torch and numpy
# ---------------------------------------------------------------------------

def _strings(norb, nelec):
    return np.array(sorted(sum(1 << o for o in occ) for occ in itertools.combinations(range(norb), nelec)),
                    dtype=np.int64)


def _parity(x):
    x = x.copy()
    for s in (32, 16, 8, 4, 2, 1):
        x ^= x >> s
    return x & 1


def _excitations(norb, nelec):
    """E_pq on every string: target address and sign (0 where it vanishes),
    arrays [norb, norb, nstrings] on the device."""
    strs = _strings(norb, nelec)
    rank = np.zeros(1 << norb, dtype=np.int64)
    rank[strs] = np.arange(strs.size)
    to = np.zeros((norb, norb, strs.size), dtype=np.int64)
    sg = np.zeros((norb, norb, strs.size))
    for p in range(norb):
        for q in range(norb):
            ok = (strs >> q) & 1 == 1
            if p != q:
                ok &= (strs >> p) & 1 == 0
            lo, hi = min(p, q), max(p, q)
            between = ((1 << hi) - 1) & ~((1 << (lo + 1)) - 1) if p != q else 0
            s = np.where(_parity(strs & between) == 1, -1.0, 1.0)
            t = np.where(ok, (strs & ~(1 << q)) | (1 << p), strs)
            to[p, q] = rank[t]
            sg[p, q] = np.where(ok, s, 0.0)
    dev = _device()
    return torch.as_tensor(to, device=dev), torch.as_tensor(sg, device=dev)


def _rows(norb, nrow, ncol):
    """Alpha strings handled together: about 4 GB of pair rows."""
    return max(1, min(nrow, int(4e9 / (8.0 * norb * norb * ncol))))


def _t_rows(c, xa, xb, norb, rows, spin=2):
    """T[p, q, J] = <J|E_pq|c> for the determinants of the alpha strings in
    rows (spin 0: alpha excitations, 1: beta, 2: both)."""
    T = torch.zeros((norb, norb, rows.numel(), c.shape[1]), dtype=torch.float64, device=c.device)
    for p in range(norb):
        for q in range(norb):
            if spin != 1:  # <J|E_pq|K> is found from E_qp on J
                T[p, q] += xa[1][q, p][rows][:, None] * c[xa[0][q, p][rows]]
            if spin != 0:
                T[p, q] += c[rows][:, xb[0][q, p]] * xb[1][q, p][None, :]
    return T


def _exact_sigma(case, seed):
    norb, na, nb = case["norb"], case["na"], case["nb"]
    h1, eri = _integrals(norb, seed, case["spin_h1"])
    hc = h1.mean(axis=0) if case["spin_h1"] else h1
    # h1 folded into the two-electron operator through N = sum_k E_kk
    f = (hc - 0.5 * np.einsum("jiik->jk", eri)) / (na + nb + 1e-100)
    h2 = eri.copy()
    for k in range(norb):
        h2[k, k] += f
        h2[:, :, k, k] += f
    c = _vector(case, seed)
    dev = c.device
    h = torch.as_tensor(0.5 * h2, device=dev).reshape(norb * norb, norb * norb)
    xa, xb = _excitations(norb, na), _excitations(norb, nb)
    out = torch.zeros_like(c)
    step = _rows(norb, *c.shape)
    for r0 in range(0, c.shape[0], step):
        rows = torch.arange(r0, min(c.shape[0], r0 + step), device=dev)
        T = _t_rows(c, xa, xb, norb, rows)
        V = (h @ T.reshape(norb * norb, -1)).reshape(T.shape)
        del T
        for p in range(norb):
            for q in range(norb):
                out.index_add_(0, xa[0][p, q][rows], xa[1][p, q][rows][:, None] * V[p, q])
                # <K|E_pq|J> over beta strings, from E_qp on K
                out[rows] += V[p, q][:, xb[0][q, p]] * xb[1][q, p][None, :]
        del V
    if case["spin_h1"]:
        hs = 0.5 * (h1[0] - h1[1])
        rows = torch.arange(c.shape[0], device=dev)
        for p in range(norb):
            for q in range(norb):
                out += hs[p, q] * (xa[1][q, p][:, None] * c[xa[0][q, p]])
                out -= hs[p, q] * (c[:, xb[0][q, p]] * xb[1][q, p][None, :])
    return out.cpu().numpy() if case["host"] else out


def _exact_rdm(case, seed):
    norb, na, nb, call = case["norb"], case["na"], case["nb"], case["call"]
    ket = bra = _vector(case, seed)
    if call.startswith("trans"):
        ket = _vector(case, seed + 500009)
    dev = bra.device
    n2 = norb * norb
    xa, xb = _excitations(norb, na), _excitations(norb, nb)
    spins = (0, 1) if call.endswith("s") else (2,)
    first = {s: torch.zeros(n2, dtype=torch.float64, device=dev) for s in spins}
    pairs = [(s, t) for s in spins for t in spins if s <= t]
    second = {k: torch.zeros((n2, n2), dtype=torch.float64, device=dev) for k in pairs}
    step = max(1, _rows(norb, *bra.shape) // (len(spins) * 2))
    for r0 in range(0, bra.shape[0], step):
        rows = torch.arange(r0, min(bra.shape[0], r0 + step), device=dev)
        tk = {s: _t_rows(ket, xa, xb, norb, rows, s).reshape(n2, -1) for s in spins}
        tb = tk if ket is bra else {s: _t_rows(bra, xa, xb, norb, rows, s).reshape(n2, -1) for s in spins}
        for s in spins:
            first[s] += tk[s] @ bra[rows].reshape(-1)
        for s, t in pairs:
            second[s, t] += tb[s] @ tk[t].T
    # first[s][p, q] = <E_pq>; dm1[p, q] = <q+ p>
    e1 = {s: first[s].reshape(norb, norb) for s in spins}
    dm1 = [e1[s].T.contiguous() for s in spins]
    if call == "make_rdm1":
        return dm1[0]
    dm2 = []
    for s, t in pairs:
        # <E_pq E_rs> = sum_J Tb[q, p, J] Tk[r, s, J]
        g = second[s, t].reshape(norb, norb, norb, norb).permute(1, 0, 2, 3).clone()
        if s == t:
            for q in range(norb):
                g[:, q, q, :] -= e1[s]
        dm2.append(g.contiguous())
    return (tuple(dm1), tuple(dm2)) if len(spins) == 2 else (dm1[0], dm2[0])


def _count_csfs(nspin, smult):
    twos = smult - 1
    if twos > nspin or (nspin - twos) % 2:
        return 0
    n0 = (nspin - twos) // 2
    return comb(nspin, n0) - (comb(nspin, n0 - 1) if n0 else 0)


def _couplings(nspin, smult):
    """Step-up bits of the genealogical paths from spin 0 to smult in the
    engine's order: by the number of paths left of each step up."""
    found = []

    def walk(k, s2, bits):
        if s2 < 0 or s2 + (nspin - k) < smult - 1 or s2 - (nspin - k) > smult - 1:
            return
        if k == nspin:
            found.append(bits)
            return
        walk(k + 1, s2 + 1, bits | 1 << k)
        walk(k + 1, s2 - 1, bits)

    walk(0, 0, 0)
    return np.array(found, dtype=np.int64)


def _spin_functions(nspin, m2, smult):
    """U[det, csf]: Clebsch-Gordan products along the coupling paths, for
    determinants of m2 = na - nb in ascending spin strings."""
    dets = _strings(nspin, (nspin + m2) // 2)[:, None]
    if nspin == 0:
        return torch.ones((1, 1), dtype=torch.float64, device=_device())
    path = _couplings(nspin, smult)[None, :]
    shape = (dets.shape[0], path.shape[1])
    s2 = np.ones(shape, dtype=np.int64)
    m = np.broadcast_to(np.where(dets & 1, 1, -1), shape).copy()
    u = np.ones(shape)
    up_seen = np.broadcast_to(dets & 1, shape).copy()
    neg = np.zeros(shape, dtype=np.int64)
    for k in range(1, nspin):
        sup = np.broadcast_to((path >> k) & 1, shape)
        mup = np.broadcast_to((dets >> k) & 1, shape)
        m += np.where(mup == 1, 1, -1)
        # |S+1/2, M>, |S-1/2, M> from |S, M -+ 1/2> and the new electron
        num = np.where(sup == mup, s2 + m + 1, s2 + 1 - m) / (2.0 * (s2 + 1))
        u *= np.sqrt(np.maximum(num, 0.0))
        neg += (mup == 1) & (sup == 0)
        # alpha operators stand left of the beta ones: a beta electron passes
        # the alpha electrons before it
        neg += np.where(mup == 0, up_seen, 0)
        up_seen += mup
        s2 += np.where(sup == 1, 1, -1)
    return torch.as_tensor(np.where(neg & 1, -u, u), device=_device())


def _blocks(norb, na, nb, smult):
    """Per number of pairs: determinant addresses [conf, det], singly
    occupied orbitals [conf, nspin], signed spin functions."""
    dev = _device()
    ra, rb = (torch.zeros(1 << norb, dtype=torch.int64, device=dev) for _ in range(2))
    for r, ne in ((ra, na), (rb, nb)):
        s = torch.as_tensor(_strings(norb, ne), device=dev)
        r[s] = torch.arange(s.numel(), device=dev)
    nbs = comb(norb, nb)
    for npair in range(max(0, na + nb - norb), min(na, nb) + 1):
        ns = na + nb - 2 * npair
        d = torch.as_tensor(_strings(norb, npair), device=dev)
        s = torch.as_tensor(_strings(norb - npair, ns), device=dev)
        D, S = d[:, None].expand(-1, s.numel()).reshape(-1), s[None, :].expand(d.numel(), -1).reshape(-1)
        somo = torch.zeros((D.numel(), ns), dtype=torch.int64, device=dev)
        free, spin = torch.zeros_like(D), torch.zeros_like(D)
        for o in range(norb):
            open_ = (D >> o) & 1 == 0
            single = open_ & ((S >> free) & 1 == 1)
            if ns:
                hit = torch.nonzero(single).reshape(-1)
                somo[hit, spin[hit]] = o
            spin += single
            free += open_
        dets = torch.as_tensor(_strings(ns, (ns + na - nb) // 2), device=dev)
        a, b = (D[:, None].expand(-1, dets.numel()).clone() for _ in range(2))
        for k in range(ns):
            bit = torch.ones_like(D)[:, None] << somo[:, k:k + 1]
            up = ((dets >> k) & 1)[None, :]
            a += bit * up
            b += bit * (1 - up)
        sign = -1.0 if (npair * (npair - 1) // 2 + npair * max(0, nb - npair)) % 2 else 1.0
        u = None
        if _count_csfs(ns, smult):
            u = sign * _spin_functions(ns, na - nb, smult)
        yield ra[a] * nbs + rb[b], somo, u


def _exact_transform(case, seed):
    norb, na, nb = case["norb"], case["na"], case["nb"]
    x = _csf_vectors(case, seed)
    det = torch.zeros((x.shape[0], comb(norb, na) * comb(norb, nb)), dtype=torch.float64, device=x.device)
    back = []
    at = 0
    for addr, _, u in _blocks(norb, na, nb, case["smult"]):
        if u is None:
            continue
        n = addr.shape[0] * u.shape[1]
        y = x[:, at:at + n].reshape(x.shape[0], addr.shape[0], u.shape[1]) @ u.T
        det[:, addr.reshape(-1)] = y.reshape(x.shape[0], -1)
        back.append((y @ u).reshape(x.shape[0], -1))
        at += n
    return dict(det=det, csf=torch.cat(back, dim=1))


def _exact_diagonal(case, seed):
    norb, na, nb = case["norb"], case["na"], case["nb"]
    h1, eri = _integrals(norb, seed)
    J, K = np.einsum("iijj->ij", eri), np.einsum("ijji->ij", eri)
    oa, ob = ((((_strings(norb, n)[:, None] >> np.arange(norb)) & 1) != 0).astype(float) for n in (na, nb))
    ea, eb = (o @ np.diag(h1) + 0.5 * np.einsum("ai,ij,aj->a", o, J - K, o) for o in (oa, ob))
    hd = torch.as_tensor(ea[:, None] + eb[None, :] + oa @ J @ ob.T, device=_device()).reshape(-1)
    kt = torch.as_tensor(K, device=_device())
    out = []
    for addr, somo, u in _blocks(norb, na, nb, case["smult"]):
        if u is None:
            continue
        v = hd[addr] @ (u * u)
        ns = somo.shape[1]
        dets = _strings(ns, (ns + na - nb) // 2)
        rank = np.zeros(1 << ns, dtype=np.int64)
        rank[dets] = np.arange(dets.size)
        for b in range(1, ns):
            for a in range(b):
                # determinants that differ by exchanging the spins at a and b
                differ = np.nonzero(((dets >> a) ^ (dets >> b)) & 1)[0]
                other = rank[dets[differ] ^ ((1 << a) | (1 << b))]
                z = (u[torch.as_tensor(differ, device=u.device)] * u[torch.as_tensor(other, device=u.device)]).sum(0)
                z = -z if (b - a - 1) & 1 else z
                v += kt[somo[:, a], somo[:, b]][:, None] * z[None, :]
        out.append(v.reshape(-1))
    return dict(det=hd, csf=torch.cat(out))


def _exact_energies(norb, na, nb, smult, nroots, h1, eri):
    """Lowest eigenvalues of the dense CSF Hamiltonian
    sum_pq f_pq E_pq + 1/2 sum (pq|rs) E_pq E_rs, f = h - 1/2 sum_r (pr|rq)."""
    dev = _device()
    xa, xb = _excitations(norb, na), _excitations(norb, nb)
    shape = (xa[0].shape[2], xb[0].shape[2])
    ncsf = count_all_csfs(norb, na, nb, smult)
    u = torch.zeros((shape[0] * shape[1], ncsf), dtype=torch.float64, device=dev)
    at = 0
    for addr, _, f in _blocks(norb, na, nb, smult):
        if f is None:
            continue
        cols = at + torch.arange(addr.shape[0] * f.shape[1], device=dev).reshape(addr.shape[0], 1, f.shape[1])
        u[addr[:, :, None], cols] = f[None]
        at += addr.shape[0] * f.shape[1]
    w = u.reshape(*shape, ncsf)
    eu = torch.stack([(xa[1][q, p][:, None, None] * w[xa[0][q, p]]
                       + xb[1][q, p][None, :, None] * w[:, xb[0][q, p]]).reshape(-1, ncsf)
                      for p in range(norb) for q in range(norb)])
    f1 = torch.as_tensor(h1 - 0.5 * np.einsum("prrq->pq", eri), device=dev).reshape(-1)
    e2 = torch.as_tensor(0.5 * eri, device=dev).reshape(norb * norb, norb * norb)
    H = torch.zeros((ncsf, ncsf), dtype=torch.float64, device=dev)
    for p in range(norb):
        for q in range(norb):
            i = p * norb + q
            H += eu[q * norb + p].T @ (f1[i] * u + torch.tensordot(e2[i], eu, dims=1))
    return torch.linalg.eigvalsh(0.5 * (H + H.T))[:nroots]


def exact(case, seed):
    kind = case["kind"]
    if kind == "sigma":
        return _exact_sigma(case, seed)
    if kind == "rdm":
        return _exact_rdm(case, seed)
    if kind == "transform":
        return _exact_transform(case, seed)
    if kind == "diagonal":
        return _exact_diagonal(case, seed)
    if kind in ("solve", "gradient") and case["norb"] <= 8:
        norb, na, nb = case["norb"], case["na"], case["nb"]
        h1, eri = _integrals(norb, seed)
        k = min(case["nroots"], count_all_csfs(norb, na, nb, case["smult"]))
        e = _exact_energies(norb, na, nb, case["smult"], k, h1, eri)
        if kind == "solve":
            return dict(e=e.cpu().numpy(), ci=None, rdm=None)
        return dict(e=e, h1=None, eri=None)
    # a dense diagonalisation of the larger spaces takes too long
    return None
