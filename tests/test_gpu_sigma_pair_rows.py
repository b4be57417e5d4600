"""The row-pair sigma kernel (4 to 13 orbitals) at the edges of its tiles: 10 to
91 pair rows (tiles of 16, a tail of 16 or 8, k-steps in shared memory), 1 to
1716 columns in tiles of 32, fewer tiles than SMs, no electrons, every mode, one
problem, and job tables whose tiles are dealt out in several rounds.

The reference forms D, V = h2e D and the scatter with index operations from
the oracle's link tables.  Tolerance: an element of sigma is a sum of products
over at most nla + nlb links, npair integrals and two values of c; in any order
its rounding error is below (npair + nla + nlb + 4) 2^-53 times the same sum
over absolute values, and the same again for the reference."""
from math import comb

import pytest
import torch

import restate as R

pytestmark = pytest.mark.gpu


def _links(norb, n):
    t = torch.as_tensor(R.link_table(norb, n).reshape(-1, 4), device="cuda")
    hi, lo = torch.maximum(t[:, 0], t[:, 1]), torch.minimum(t[:, 0], t[:, 1])
    src = torch.arange(comb(norb, n), device="cuda").repeat_interleave(n * (norb - n + 1))
    return src, hi * (hi + 1) // 2 + lo, t[:, 2], t[:, 3].double()


def _reference(h2e, c, norb, na, nb, absolute=False):
    f = torch.abs if absolute else (lambda x: x)
    h2e, c = f(h2e), f(c)
    Na, Nb, npair = c.shape[0], c.shape[1], h2e.shape[0]
    out = torch.zeros_like(c)
    a_src, a_pr, a_dst, a_sg = _links(norb, na)
    b_src, b_pr, b_dst, b_sg = _links(norb, nb)
    a_sg, b_sg = f(a_sg), f(b_sg)
    for lo in range(0, Na, 256):  # rows Ja at a time
        hi = min(lo + 256, Na)
        D = torch.zeros((npair, hi - lo, Nb), dtype=c.dtype, device=c.device)
        m = (a_src >= lo) & (a_src < hi)
        D.index_put_((a_pr[m], a_src[m] - lo), a_sg[m, None] * c[a_dst[m]], accumulate=True)
        D = D.transpose(1, 2)
        D.index_put_((b_pr, b_src), b_sg[:, None] * c[lo:hi].T[b_dst], accumulate=True)
        V = torch.einsum("pq,qji->pji", h2e, D)
        out.index_put_((a_dst[m],), a_sg[m, None] * V[a_pr[m], :, a_src[m] - lo], accumulate=True)
        row = torch.zeros((Nb, hi - lo), dtype=c.dtype, device=c.device)
        row.index_put_((b_dst,), b_sg[:, None] * V[b_pr, b_src], accumulate=True)
        out[lo:hi] += row.T
    return out


def _problem(norb, na, nb, eta, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    npair = norb * (norb + 1) // 2
    h = torch.randn((npair, npair), generator=g, dtype=torch.float64, device="cuda")
    c = torch.randn((comb(norb, na), comb(norb, nb)), generator=g, dtype=torch.float64, device="cuda")
    if eta is not None:
        c = c + eta * c.T
    return h + h.T, c


def _check(sigma, h, c, norb, na, nb):
    ref = _reference(h, c, norb, na, nb)
    terms = h.shape[0] + na * (norb - na + 1) + nb * (norb - nb + 1) + 4
    bound = 2 * terms * 2.0 ** -53 * _reference(h, c, norb, na, nb, absolute=True)
    assert bool(((sigma.reshape(c.shape) - ref).abs() <= bound).all())


CASES = [(4, 2, 2, 1), (4, 0, 1, None), (4, 4, 4, None), (5, 3, 2, None), (5, 2, 2, -1), (6, 3, 3, None), (6, 3, 0, None),
         (7, 3, 3, 1), (7, 6, 1, None), (8, 4, 4, -1), (8, 4, 3, None), (9, 4, 4, 1), (9, 2, 7, None), (10, 5, 5, None),
         (10, 1, 0, None), (11, 5, 5, -1), (11, 6, 5, None), (12, 6, 6, 1), (12, 11, 2, None), (13, 7, 6, None),
         (13, 6, 6, 1), (13, 13, 7, None)]


@pytest.mark.parametrize("norb,na,nb,eta", CASES)
def test_one_problem(norb, na, nb, eta):
    from pyscf_forge_b200.fci import direct_spin1 as D
    h, c = _problem(norb, na, nb, eta, seed=norb)
    _check(D.dev_contract_2e(h, c.reshape(-1), norb, (na, nb), eta=eta), h, c, norb, na, nb)


@pytest.mark.parametrize("norb,shapes", [
    (4, [(2, 2, 1), (1, 1, -1), (3, 0, None)] * 5), (6, [(3, 3, 1), (3, 2, None)] * 20), (7, [(4, 3, None), (0, 0, None)]),
    (8, [(4, 4, 1), (4, 4, -1), (8, 1, None)] * 12), (9, [(5, 4, None), (4, 4, 1)] * 3),
    (11, [(5, 5, 1), (2, 1, None), (6, 5, None)] * 2), (12, [(6, 6, 1), (1, 1, -1), (6, 6, None), (7, 6, None)] * 2),
    (13, [(7, 6, None), (2, 2, 1), (6, 6, -1)])])
def test_job_table(monkeypatch, norb, shapes):
    from pyscf_forge_b200 import batched as B
    monkeypatch.setenv("CSFFCI_SIGMA_VARIANT", "4")
    probs = [_problem(norb, na, nb, eta, seed=i) for i, (na, nb, eta) in enumerate(shapes)]
    outs = B.sigma_many([(h, c.reshape(-1), norb, (na, nb), eta) for (h, c), (na, nb, eta) in zip(probs, shapes)])
    for (h, c), (na, nb, _), out in zip(probs, shapes, outs):
        _check(out, h, c, norb, na, nb)
