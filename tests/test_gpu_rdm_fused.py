"""The fused RDM kernel at the edges of its tiles (16 determinants, row
blocks of 8, output tiles of 16 x 8 shared by 12 warps), against the oracle's
excitation vectors: every orbital count it covers, odd and unequal electron
numbers, empty and full spins, general and (anti)symmetric vectors, bra == ket
and bra != ket, spin-free and spin-resolved.

Tolerance: each element is a sum over at most 1e5 determinants of products of
normalised vectors' excitations, |T_a||T_b| <= N^2 <= 900 in all; FP64
rounding of such a sum in any order stays below 1e5 * 1.1e-16 * |T_a||T_b|,
and in practice (random signs) below 1e-12 for the vectors here."""
import numpy as np
import pytest

import restate as R

pytestmark = pytest.mark.gpu

CASES = [(2, 1, 1), (3, 2, 1), (4, 2, 2), (4, 0, 0), (4, 4, 0), (5, 3, 2), (5, 5, 5), (6, 3, 3), (7, 4, 3), (8, 4, 4),
         (9, 2, 3), (10, 3, 3), (11, 3, 2), (12, 2, 2), (13, 2, 1), (14, 2, 2), (15, 2, 2), (16, 2, 2), (16, 1, 2),
         (16, 15, 14)]


def _t_rows(c, norb, na, nb):
    """T^alpha, T^beta [norb*norb, Na, Nb]: <J|E_pq|c> of each spin."""
    la, lb = R.link_table(norb, na), R.link_table(norb, nb)
    ta = np.zeros((norb * norb,) + c.shape)
    tb = np.zeros_like(ta)
    for J in range(c.shape[0]):
        for p, q, K, s in la[J]:
            ta[q * norb + p, J] += s * c[K]
    for J in range(c.shape[1]):
        for p, q, K, s in lb[J]:
            tb[q * norb + p, :, J] += s * c[:, K]
    return ta.reshape(norb * norb, -1), tb.reshape(norb * norb, -1)


def _reference(bra, ket, norb, na, nb):
    n = norb
    ba, bb = _t_rows(bra, n, na, nb)
    ka, kb = _t_rows(ket, n, na, nb)

    def block(x, y, d1):
        g = (x @ y.T).reshape(n, n, n, n).transpose(1, 0, 2, 3).copy()  # <E_pq E_rs>
        if d1 is not None:
            for q in range(n):
                g[:, q, q, :] -= d1
        return g

    ea, eb = ((k @ bra.ravel()).reshape(n, n) for k in (ka, kb))  # <E_pq>
    return (ea.T, eb.T), (block(ba, ka, ea), block(ba, kb, None), block(bb, kb, eb)), block(ba + bb, ka + kb, ea + eb)


@pytest.mark.parametrize("norb,na,nb", CASES)
@pytest.mark.parametrize("mode", ["same", "sym", "anti", "trans"])
def test_rdm12_and_rdm12s(norb, na, nb, mode):
    import torch
    from pyscf_forge_b200.fci import direct_spin1 as D
    if mode in ("sym", "anti") and na != nb:
        pytest.skip("(anti)symmetric vectors need na == nb")
    rng = np.random.default_rng(100 * norb + 10 * na + nb)
    shape = (R.num_strings(norb, na), R.num_strings(norb, nb))
    ket = rng.normal(size=shape)
    if mode == "sym":
        ket = ket + ket.T
    elif mode == "anti":
        ket = ket - ket.T
        if not ket.any():
            pytest.skip("no antisymmetric vector of one string")
    ket /= np.linalg.norm(ket)
    bra = ket
    if mode == "trans":
        bra = rng.normal(size=shape)
        bra /= np.linalg.norm(bra)
    (d1a, d1b), (aa, ab, bb), d2 = _reference(bra, ket, norb, na, nb)
    kd = torch.as_tensor(ket, device="cuda").reshape(-1)
    bd = kd if bra is ket else torch.as_tensor(bra, device="cuda").reshape(-1)
    dm1, dm2 = D.dev_rdm12(bd, None if bd is kd else kd, norb, (na, nb))
    assert np.abs(dm1.cpu().numpy() - d1a - d1b).max() < 1e-12
    assert np.abs(dm2.cpu().numpy() - d2).max() < 1e-12
    s1, s2 = D.dev_rdm12s(bd, None if bd is kd else kd, norb, (na, nb))
    for got, want in zip(s1 + s2, (d1a, d1b, aa, ab, bb)):
        assert np.abs(got.cpu().numpy() - want).max() < 1e-12


def test_repeats_bit_for_bit_and_large_rows():
    """A vector of several thousand tiles (more tiles than CTAs, partial last
    tiles): reruns are equal, and the traces are those of the electrons."""
    import torch
    from pyscf_forge_b200.fci import direct_spin1 as D
    norb, na, nb = 11, 6, 5
    g = torch.Generator(device="cuda").manual_seed(3)
    c = torch.randn(R.num_strings(norb, na) * R.num_strings(norb, nb), generator=g, dtype=torch.float64,
                    device="cuda")
    c /= torch.linalg.vector_norm(c)
    d1, d2 = D.dev_rdm12(c, None, norb, (na, nb))
    e1, e2 = D.dev_rdm12(c, None, norb, (na, nb))
    assert torch.equal(d1, e1) and torch.equal(d2, e2)
    n = na + nb
    assert abs(float(torch.trace(d1)) - n) < 1e-11
    assert abs(float(torch.einsum("iijj->", d2)) - n * (n - 1)) < 1e-10
