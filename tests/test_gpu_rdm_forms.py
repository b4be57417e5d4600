"""The two forms of the density matrices, fused kernel and T slab, at the sizes
where each is taken.

Large spaces against excitation rows formed and contracted by torch on the
device, a block of alpha strings at a time: more links of a spin than a mover
lane holds (48, or 80 with one vector at 13 to 15 orbitals), several passes
over the determinants (two vectors from 12 orbitals on), the fewest stages that
shared memory allows (15 orbitals, alpha-beta), and vectors too wide for it.

Tolerance there: for normalised vectors an element is at most 4, so each of
the ndet additions (in either sum) rounds by at most 4 * 2^-53; taken as
independent these stay within 8 * 4 * 2^-53 * sqrt(ndet)."""
from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _links(norb, nelec):
    """(pq row, target, sign) of every link, each [strings, links], where
    T[pq][J] = <J|E_pq|c> takes sign * c[target]."""
    import torch
    from pyscf_forge_b200.fci import direct_spin1 as D
    t = D.decode_link_table(D.dev_link_table(norb, nelec))
    t = t[:, :nelec * (norb - nelec + 1)]
    t = torch.as_tensor(np.ascontiguousarray(t), device="cuda")
    return t[..., 1] * norb + t[..., 0], t[..., 2], t[..., 3].double()


def _rows(c, r0, r1, n2, la, lb):
    """T of the alpha and of the beta excitations for alpha strings r0..r1-1."""
    import torch
    ta = torch.zeros((n2, r1 - r0, c.shape[1]), dtype=torch.float64, device="cuda")
    tb = torch.zeros_like(ta)
    rows, cols = (torch.arange(n, device="cuda") for n in (r1 - r0, c.shape[1]))
    pq, to, sg = (x[r0:r1] for x in la)
    for l in range(pq.shape[1]):
        ta[pq[:, l], rows] += sg[:, l, None] * c[to[:, l]]
    pq, to, sg = lb
    for l in range(pq.shape[1]):
        tb[pq[:, l], :, cols] += (sg[:, l] * c[r0:r1, to[:, l]]).T
    return ta.reshape(n2, -1), tb.reshape(n2, -1)


def _reference(bra, ket, norb, na, nb):
    """Spin-resolved (dm1a, dm1b), (dm2aa, dm2ab, dm2bb)."""
    import torch
    n, n2 = norb, norb * norb
    la, lb = _links(norb, na), _links(norb, nb)
    step = max(1, (1 << 27) // (n2 * bra.shape[1]))
    g = torch.zeros((3, n2, n2), dtype=torch.float64, device="cuda")
    e = torch.zeros((2, n2), dtype=torch.float64, device="cuda")
    for r0 in range(0, bra.shape[0], step):
        r1 = min(r0 + step, bra.shape[0])
        ka, kb = _rows(ket, r0, r1, n2, la, lb)
        ba, bb = (ka, kb) if bra is ket else _rows(bra, r0, r1, n2, la, lb)
        for i, (x, y) in enumerate(((ba, ka), (ba, kb), (bb, kb))):
            g[i] += x @ y.T
        e[0] += ka @ bra[r0:r1].reshape(-1)
        e[1] += kb @ bra[r0:r1].reshape(-1)
    g = g.reshape(3, n, n, n, n).transpose(1, 2).contiguous()  # <E_pq E_rs>
    e = e.reshape(2, n, n)                                     # <E_pq>
    for q in range(n):
        g[0][:, q, q, :] -= e[0]
        g[2][:, q, q, :] -= e[1]
    return [e[0].T, e[1].T], [g[0], g[1], g[2]]


# (bra is ket) and the space
LARGE = [(False, 12, 4, 3), (True, 13, 7, 6), (False, 13, 7, 6), (True, 14, 7, 7), (False, 14, 7, 7),
         (False, 15, 4, 3), (True, 15, 8, 7), (False, 15, 3, 7), (True, 16, 8, 3), (True, 16, 3, 8), (False, 16, 4, 3)]


@pytest.mark.parametrize("same,norb,na,nb", LARGE)
def test_large_spaces(same, norb, na, nb):
    import torch
    from pyscf_forge_b200.fci import direct_spin1 as D
    gen = torch.Generator(device="cuda").manual_seed(norb * 100 + na * 10 + nb)
    shape = (comb(norb, na), comb(norb, nb))
    v = [torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen) for _ in range(1 if same else 2)]
    v = [x / torch.linalg.vector_norm(x) for x in v]
    bra, ket = v[0], v[-1]
    tol = 32 * 2.0 ** -53 * (shape[0] * shape[1]) ** 0.5
    d1, d2 = _reference(bra, ket, norb, na, nb)
    flat = [x.reshape(-1) for x in (bra, ket)]
    got1, got2 = D.dev_rdm12s(flat[0], None if same else flat[1], norb, (na, nb))
    for x, y in zip(got1 + got2, d1 + d2):
        assert float((x - y).abs().max()) < tol
    m1, m2 = D.dev_rdm12(flat[0], None if same else flat[1], norb, (na, nb))
    assert float((m1 - d1[0] - d1[1]).abs().max()) < 2 * tol
    # <E^a_pq E^b_rs> + <E^b_pq E^a_rs>
    assert float((m2 - d2[0] - d2[2] - d2[1] - d2[1].permute(2, 3, 0, 1)).abs().max()) < 4 * tol


@pytest.mark.parametrize("norb,n", [(13, 5), (16, 4)])
@pytest.mark.parametrize("eta", [1, -1])
def test_large_symmetric_spaces(norb, n, eta):
    """c = +-c^T, which forms the strings' lower triangle alone, with 45 and 52
    links a spin."""
    import torch
    from pyscf_forge_b200.fci import direct_spin1 as D
    gen = torch.Generator(device="cuda").manual_seed(norb)
    c = torch.randn((comb(norb, n),) * 2, dtype=torch.float64, device="cuda", generator=gen)
    c = c + eta * c.T
    c /= torch.linalg.vector_norm(c)
    tol = 32 * 2.0 ** -53 * c.numel() ** 0.5
    d1, d2 = _reference(c, c, norb, n, n)
    m1, m2 = D.dev_rdm12(c.reshape(-1), None, norb, (n, n))
    assert float((m1 - d1[0] - d1[1]).abs().max()) < 2 * tol
    assert float((m2 - d2[0] - d2[2] - d2[1] - d2[1].permute(2, 3, 0, 1)).abs().max()) < 4 * tol


# the form that is faster by a wide margin at these sizes: (bra is ket, space, fused)
FORMS = [(False, 16, 8, 0, False), (False, 14, 7, 0, False), (True, 16, 8, 0, False), (False, 16, 2, 2, False),
         (False, 13, 1, 1, False), (False, 12, 4, 3, True), (False, 16, 3, 3, True), (False, 11, 5, 4, True),
         (True, 16, 3, 2, True), (True, 6, 3, 3, True)]


@pytest.mark.parametrize("same,norb,na,nb,fused", FORMS)
def test_form_taken(same, norb, na, nb, fused):
    """Few columns or few determinants cost the fused kernel whole tiles and
    passes: 1.54 ms against 0.16 at (16, 8, 0) with two vectors."""
    import torch
    from pyscf_forge_b200 import _capi
    from pyscf_forge_b200.fci import direct_spin1 as D
    c = torch.ones(comb(norb, na) * comb(norb, nb), dtype=torch.float64, device="cuda")
    b = c if same else c.clone()
    for call in (D.dev_rdm12, D.dev_rdm12s):
        _capi.profile_enable(True)
        try:
            call(b, None if same else c, norb, (na, nb))
            ran = _capi.profile_report()
        finally:
            _capi.profile_enable(False)
        assert ("k_rdm_fused" in ran, "k_tslab_tile" in ran) == (fused, not fused)


@pytest.mark.parametrize("norb,na,nb", [(2, 1, 0), (5, 0, 1), (6, 3, 1), (8, 1, 4), (7, 4, 3), (12, 1, 3), (16, 1, 1),
                                        (17, 1, 1)])
@pytest.mark.parametrize("same", [True, False])
def test_what_vanishes_is_zero(norb, na, nb, same):
    """The two-particle density of fewer than two electrons, and p+ r+ s q of one
    spin with p = r or q = s, exactly."""
    import torch
    from pyscf_forge_b200.fci import direct_spin1 as D
    gen = torch.Generator(device="cuda").manual_seed(norb)
    c = [torch.randn(comb(norb, na) * comb(norb, nb), dtype=torch.float64, device="cuda", generator=gen) for _ in range(2)]
    _, (aa, _, bb) = D.dev_rdm12s(c[0], None if same else c[1], norb, (na, nb))
    for n, dm2 in ((na, aa), (nb, bb)):
        assert bool(dm2.any()) == (n > 1)
        assert not torch.einsum("pqps->pqs", dm2).any() and not torch.einsum("pqrq->pqr", dm2).any()
    _, dm2 = D.dev_rdm12(c[0], None if same else c[1], norb, (na, nb))
    assert bool(dm2.any()) == (na + nb > 1)
