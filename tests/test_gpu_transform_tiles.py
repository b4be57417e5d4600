"""The det <-> CSF transforms and the CSF diagonal at the edges of their
tiles: rows that do not fill 16, columns of 1 to several chunks of 32 and 64,
K split over a CTA's warps, the upper-orbital order of large spaces, blocks
without CSFs, several vectors.

Tolerances: a coefficient is a sum of at most 3432 products of normalised
spin functions and N(0, 1) values; FP64 rounding of such a sum in any order is
below 3432 * 1.1e-16 * (sum of |terms| < 60) = 3e-11, in practice below 1e-13.
The diagonal sums at most 252 terms of weight one in all, of values below
100."""
import numpy as np
import pytest

import restate as R
from conftest import seeded_integrals

pytestmark = pytest.mark.gpu

SMALL = [(4, 2, 1, 2), (5, 2, 2, 3), (6, 5, 1, 5), (7, 3, 3, 7), (8, 4, 4, 1), (8, 5, 3, 5), (9, 5, 4, 2), (9, 3, 3, 3)]


@pytest.mark.parametrize("norb,na,nb,smult", SMALL)
@pytest.mark.parametrize("nvec", [1, 3])
def test_against_oracle(norb, na, nb, smult, nvec):
    import torch
    from pyscf_forge_b200.csf_fci.csfstring import CSFTransformer
    t = CSFTransformer(norb, na, nb, smult)
    rng = np.random.default_rng(norb)
    x = rng.normal(size=(nvec, t.ncsf))
    d = rng.normal(size=(nvec, t.ndet))
    det = t.dev_csf2det(torch.as_tensor(x, device="cuda")).cpu().numpy()
    csf = t.dev_det2csf(torch.as_tensor(d, device="cuda")).cpu().numpy()
    assert np.abs(det - R.transform_det2csf(x, norb, na, nb, smult, reverse=True)).max() < 1e-12
    assert np.abs(csf - R.transform_det2csf(d, norb, na, nb, smult)).max() < 1e-12


@pytest.mark.parametrize("norb,na,nb,smult,nvec", [(12, 6, 6, 1, 3), (13, 7, 6, 2, 3), (14, 8, 6, 5, 1), (14, 7, 7, 3, 2)])
def test_block_by_block(norb, na, nb, smult, nvec):
    """All blocks in one call against one call per block (below the size of
    the upper-orbital order), and back again."""
    import torch
    from pyscf_forge_b200 import _capi
    from pyscf_forge_b200._runtime import ptr, stream
    from pyscf_forge_b200.csf_fci.csfstring import CSFTransformer
    t = CSFTransformer(norb, na, nb, smult)
    g = torch.Generator(device="cuda").manual_seed(norb)
    x = torch.randn((nvec, t.ncsf), generator=g, dtype=torch.float64, device="cuda")
    det = t.dev_csf2det(x)
    one = torch.zeros_like(det)
    blocks = t._c_blocks()
    for v in range(nvec):
        for b in blocks:
            if b.ncsf:
                _capi.call("csffci_csf2det", 1, ptr(x[v]), t.ncsf, ptr(one[v]), t.ndet, t.ndet, ptr(t.csd_mask),
                           (_capi.Block * 1)(b), 1, stream())
    assert float((det - one).abs().max()) < 1e-13
    assert float((t.dev_det2csf(det) - x).abs().max()) < 1e-12


@pytest.mark.parametrize("norb,na,nb", [(12, 6, 6), (14, 7, 7)])
def test_singlet_vectors_are_exactly_symmetric(norb, na, nb):
    import torch
    from pyscf_forge_b200.csf_fci.csfstring import CSFTransformer
    t = CSFTransformer(norb, na, nb, 1)
    x = torch.randn((1, t.ncsf), dtype=torch.float64, device="cuda")
    c = t.dev_csf2det(x).reshape(t.ndeta, t.ndetb)
    assert torch.equal(c, t.spin_parity * c.T)


@pytest.mark.parametrize("norb,na,nb,smult", [(6, 3, 3, 1), (7, 4, 3, 4), (8, 4, 4, 3), (8, 5, 2, 4)])
def test_diagonal(norb, na, nb, smult):
    import pyscf_forge_b200 as P
    h1, eri = seeded_integrals(norb, 2 * norb, norb)
    sol = P.csf_solver(None, smult=smult)
    hd = sol.make_hdiag_csf(h1, eri, norb, (na, nb))
    assert np.abs(hd - R.make_hdiag_csf(h1, eri, norb, (na, nb), smult)).max() < 1e-11
