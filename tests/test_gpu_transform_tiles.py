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


# vectors dealt out among the warps, K split over a CTA, launches of some of
# the vectors, the upper-orbital order and blocks without CSFs
MANY = [(6, 3, 3, 1, 256), (7, 4, 3, 4, 17), (8, 4, 4, 3, 64), (10, 5, 5, 1, 140), (11, 8, 3, 6, 33), (12, 8, 4, 9, 40),
        (13, 7, 6, 2, 9), (12, 6, 6, 3, 15), (18, 3, 15, 17, 20)]


@pytest.mark.parametrize("norb,na,nb,smult,nvec", MANY)
def test_many_vectors_as_one_by_one(norb, na, nb, smult, nvec):
    """A vector's coefficients do not depend on those beside it, to the bit."""
    import torch
    from pyscf_forge_b200.csf_fci.csfstring import CSFTransformer
    t = CSFTransformer(norb, na, nb, smult)
    g = torch.Generator(device="cuda").manual_seed(nvec)
    x = torch.randn((nvec, t.ncsf), generator=g, dtype=torch.float64, device="cuda")
    d = torch.randn((nvec, t.ndet), generator=g, dtype=torch.float64, device="cuda")
    det, csf = t.dev_csf2det(x), t.dev_det2csf(d)
    for v in range(nvec):
        assert torch.equal(det[v], t.dev_csf2det(x[v:v + 1])[0])
        assert torch.equal(csf[v], t.dev_det2csf(d[v:v + 1])[0])


def _us(call):
    """Device time of one call, microseconds (the least of five)."""
    import torch
    call()
    best = float("inf")
    for _ in range(5):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        torch.cuda.synchronize()
        e[0].record()
        for _ in range(10):
            call()
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]) * 100)
    return best


@pytest.mark.parametrize("norb,na,nb,smult", [(6, 3, 3, 3), (7, 4, 3, 4), (10, 3, 3, 3)])
def test_many_vectors_fill_the_gpu(norb, na, nb, smult):
    """256 vectors of a space far too small for the GPU cost a few times one,
    not the vectors one after another (25 to 30 times)."""
    import torch
    from pyscf_forge_b200.csf_fci.csfstring import CSFTransformer
    t = CSFTransformer(norb, na, nb, smult)
    x = torch.zeros((256, t.ncsf), dtype=torch.float64, device="cuda")
    d = torch.zeros((256, t.ndet), dtype=torch.float64, device="cuda")
    assert _us(lambda: t.dev_csf2det(x)) < 8 * _us(lambda: t.dev_csf2det(x[:1]))
    assert _us(lambda: t.dev_det2csf(d)) < 8 * _us(lambda: t.dev_det2csf(d[:1]))


@pytest.mark.parametrize("norb,na,nb,smult,nvec", [(18, 15, 3, 17, 16), (20, 17, 3, 19, 16), (16, 12, 4, 13, 8)])
def test_determinants_without_csfs(norb, na, nb, smult, nvec):
    """Most determinants of a high-spin space are in configurations without
    CSFs: zeros in the result, at the cost of a few passes over it (by their own
    tasks 13 to 16)."""
    import torch
    from pyscf_forge_b200.csf_fci.csfstring import CSFTransformer
    t = CSFTransformer(norb, na, nb, smult)
    x = torch.ones((nvec, t.ncsf), dtype=torch.float64, device="cuda")
    det = t.dev_csf2det(x)
    for b in t._blocks:
        rows = t.csd_mask[b["csd_offset"]:b["csd_offset"] + b["nconf"] * b["ndet"]].long()
        if b["ncsf"] == 0:
            assert not det[:, rows].any()
        else:
            assert det[:, rows].any()
    assert _us(lambda: t.dev_csf2det(x)) < 11 * _us(lambda: det.zero_())


@pytest.mark.parametrize("norb,na,nb,smult", [(10, 5, 5, 1), (12, 6, 6, 3), (12, 7, 4, 4), (14, 7, 7, 3), (16, 4, 4, 1)])
def test_diagonal_of_large_spaces(norb, na, nb, smult):
    """Up to 14 open shells, 91 exchange pairs and 1001 CSFs a configuration:
    sum_x U[x,k]^2 hdiag[x] + sum_ab K(a,b) Z[ab,k] on 40 configurations of every
    block, the open shells taken from the strings of a determinant.

    Tolerance: both sums have at most 3432 + 91 terms, of weights that add up to
    1 and 91 at most, of N(0, 1) values (below 8): rounding below
    4000 * 92 * 8 * 1.1e-16 = 4e-10 in any order, 1e-11 and less in practice."""
    import torch
    from pyscf_forge_b200 import _capi
    from pyscf_forge_b200._runtime import ptr, stream
    from pyscf_forge_b200.csf_fci.csfstring import CSFTransformer
    t = CSFTransformer(norb, na, nb, smult)
    g = torch.Generator(device="cuda").manual_seed(norb)
    npair = norb * (norb + 1) // 2
    hd = torch.randn(t.ndet, generator=g, dtype=torch.float64, device="cuda")
    eri = torch.randn((npair, npair), generator=g, dtype=torch.float64, device="cuda")
    got = t.dev_hdiag_csf(hd, eri)
    strs = []
    for n, count in ((na, t.ndeta), (nb, t.ndetb)):
        s = torch.empty(count, dtype=torch.int64, device="cuda")
        _capi.call("csffci_gen_strings", norb, n, ptr(s), stream())
        strs.append(s)
    kk = eri.diagonal()
    for b in t._blocks:
        if not b["ncsf"]:
            continue
        conf = torch.randint(b["nconf"], (min(40, b["nconf"]),), generator=g, device="cuda")
        rows = conf[:, None] * b["ndet"] + torch.arange(b["ndet"], device="cuda")
        dets = t.csd_mask[b["csd_offset"] + rows].long()
        want = hd[dets] @ b["umat"].reshape(b["ndet"], b["ncsf"]) ** 2
        if b["nspin"] >= 2:
            open_ = strs[0][dets[:, 0] // t.ndetb] ^ strs[1][dets[:, 0] % t.ndetb]
            bits = (open_[:, None] >> torch.arange(norb, device="cuda")) & 1
            somo = bits.nonzero()[:, 1].reshape(len(conf), b["nspin"])
            ab = [(i, j) for j in range(b["nspin"]) for i in range(j)]
            lo, hi = (somo[:, [p[q] for p in ab]] for q in (0, 1))
            want = want + kk[hi * (hi + 1) // 2 + lo] @ b["zmat"]
        cols = b["csf_offset"] + conf[:, None] * b["ncsf"] + torch.arange(b["ncsf"], device="cuda")
        assert float((got[cols] - want).abs().max()) < 4e-10
