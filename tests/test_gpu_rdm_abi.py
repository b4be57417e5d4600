"""csffci_rdm12 and csffci_rdm12s through the C ABI with what a caller other
than the Python layer may hand over: link tables that are aligned like their
entries (4 bytes) and whose padding byte was never written, and workspaces of the size
that the slab form alone needs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vectors(norb, na, nb, same, seed):
    import torch
    from math import comb
    rng = np.random.default_rng(seed)
    v = [torch.as_tensor(x / np.linalg.norm(x), device="cuda")
         for x in rng.normal(size=(2, comb(norb, na) * comb(norb, nb)))]
    return (v[0], v[0]) if same else tuple(v)


def _rdms(norb, nelec, bra, ket, la, lb, nbytes=None):
    """(dm1, dm2) and the spin-resolved five, of csffci_rdm12 and rdm12s."""
    import torch
    from pyscf_forge_b200 import _capi
    from pyscf_forge_b200._runtime import ptr, stream
    na, nb = nelec
    out = []
    for call, shapes in (("csffci_rdm12", (2, 4)), ("csffci_rdm12s", (2, 2, 4, 4, 4))):
        dm = [torch.full((norb,) * r, float("nan"), dtype=torch.float64, device="cuda") for r in shapes]
        need = _capi.query(call + "_workspace", norb, na, nb) if nbytes is None else nbytes[call]
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        _capi.call(call, norb, na, nb, ptr(la), ptr(lb), ptr(bra), ptr(ket), *[ptr(d) for d in dm], ptr(ws), need,
                   stream())
        out += dm
    torch.cuda.synchronize()
    return [d.cpu().numpy() for d in out]


def _table(link, pad, offset):
    """The link table with another padding byte, offset bytes into a buffer."""
    import torch
    raw = link.contiguous().view(torch.uint8).reshape(-1, 8).clone()
    raw[:, 7] = pad
    buf = torch.zeros(raw.numel() + 16, dtype=torch.uint8, device="cuda")
    buf[offset:offset + raw.numel()] = raw.reshape(-1)
    return buf[offset:]


@pytest.mark.parametrize("norb,nelec", [(2, (1, 1)), (6, (3, 2)), (8, (4, 4)), (12, (2, 3))])
@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("pad,offset", [(0, 0), (255, 0), (0, 4), (255, 4)])
def test_link_tables_by_their_documented_fields(norb, nelec, same, pad, offset):
    """The same bits as with the library's own tables: the densities read
    address, operator and sign only."""
    from pyscf_forge_b200.fci import direct_spin1 as D
    bra, ket = _vectors(norb, *nelec, same, norb)
    la, lb = (D.dev_link_table(norb, n) for n in nelec)
    want = _rdms(norb, nelec, bra, ket, la, lb)
    got = _rdms(norb, nelec, bra, ket, _table(la, pad, offset), _table(lb, pad, offset))
    for x, y in zip(got, want):
        assert np.array_equal(x, y)


# bytes that the slab form needs: csffci_rdm12, csffci_rdm12s
SLAB_BYTES = {(4, 2, 2): (14592, 28160), (6, 3, 3): (252736, 504448), (8, 4, 4): (5216256, 10300416),
              (16, 1, 0): (1119232, 2237440)}


@pytest.mark.parametrize("space", sorted(SLAB_BYTES))
@pytest.mark.parametrize("same", [True, False])
def test_workspace_of_the_slab_form(space, same):
    """The slab form's workspace is taken, with the same densities to the
    rounding of sums of at most 4900 normalised products; one byte less is
    refused."""
    from pyscf_forge_b200.fci import direct_spin1 as D
    norb, na, nb = space
    bra, ket = _vectors(norb, na, nb, same, norb + 1)
    la, lb = (D.dev_link_table(norb, n) for n in (na, nb))
    least = dict(zip(("csffci_rdm12", "csffci_rdm12s"), SLAB_BYTES[space]))
    want = _rdms(norb, (na, nb), bra, ket, la, lb)
    got = _rdms(norb, (na, nb), bra, ket, la, lb, least)
    for x, y in zip(got, want):
        assert np.abs(x - y).max() < 1e-12
    for call in least:
        with pytest.raises(MemoryError):
            _rdms(norb, (na, nb), bra, ket, la, lb, dict(least, **{call: least[call] - 1}))
