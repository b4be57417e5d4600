"""Calls of different sizes from two threads, each on its own stream and with its
own buffers: kernels whose shared memory depends on the space take the same
limit from every call, so none fails because another is being prepared."""
import threading
from math import comb

import pytest

pytestmark = pytest.mark.gpu


def _contract_1e(norb, na, nb):
    import torch
    from pyscf_forge_b200 import _capi
    from pyscf_forge_b200._runtime import ptr
    from pyscf_forge_b200.fci import direct_spin1 as D
    h = torch.randn((norb, norb), dtype=torch.float64, device="cuda")
    c = torch.randn(comb(norb, na) * comb(norb, nb), dtype=torch.float64, device="cuda")
    out = torch.zeros_like(c)
    la, lb = D.dev_link_table(norb, na), D.dev_link_table(norb, nb)
    return lambda s: _capi.call("csffci_contract_1e", norb, na, nb, ptr(h), ptr(h), ptr(la), ptr(lb), ptr(c), ptr(out), s)


def _sigma(norb, na, nb):
    import torch
    from pyscf_forge_b200 import _capi
    from pyscf_forge_b200._runtime import ptr
    from pyscf_forge_b200.fci import direct_spin1 as D
    npair = norb * (norb + 1) // 2
    h = torch.randn((npair, npair), dtype=torch.float64, device="cuda")
    c = torch.randn(comb(norb, na) * comb(norb, nb), dtype=torch.float64, device="cuda")
    out = torch.zeros_like(c)
    la, lb = D.dev_link_table(norb, na), D.dev_link_table(norb, nb)
    return lambda s: _capi.call("csffci_sigma", norb, na, nb, ptr(h), ptr(la), ptr(lb), ptr(c), ptr(out), 0, 1, None, 0, s)


def _rdm(norb, na, nb):
    import torch
    from pyscf_forge_b200 import _capi
    from pyscf_forge_b200._runtime import ptr
    from pyscf_forge_b200.fci import direct_spin1 as D
    c = torch.randn(comb(norb, na) * comb(norb, nb), dtype=torch.float64, device="cuda")
    d1 = torch.empty((norb,) * 2, dtype=torch.float64, device="cuda")
    d2 = torch.empty((norb,) * 4, dtype=torch.float64, device="cuda")
    n = _capi.query("csffci_rdm12_workspace", norb, na, nb)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    la, lb = D.dev_link_table(norb, na), D.dev_link_table(norb, nb)
    return lambda s: _capi.call("csffci_rdm12", norb, na, nb, ptr(la), ptr(lb), ptr(c), ptr(c), ptr(d1), ptr(d2), ptr(ws),
                                n, s)


@pytest.mark.parametrize("make,spaces", [(_contract_1e, [(14, 2, 7), (13, 2, 6)]), (_sigma, [(11, 1, 5), (11, 2, 1)]),
                                         (_rdm, [(12, 1, 6), (12, 2, 2)])])
def test_two_threads(make, spaces):
    import ctypes
    import torch
    calls = [make(*sp) for sp in spaces]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    failed = []

    def work(call, stream):
        try:
            for i in range(3000):
                call(ctypes.c_void_p(stream.cuda_stream))
                if i % 200 == 199:
                    stream.synchronize()
        except Exception as e:  # noqa: BLE001 -- reported by the test
            failed.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
