"""The determinant diagonal on either side of its table rule (rows of at least
128 columns), one to four tables of 7 orbitals, rows that do not fill a block,
few rows (columns split over blocks), different alpha and beta integrals.

Tolerance: a value is a sum of at most (na + nb)^2 + na + nb < 400 integrals of
size below 4; FP64 rounding in any order stays below 400^2 * 4 * 1.1e-16 =
7e-11 and in practice three orders lower; 1e-11 is asked for."""
import numpy as np
import pytest

import restate as R
from conftest import seeded_integrals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,na,nb", [(1, 1, 0), (4, 2, 1), (7, 3, 3), (8, 4, 4), (9, 4, 4), (9, 0, 4), (10, 3, 4),
                                        (14, 7, 7), (14, 1, 7), (15, 13, 6), (16, 3, 4), (20, 2, 3), (22, 0, 4),
                                        (22, 3, 1)])
def test_against_oracle(norb, na, nb):
    from pyscf_forge_b200.fci import direct_spin1 as D
    from pyscf_forge_b200._runtime import eri_pair_matrix
    ha, eri = seeded_integrals(norb, 2 * norb, seed=norb + na)
    hb = ha + 0.1 * np.diag(np.arange(norb))
    got = D.dev_make_hdiag(ha, hb, eri_pair_matrix(eri, norb), norb, (na, nb)).cpu().numpy()
    assert np.abs(got - R.make_hdiag(np.array([ha, hb]), eri, norb, (na, nb))).max() < 1e-11


@pytest.mark.parametrize("norb,na,nb", [(3, 1, 0), (5, 0, 2), (7, 4, 3), (9, 4, 5), (10, 1, 4), (11, 6, 5), (13, 12, 4),
                                        (16, 1, 8)])
def test_contract_1e_against_oracle(norb, na, nb):
    """The one-electron contraction: rows that do not fill a block, columns of
    one to fifty blocks, rows in shared memory past 48 KB and rows that do not
    fit (12870 columns).  At most 72 products of N(0, 1) values and a value
    already there: rounding below 1e-13."""
    import torch
    from math import comb
    from pyscf_forge_b200.fci import direct_spin1 as D
    rng = np.random.default_rng(norb)
    ha, hb = rng.normal(size=(2, norb, norb))
    ci, out = rng.normal(size=(2, comb(norb, na) * comb(norb, nb)))
    got = D.dev_contract_1e(ha, hb, torch.as_tensor(ci, device="cuda"), norb, (na, nb),
                            torch.as_tensor(out, device="cuda")).cpu().numpy()
    assert np.abs(got - out - R.contract_1e_ab(ha, hb, ci, norb, (na, nb)).ravel()).max() < 1e-12


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


@pytest.mark.parametrize("norb,nelec", [(20, 10), (24, 9), (30, 5)])
def test_contract_1e_of_one_column(norb, nelec):
    """A vector of one beta string costs about what one of one alpha string
    does (five times as much by rows), and both give the same."""
    import torch
    from math import comb
    from pyscf_forge_b200.fci import direct_spin1 as D
    rng = np.random.default_rng(norb)
    h = torch.as_tensor(rng.normal(size=(norb, norb)), device="cuda")
    ci = torch.as_tensor(rng.normal(size=comb(norb, nelec)), device="cuda")
    out = [torch.zeros_like(ci) for _ in range(2)]
    D.dev_contract_1e(h, h, ci, norb, (nelec, 0), out[0])
    D.dev_contract_1e(h, h, ci, norb, (0, nelec), out[1])
    assert float((out[0] - out[1]).abs().max()) < 1e-10  # at most 200 products below 30
    assert _us(lambda: D.dev_contract_1e(h, h, ci, norb, (nelec, 0), out[0])) \
        < 2.5 * _us(lambda: D.dev_contract_1e(h, h, ci, norb, (0, nelec), out[1]))


@pytest.mark.parametrize("norb,na,nb", [(18, 7, 1), (20, 6, 0), (20, 1, 6), (40, 0, 4)])
def test_more_than_20000_strings(norb, na, nb):
    """A thread per string, with its orbitals alone."""
    test_against_oracle(norb, na, nb)


def test_cost_of_many_strings():
    """735 471 beta strings: 0.21 ms, 1.6 ms with a warp for each."""
    import torch
    from pyscf_forge_b200.fci import direct_spin1 as D
    h = torch.zeros((24, 24), dtype=torch.float64, device="cuda")
    eri = torch.zeros((300, 300), dtype=torch.float64, device="cuda")
    assert _us(lambda: D.dev_make_hdiag(h, h, eri, 24, (0, 8))) < 700
