"""The device-resident Davidson at the edges of its small kernels: 1, 5 and 8
roots (register arrays of 4 and 8), subspaces of 2 to 64 vectors (the most the
eigensolver takes), problems of 1 to hundreds of 256-element chunks in one
batch.  Energies against dense diagonalisation of the oracle's CSF Hamiltonian
(1e-9: the solver stops at an energy change of 1e-11 and a residual of 3e-6,
whose square over gaps above 1e-2 is below 1e-9), large spaces against a
solve with other subspace sizes."""
import numpy as np
import pytest

import restate as R
from conftest import seeded_integrals

pytestmark = pytest.mark.gpu


def _dense(norb, na, nb, smult, h1, eri, k):
    h2 = R.absorb_h1e(h1, eri, norb, (na, nb), 0.5)
    nd = R.num_strings(norb, na) * R.num_strings(norb, nb)
    H = np.array([R.contract_2e(h2, np.eye(nd)[i], norb, (na, nb)).ravel() for i in range(nd)])
    H = R.transform_det2csf(R.transform_det2csf(H, norb, na, nb, smult).T, norb, na, nb, smult)
    return np.linalg.eigvalsh(H)[:k]


@pytest.mark.parametrize("nroots,max_space", [(1, 62), (1, 8), (5, 30), (8, 48), (8, 20)])
def test_small_space_against_dense(nroots, max_space):
    from pyscf_forge_b200 import batched
    norb, na, nb, smult = 6, 3, 3, 1
    h1, eri = seeded_integrals(norb, 2 * norb, 3)
    want = _dense(norb, na, nb, smult, h1, eri, nroots)
    sol = batched.BatchedCSFSolver(conv_tol=1e-11, max_cycle=400, max_space=max_space, pspace_size=0)
    (e, _, _, conv), = sol.kernel([batched.Problem(norb, (na, nb), smult, nroots, h1, eri)], with_rdm=False)
    assert conv
    assert np.abs(e - want).max() < 1e-9


def test_chunk_counts_in_one_batch():
    from pyscf_forge_b200 import batched
    cases = [(5, 3, 2, 2, 2), (8, 4, 4, 1, 3), (9, 5, 4, 2, 1), (10, 5, 5, 3, 4), (11, 6, 5, 2, 2)]
    probs = []
    for i, (n, a, b, s, k) in enumerate(cases):
        h1, eri = seeded_integrals(n, 2 * n, 40 + i)
        probs.append(batched.Problem(n, (a, b), s, k, h1, eri))
    one = batched.BatchedCSFSolver(conv_tol=1e-11, max_cycle=400, max_space=30, pspace_size=0).kernel(probs, with_rdm=False)
    two = [batched.BatchedCSFSolver(conv_tol=1e-11, max_cycle=400, max_space=40, pspace_size=0).kernel([p], with_rdm=False)[0]
           for p in probs]
    for (e1, _, _, c1), (e2, _, _, c2) in zip(one, two):
        assert c1 and c2
        assert np.abs(e1 - e2).max() < 1e-9
