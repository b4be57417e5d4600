"""CPU: the host-driven Davidson with a caller's own preconditioner, its device
products (Gram, combination) replaced by plain torch.  A preconditioner may
hand back the same buffer for every root, as a program that allocates nothing
inside its loop does: the run is then the same as with a fresh result each."""
import numpy as np
import pytest
import torch


@pytest.fixture
def davidson(monkeypatch):
    from pyscf_forge_b200.fci import davidson as mod

    def combine(y, x, coef, beta=0.0):
        c = torch.as_tensor(coef)
        ny = c.shape[0]
        y[:ny] = (beta * y[:ny] if beta else 0.0) + c @ x
        return y

    monkeypatch.setattr(mod, "gram", lambda x, y: x @ y.T)
    monkeypatch.setattr(mod, "combine", combine)
    return mod.davidson


@pytest.mark.parametrize("nroots", [1, 3, 5])
def test_preconditioner_with_one_buffer(davidson, nroots):
    n = 120
    rng = np.random.default_rng(nroots)
    a = rng.normal(scale=0.05, size=(n, n))
    a = torch.as_tensor(a + a.T + np.diag(np.linspace(0.0, 8.0, n)))
    hd = torch.diagonal(a)
    kept = torch.empty(n, dtype=torch.float64)

    def fresh(r, e, x):
        return r / (hd - e + 1e-3)

    def reusing(r, e, x):
        return torch.div(r, hd - e + 1e-3, out=kept)

    runs = []
    for pre in (fresh, reusing):
        stats = {}
        conv, e, x = davidson(lambda v: v @ a, torch.eye(n, dtype=torch.float64)[:nroots], pre, nroots=nroots,
                              max_space=20, stats=stats)
        assert all(conv)
        runs.append((stats["niter"], e, x))
    np.testing.assert_allclose(runs[0][1], np.linalg.eigvalsh(a.numpy())[:nroots], atol=1e-9)
    assert runs[0][0] == runs[1][0]
    assert np.array_equal(runs[0][1], runs[1][1]) and torch.equal(runs[0][2], runs[1][2])
