"""The Gram and combination kernels of the host-driven Davidson at the edges of
their forms: chunks of 2048 elements, rows split over blocks (1 to 64) and too
many for it (65), one to four narrow rows on either side; combinations below
and above 606208 elements, ragged ends, one to five rows.

Tolerance: a sum of n products in any order is within n 2^-53 times the sum of
their absolute values (beta y counts as one more), for the reference as well."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _draw(*shape):
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(sum(shape)))


@pytest.mark.parametrize("n", [1, 2047, 2049, 70001, 1300000])
@pytest.mark.parametrize("nx,ny", [(1, 1), (5, 1), (1, 6), (9, 2), (13, 3), (3, 64), (64, 4), (65, 2)])
def test_gram(n, nx, ny):
    from pyscf_forge_b200.fci.davidson import gram
    x, y = _draw(nx, n + 3)[:, :n], _draw(ny, n)
    bound = 2 * n * 2.0 ** -53 * (x.abs() @ y.abs().T)
    assert bool(((gram(x, y) - x @ y.T).abs() <= bound).all())


@pytest.mark.parametrize("n", [1, 255, 606207, 606208, 700001])
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 1), (9, 2), (4, 3), (14, 5)])
@pytest.mark.parametrize("beta", [0.0, -0.5])
def test_combine(n, nx, ny, beta):
    from pyscf_forge_b200.fci.davidson import combine
    x, y, c = _draw(nx, n + 1)[:, :n], _draw(ny, n), _draw(ny, nx)
    ref, bound = beta * y + c @ x, 2 * (nx + 2) * 2.0 ** -53 * (abs(beta) * y.abs() + c.abs() @ x.abs())
    assert bool(((combine(y.clone(), x, c, beta=beta) - ref).abs() <= bound).all())


@pytest.mark.parametrize("n", [4097, 70001])
@pytest.mark.parametrize("nx,ny", [(7, 1), (2, 9)])
def test_gram_in_half_the_workspace(n, nx, ny):
    """One or two narrow vectors: half the blocks' worth of workspace is
    enough, less is refused."""
    from pyscf_forge_b200 import _capi
    from pyscf_forge_b200._runtime import ptr, stream
    x, y = _draw(nx, n), _draw(ny, n)
    out = torch.empty((nx, ny), dtype=torch.float64, device="cuda")
    least = -(-n // 4096) * nx * ny * 8
    work = torch.empty(least, dtype=torch.uint8, device="cuda")
    args = (nx, ptr(x), n, ny, ptr(y), n, n, ptr(out), ptr(work))
    _capi.call("csffci_gram", *args, least, stream())
    assert bool(((out - x @ y.T).abs() <= 2 * n * 2.0 ** -53 * (x.abs() @ y.abs().T)).all())
    with pytest.raises(MemoryError):
        _capi.call("csffci_gram", *args, least - 8, stream())
