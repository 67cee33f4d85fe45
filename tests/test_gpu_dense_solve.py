"""Charges of a dense Hessian: the one-kernel Cholesky against the bordered LU, at
the edges of its tiles of 32 and of its range, with one constraint and none, and
a matrix that is not positive definite.

H = G G^T / n + I / 2 has a condition number below 10: forward errors of either
solve stay under 10 n eps, 100 n eps is asked for."""
import pytest
import torch

from _gpu_helpers import rel

pytestmark = pytest.mark.gpu


def _system(n, dev):
    g = torch.Generator().manual_seed(n)
    G = torch.randn(n, n, dtype=torch.float64, generator=g)
    H = G @ G.T / n + 0.5 * torch.eye(n, dtype=torch.float64)
    return ((H + H.T) / 2).to(dev), torch.randn(n, dtype=torch.float64, generator=g).to(dev)


def _lu(H, chi, C, b):
    n = H.shape[0]
    if C is None:
        return torch.linalg.solve(H, -chi)
    A = torch.cat([torch.cat([H, C.T], 1), torch.cat([C, torch.zeros(1, 1, dtype=H.dtype, device=H.device)], 1)], 0)
    return torch.linalg.solve(A, torch.cat([-chi, b]))[:n]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 429, 1024, 1025])
@pytest.mark.parametrize("constrained", [True, False])
def test_dense_solve(cuda, n, constrained):
    from admp_b200.qeq import _kkt
    H, chi = _system(n, cuda)
    C = torch.linspace(0.5, 1.5, n, dtype=torch.float64, device=cuda)[None] if constrained else None
    b = torch.tensor([0.7], dtype=torch.float64, device=cuda) if constrained else None
    assert rel(_kkt(H, chi, C, b), _lu(H, chi, C, b)) < 100 * n * 2.3e-16


@pytest.mark.parametrize("k", [0, 40, 99])
def test_indefinite_takes_the_lu(cuda, k):
    from admp_b200.qeq import _kkt
    H, chi = _system(100, cuda)
    H[k, k] = -3.0
    assert rel(_kkt(H, chi, None, None), _lu(H, chi, None, None)) < 1e-11
