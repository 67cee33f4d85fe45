"""More frames than a launch grid's second dimension holds (65,535): energies and
gradients of the site and damping operators against torch."""
import pytest
import torch

from _gpu_helpers import rel

pytestmark = pytest.mark.gpu

N = 2


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 1e-5)])
@pytest.mark.parametrize("nf", [65535, 65536, 70001])
def test_site(cuda, nf, dtype, tol):
    g = torch.Generator().manual_seed(nf)
    q, chi, h = (torch.rand(nf, N, dtype=dtype, generator=g).to(cuda).requires_grad_(True) for _ in range(3))
    w = torch.rand(nf, dtype=dtype, generator=g).to(cuda)
    e = torch.ops.admp_b200.site(q, chi, h)
    want = (chi * q + h * q * q).sum(1)
    assert rel(e, want) < tol
    for x, y in zip(torch.autograd.grad((e * w).sum(), [q, chi, h]), torch.autograd.grad((want * w).sum(), [q, chi, h])):
        assert rel(x, y) < tol


@pytest.mark.parametrize("pairs", [0, 1])
def test_damping(cuda, pairs):
    from admp_b200.utils import DIELECTRIC
    nf = 70001
    g = torch.Generator().manual_seed(7)
    q, eta = (torch.rand(nf, N, dtype=torch.float64, generator=g).to(cuda).add(0.5).requires_grad_(True) for _ in range(2))
    ds = torch.rand(nf, pairs, dtype=torch.float64, generator=g).to(cuda).add(0.5).requires_grad_(True)
    ij = torch.tensor([[0, 1]], device=cuda)[:pairs].expand(nf, pairs, 2)
    bs = torch.ones(nf, pairs, dtype=torch.long, device=cuda)
    e = torch.ops.admp_b200.damping(ds, q, eta, ij, bs, DIELECTRIC)
    want = (DIELECTRIC * q * q / (2 * torch.pi ** 0.5 * eta)).sum(1)
    if pairs:
        width = torch.sqrt((eta[:, 0] ** 2 + eta[:, 1] ** 2) / 2)
        want = want - DIELECTRIC * torch.erfc(ds[:, 0] / (2 * width)) * q[:, 0] * q[:, 1] / ds[:, 0]
    assert rel(e, want) < 1e-12
    wrt = [q, eta, ds] if pairs else [q, eta]
    for x, y in zip(torch.autograd.grad(e.sum(), wrt), torch.autograd.grad(want.sum(), wrt)):
        assert rel(x, y) < 1e-12
