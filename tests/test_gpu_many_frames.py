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
    from admp_b200 import qeq  # noqa: F401  (loads the operators)
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
    from admp_b200 import qeq  # noqa: F401
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


@pytest.mark.parametrize("nf", [8, 9, 256, 257])
def test_coulomb_frames(cuda, nf):
    """Either form of the system table and several calls' worth of frames: each frame's
    energy and gradients are those of the frame by itself (atomics in another order)."""
    from admp_b200.pme import CoulombForceModule
    g = torch.Generator().manual_seed(nf)
    pos = (torch.rand(nf, 5, 3, dtype=torch.float64, generator=g) * 9).to(cuda).requires_grad_(True)
    q = torch.rand(nf, 5, dtype=torch.float64, generator=g).to(cuda).requires_grad_(True)
    box = (torch.eye(3, dtype=torch.float64) * torch.linspace(9, 11, nf, dtype=torch.float64)[:, None, None]).to(cuda)
    ij = torch.tensor([[0, 1], [2, 3]], device=cuda).expand(nf, 2, 2)
    ds = torch.full((nf, 2), 2.5, dtype=torch.float64, device=cuda)
    bs = torch.ones(nf, 2, dtype=torch.long, device=cuda)
    m = CoulombForceModule(4.0, 1e-4, kmesh=10, slab_corr=True)
    e = m(pos, box, ij, ds, bs, {"charge": q})
    gp, gq = torch.autograd.grad(e.sum(), [pos, q])
    for f in {0, 1, nf // 2, nf - 2, nf - 1}:
        p1, q1 = pos[f].detach().requires_grad_(True), q[f].detach().requires_grad_(True)
        e1 = m(p1, box[f], ij[f], ds[f], bs[f], {"charge": q1})
        g1 = torch.autograd.grad(e1.sum(), [p1, q1])
        assert rel(e[f], e1) < 1e-12 and rel(gp[f], g1[0]) < 1e-11 and rel(gq[f], g1[1]) < 1e-11
