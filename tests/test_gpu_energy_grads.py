"""Gradients of the energy operators: int64 and floating buffer scales, several
frames with their own weights, and the product rule through a dL/dE that itself
needs a gradient."""
import numpy as np
import pytest
import torch

from _gpu_helpers import T, rel

pytestmark = pytest.mark.gpu


def _frames(cuda, nf, dtype):
    from admp_b200 import synthetic
    from admp_b200.nblist import frame_pair_lists
    pos, box, chi, hard, eta, _ = synthetic.water_frames(nf, 5, n_mol=20, box_len=13.0)
    p, b = T(pos, cuda, dtype, grad=True), T(box, cuda, dtype, grad=True)
    q = T(np.random.default_rng(1).normal(size=pos.shape[:2]), cuda, dtype, grad=True)
    pairs, ds, bs = frame_pair_lists(p, b, 6.0)
    par = {"charge": q, "chi": T(chi, cuda, dtype).expand(nf, -1), "hardness": T(hard, cuda, dtype).expand(nf, -1),
           "eta": T(eta, cuda, dtype).expand(nf, -1)}
    return p, b, q, pairs, ds, bs, par


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("nf", [1, 3])
def test_scales_and_frame_weights(cuda, nf, dtype):
    from admp_b200.qeq import QEqForceModule
    m = QEqForceModule(6.0, 5e-4, kmesh=14)
    p, b, q, pairs, ds, bs, par = _frames(cuda, nf, dtype)
    w = torch.linspace(0.5, 2.0, nf, dtype=dtype, device=cuda)
    out = []
    for scales in (bs, bs.to(dtype)):
        e = m(p, b, pairs, ds, scales, par)
        out.append([e.detach(), *torch.autograd.grad((e * w).sum(), [p, b, q], retain_graph=True)])
    tol = 1e-12 if dtype == torch.float64 else 1e-4  # atomics in another order
    for x, y in zip(*out):
        assert rel(x, y) < tol
    # each frame's gradient scales with its own weight
    one = torch.autograd.grad(m(p, b, pairs, ds, bs, par).sum(), q)[0]
    assert rel(out[0][3], one * w[:, None]) < tol


def test_gradient_of_a_weighted_force(cuda):
    """F = -d(lam E)/dr with create_graph: dF/dlam is the force itself."""
    from admp_b200.pme import CoulombForceModule
    m = CoulombForceModule(6.0, 5e-4, kmesh=14)
    p, b, q, pairs, ds, bs, par = _frames(cuda, 1, torch.float64)
    lam = torch.tensor(1.7, dtype=torch.float64, device=cuda, requires_grad=True)
    e = m(p, b, pairs, ds.detach(), bs, par)
    f = torch.autograd.grad((lam * e).sum(), p, create_graph=True)[0]
    g = torch.autograd.grad(f.square().sum(), lam)[0]
    assert abs(float(g) - 2 * float(f.detach().square().sum()) / 1.7) < 1e-9 * abs(float(g))
