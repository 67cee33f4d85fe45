"""All frames' derivatives in one batched backward, and saved tensors moved by a
hook: the energy operators' backward against one backward per frame."""
import pytest
import torch

from _gpu_helpers import rel
from test_gpu_energy_grads import _frames

pytestmark = pytest.mark.gpu


def _modules():
    from admp_b200.pme import CoulombForceModule
    from admp_b200.qeq import GaussianDampingForceModule, QEqForceModule, SiteForceModule
    return {"coulomb": CoulombForceModule(6.0, 5e-4, kmesh=14), "damping": GaussianDampingForceModule(),
            "site": SiteForceModule(), "qeq": QEqForceModule(6.0, 5e-4, kmesh=14)}


@pytest.mark.parametrize("name", ["coulomb", "damping", "site", "qeq"])
@pytest.mark.parametrize("nf", [1, 3])
def test_batched_backward(cuda, name, nf):
    p, b, q, pairs, ds, bs, par = _frames(cuda, nf, torch.float64)
    e = _modules()[name](p, b, pairs, ds.detach(), bs, par)
    eye = torch.eye(nf, dtype=torch.float64, device=cuda)
    wrt = [q] if name in ("damping", "site") else [q, p]
    many = torch.autograd.grad(e, wrt, eye, is_grads_batched=True, retain_graph=True)
    for k in range(nf):
        one = torch.autograd.grad(e, wrt, eye[k], retain_graph=True)
        for x, y in zip(many, one):
            assert rel(x[k], y) < 1e-14  # the same products
    # the frames do not share a gradient
    assert nf == 1 or not many[0][0, 1:].any()


def test_vectorised_jacobian(cuda):
    p, b, q, pairs, ds, bs, par = _frames(cuda, 3, torch.float64)
    m = _modules()["qeq"]
    f = lambda c: m(p.detach(), b.detach(), pairs, ds.detach(), bs, dict(par, charge=c))  # noqa: E731
    a = torch.autograd.functional.jacobian(f, q.detach(), vectorize=True)
    assert rel(a, torch.autograd.functional.jacobian(f, q.detach())) < 1e-12


def test_saved_gradients_in_another_layout(cuda):
    """A hook that hands the saved gradients back transposed in memory."""
    p, b, q, pairs, ds, bs, par = _frames(cuda, 3, torch.float64)
    m = _modules()["coulomb"]
    w = torch.tensor([1.0, -2.0, 0.5], dtype=torch.float64, device=cuda)
    want = torch.autograd.grad((m(p, b, pairs, ds.detach(), bs, par) * w).sum(), [p, q])
    flip = lambda t: t.transpose(0, -1).contiguous().transpose(0, -1)  # noqa: E731
    with torch.autograd.graph.saved_tensors_hooks(flip, lambda t: t):
        e = m(p, b, pairs, ds.detach(), bs, par)
    got = torch.autograd.grad((e * w).sum(), [p, q])
    for x, y in zip(got, want):
        assert rel(x, y) < 1e-12
