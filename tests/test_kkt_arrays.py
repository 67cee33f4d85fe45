"""The dense charge solve takes its arrays by pointer only where their sizes and
devices are what the kernel indexes; every other form goes to the bordered
system, which solves it (host arrays) or raises torch's own error."""
import pytest
import torch

from _gpu_helpers import rel

N = 12
WRONG = {"narrow C": dict(C=(1, N - 1)), "wide C": dict(C=(1, N + 5)), "short chi": dict(chi=(N - 3,)),
         "long chi": dict(chi=(N + 1,)), "empty b": dict(b=(0,)), "two b": dict(b=(2,)),
         "short chi, no C": dict(chi=(N - 3,), C=None), "oblong H": dict(H=(N, N - 1))}


def _arrays(dev, H=(N, N), chi=(N,), C=(1, N), b=(1,)):
    g = torch.Generator().manual_seed(3)
    r = lambda shape: torch.rand(shape, dtype=torch.float64, generator=g)  # noqa: E731
    h = r(H)
    h = h @ h.T + torch.eye(N, dtype=torch.float64) if H == (N, N) else h
    out = [h, r(chi), None if C is None else r(C) + 0.5, None if C is None else r(b)]
    return [None if t is None else t.to(dev) for t in out]


def _refused(dev, wrong):
    from admp_b200 import _lib as L
    from admp_b200.qeq import _kkt
    with pytest.raises((RuntimeError, IndexError), match=r"(?i)size|shape|square|expected") as e:
        _kkt(*_arrays(dev, **wrong))
    assert not isinstance(e.value, L.AdmpError)  # torch's own, before anything of this library is launched


@pytest.mark.parametrize("wrong", list(WRONG))
def test_refused(wrong):
    _refused("cpu", WRONG[wrong])


@pytest.mark.parametrize("C", [None, (1, N)])
def test_host_arrays_are_solved(C):
    from admp_b200.qeq import _kkt
    h, chi, c, b = _arrays("cpu", C=C)
    q = _kkt(h, chi, c, b)
    # gradient of the energy along the constraint's null space vanishes; condition numbers below 1e3
    g = h @ q + chi
    if c is not None:
        assert abs(float(c @ q - b)) < 1e-11
        g = g - c[0] * (c[0] @ g) / (c[0] @ c[0])
    assert float(g.abs().max()) < 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("wrong", list(WRONG))
def test_refused_on_the_gpu(cuda, wrong):
    _refused(cuda, WRONG[wrong])


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 2, 3])
def test_mixed_devices_are_refused(cuda, k):
    from admp_b200.qeq import _kkt
    a = _arrays(cuda)
    a[k] = a[k].cpu()
    with pytest.raises(RuntimeError):
        _kkt(*a)
    a = _arrays(cuda)
    assert rel(_kkt(*a), _kkt(*_arrays("cpu"))) < 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("constrained", [True, False])
def test_charges_and_fermi_level_differentiate(cuda, constrained):
    """dq/dchi, dq/db and dE_fermi/dchi of solve_matrix_inversion against the inverse
    of the bordered matrix (condition number below 1e4: relative 1e-9)."""
    from admp_b200 import synthetic
    from admp_b200.nblist import TorchNeighborList
    from admp_b200.qeq import QEqForceModule
    pos, box, chi, hard, eta, _ = synthetic.water_system(11, 12.5, 3)
    t = lambda x: torch.tensor(x, dtype=torch.float64, device=cuda)  # noqa: E731
    p, bx, c, h, e = t(pos), t(box), t(chi).requires_grad_(True), t(hard), t(eta)
    n = len(pos)
    C = torch.linspace(0.5, 1.5, n, dtype=torch.float64, device=cuda)[None] if constrained else None
    b = t([0.3]).requires_grad_(True) if constrained else None
    nb = TorchNeighborList(6.0)
    pairs = nb(p, bx)
    m = QEqForceModule(6.0, 5e-4, kmesh=14)
    args = (p, bx, c, h, e, pairs, nb.get_ds(), nb.get_buffer_scales())
    _, q, _, fermi = m.solve_matrix_inversion(*args, C, b)
    w = torch.linspace(-1, 1, n, dtype=torch.float64, device=cuda)
    got = torch.autograd.grad((w * q).sum() + fermi, [c, b] if constrained else [c])
    H = m.calc_hessian(*args)
    k = 1 if constrained else 0
    A = torch.zeros(n + k, n + k, dtype=torch.float64, device=cuda)
    A[:n, :n] = H
    if constrained:
        A[n:, :n], A[:n, n:] = C, C.T
    inv = torch.linalg.inv(A)
    dq = w + H.sum(0) / n  # d(w.q + fermi)/dq
    assert rel(got[0], 1.0 / n - inv[:n, :n].T @ dq) < 1e-9
    if constrained:
        assert rel(got[1], inv[:n, n:].T @ dq) < 1e-9
