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
