"""The dense Hessian refuses arrays of other lengths than its atoms and pairs,
before anything of them reaches a kernel (so this runs without a GPU too)."""
import pytest
import torch

N, P = 6, 10
ORDER = ("positions", "box", "chi", "hardness", "eta", "pairs", "ds", "scales")
SHAPES = {"positions": (N, 3), "box": (3, 3), "chi": (N,), "hardness": (N,), "eta": (N,), "pairs": (P, 2), "ds": (P,),
          "scales": (P,)}
WRONG = [("hardness", (N - 1,)), ("hardness", (N + 1,)), ("eta", (N - 1,)), ("eta", (1,)), ("ds", (P - 1,)),
         ("ds", (P + 1,)), ("scales", (P - 1,)), ("scales", (0,)), ("pairs", (P, 1)), ("positions", (N, 2)),
         ("box", (3, 2))]


def _call(dev, **wrong):
    from admp_b200.qeq import QEqForceModule
    shapes = dict(SHAPES, **wrong)
    a = {k: torch.rand(s, dtype=torch.float64, device=dev) * 10 for k, s in shapes.items()}
    a["pairs"] = torch.zeros(shapes["pairs"], dtype=torch.long, device=dev)
    m = QEqForceModule(4.0, 1e-4, kmesh=8)
    return m.calc_hessian(*(a[k] for k in ORDER))


@pytest.mark.parametrize("name,shape", WRONG)
def test_other_lengths_are_refused(name, shape):
    with pytest.raises(RuntimeError, match="invalid for input of size"):
        _call("cpu", **{name: shape})


@pytest.mark.gpu
@pytest.mark.parametrize("name,shape", WRONG)
def test_other_lengths_are_refused_on_the_gpu(cuda, name, shape):
    with pytest.raises(RuntimeError, match="invalid for input of size"):
        _call(cuda, **{name: shape})
    assert _call(cuda).shape == (N, N)
