"""Open-boundary lists whose coordinates are not finite on a whole axis: the
bounds of the cell grid stay crossed, and the grid's size must not be taken
from them.  Refused as any non-finite position is, and the next list is right."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 2048, 2100])  # both cell builds
@pytest.mark.parametrize("axes", [(0,), (2,), (0, 1), (0, 1, 2)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_an_axis_without_a_finite_coordinate_is_refused(cuda, n, axes, value):
    from admp_b200 import _lib as L
    from admp_b200.nblist import TorchNeighborList
    pos = torch.linspace(0, 9, 3 * n, dtype=torch.float64, device=cuda).reshape(n, 3)
    bad = pos.clone()
    bad[:, list(axes)] = value
    with pytest.raises(L.AdmpError):
        TorchNeighborList(5.0)(bad, None)
    pairs = TorchNeighborList(1e-3)(pos, None)
    d = (pos[:, None] - pos[None]).norm(dim=-1) if n < 100 else None
    assert d is None or pairs.shape[0] == int((d < 1e-3).sum()) - n
