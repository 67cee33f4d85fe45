"""Charge solves of one system (one persistent launch) off the common path."""
import numpy as np
import pytest
import torch

from _gpu_helpers import T, rel

pytestmark = pytest.mark.gpu


def _water(cuda, dtype=torch.float64, n_mol=20):
    from admp_b200 import synthetic
    pos, box, chi, hard, eta, _ = synthetic.water_system(n_mol, 13.0, 3)
    from admp_b200.nblist import TorchNeighborList
    p, b = T(pos, cuda, dtype), T(box, cuda, dtype)
    nb = TorchNeighborList(6.0)
    pairs = nb(p, b)
    return p, b, T(chi, cuda, dtype), T(hard, cuda, dtype), T(eta, cuda, dtype), pairs, nb.get_ds(), nb.get_buffer_scales()


@pytest.mark.parametrize("eps", [-1.0, -1e3, 0.0])
def test_a_tolerance_that_nothing_meets_runs_to_the_limit(cuda, eps):
    from admp_b200._lib import NotConvergedWarning
    from admp_b200.qeq import QEqForceModule, pgrad_optimize
    a = _water(cuda)
    n = a[0].shape[0]
    m = QEqForceModule(6.0, 5e-4, kmesh=14, eps=eps, max_iter=5)
    with pytest.warns(NotConvergedWarning):
        pgrad_optimize(m, None, *a, torch.ones(1, n, dtype=torch.float64, device=cuda),
                       torch.zeros(1, dtype=torch.float64, device=cuda))
    assert m.converge_iter == -1
