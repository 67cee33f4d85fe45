"""Charge solves of one system (one persistent launch) off the common path."""
import numpy as np
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


def _spread_out(cuda, n=600, hard=(10.0, 1e6)):
    """A diagonal model whose eigenvalues span `hard`: hundreds of iterations."""
    g = torch.Generator().manual_seed(n)
    r = lambda *s: torch.rand(*s, dtype=torch.float64, generator=g)  # noqa: E731
    h = torch.logspace(np.log10(hard[0]), np.log10(hard[1]), n, dtype=torch.float64)[torch.randperm(n, generator=g)]
    none = torch.zeros(0, dtype=torch.float64)
    a = (r(n, 3) * 20, torch.eye(3, dtype=torch.float64) * 20, r(n) - 0.5, h, torch.ones(n, dtype=torch.float64),
         torch.zeros(0, 2, dtype=torch.long), none, none)
    return tuple(x.to(cuda) for x in a)


def test_equal_constraint_rows_do_not_end_a_long_solve(cuda):
    """A singular Gram matrix leaves a status of its own; a solve of more than one
    launch ends with its verdict like a short one.  Diagonal model: q = -(chi + lam) / 2 h."""
    from admp_b200 import _lib as L
    from admp_b200.qeq import QEqForceModule
    a = _spread_out(cuda)
    n = a[0].shape[0]
    m = QEqForceModule(6.0, 5e-4, kspace=False, rspace=False, damping=False)
    one = torch.ones(1, n, dtype=torch.float64, device=cuda)
    b = torch.full((2,), 0.5, dtype=torch.float64, device=cuda)
    q, it, _, st = m._solve(torch.zeros_like(a[2]), *a, torch.cat([one, one]), b, True, 1e-12, 4000)
    assert st == L.OK and it > 128
    w = 1 / (2 * a[3])
    lam = -((a[2] * w).sum() + 0.5) / w.sum()
    # |r| < n eps over the smallest eigenvalue 20: 3e-11 of charges up to 0.1
    assert rel(q, -(a[2] + lam) * w) < 1e-8
