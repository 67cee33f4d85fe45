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


def _against_frames(cuda, a, m, eps, C=None, b=None, max_iter=4000):
    """Charges of one system against the same system as one of two frames, which takes
    the loop of kernels.  Returns (iterations, largest difference, largest charge)."""
    from admp_b200 import _lib as L
    from admp_b200.qeq import qeq_solve_frames
    q, it, _, st = m._solve(torch.zeros_like(a[2]), *a, C, b, True, eps, max_iter)
    assert st == L.OK
    two = qeq_solve_frames(m, *(x[None].expand(2, *x.shape) for x in a[:2]), *a[2:5],
                           *(x[None].expand(2, *x.shape) for x in a[5:]), C, b, tol=eps, max_iter=max_iter)
    return it, float((q - two[1]).abs().max()), float(q.abs().max())


def _cloud(cuda, n, box, dtype, hard=20.0, seed=1):
    """Random atoms without a pair list: H = 2 hard - 2 kappa ke / sqrt(pi) and a positive
    semidefinite mesh part, so its smallest eigenvalue is above 30 at hard 20."""
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.rand(*s, dtype=torch.float64, generator=g)  # noqa: E731
    none = torch.zeros(0, dtype=torch.float64)
    a = (r(n, 3) * torch.tensor(box), torch.diag(torch.tensor(box, dtype=torch.float64)), r(n) - 0.5,
         torch.full((n,), hard, dtype=torch.float64), torch.ones(n, dtype=torch.float64),
         torch.zeros(0, 2, dtype=torch.long), none, none)
    return tuple(x.to(cuda) if x.dtype == torch.long else x.to(cuda, dtype) for x in a)


# two, four and eight atoms a warp's group; stencils kept and (60,000 with buffers of 88 x 45, 120,000 with lines of
# 128) built anew; lines in several rounds; meshes on either side of the line where the loop of kernels takes over
SIZES = [(4736, [20, 21, 22], torch.float64), (4738, [20, 21, 22], torch.float64), (9472, [20, 21, 22], torch.float32),
         (9480, [20, 21, 22], torch.float64), (60000, [6, 88, 88], torch.float64), (120000, [129, 128, 126], torch.float32),
         (300, [14, 460, 460], torch.float64), (300, [14, 460, 460], torch.float32), (300, [14, 464, 464], torch.float64),
         (150000, [20, 21, 22], torch.float64), (150001, [20, 21, 22], torch.float64)]


@pytest.mark.parametrize("n,kmesh,dtype", SIZES)
def test_sizes(cuda, n, kmesh, dtype):
    from admp_b200.qeq import QEqForceModule
    eps = 1e-14 if dtype == torch.float64 else 1e-10
    a = _cloud(cuda, n, [1.0 * k for k in kmesh], dtype)
    C, b = torch.ones(1, n, dtype=dtype, device=cuda), torch.tensor([0.7], dtype=dtype, device=cuda)
    m = QEqForceModule(6.0, 5e-4, kmesh=kmesh, rspace=False, damping=False)
    _, err, size = _against_frames(cuda, a, m, eps, C, b)
    # each solve is within n eps / 30 of the minimum; FP32 products besides: 1e-6 of the charges a few times over
    assert err < 2 * n * eps / 30 + (1e-12 if dtype == torch.float64 else 1e-5) * size


@pytest.mark.parametrize("n,pairs,kspace", [(300, 10000000, True), (300, 10000001, True), (20000, 50000, False),
                                            (20001, 50000, False)])
def test_pair_lists(cuda, n, pairs, kspace):
    """Both sides of the lines by listed pairs (nearly all of scale 0) and, without a mesh, by atoms."""
    from admp_b200.qeq import QEqForceModule
    a = _cloud(cuda, n, [20.0, 21.0, 22.0], torch.float64)
    g = torch.Generator().manual_seed(2)
    ij = torch.randint(0, n, (pairs, 2), generator=g).to(cuda)
    ds = torch.rand(pairs, dtype=torch.float64, generator=g).to(cuda) * 3 + 3
    bs = torch.zeros(pairs, dtype=torch.float64, device=cuda)
    bs[:n] = 0.5
    bs[-n:] = 0.5
    m = QEqForceModule(6.0, 5e-4, kmesh=[20, 21, 22], kspace=kspace, damping=False)
    _, err, size = _against_frames(cuda, a[:5] + (ij, ds, bs), m, 1e-14)
    # couplings below ke erfc(1.3) / 3 of a few pairs an atom: eigenvalues stay above 20
    assert err < 2 * n * 1e-14 / 20 + 1e-12 * size


@pytest.mark.parametrize("dtype,eps,tol", [(torch.float64, 1e-13, 1e-9), (torch.float32, 1e-7, 1e-4)])
@pytest.mark.parametrize("kspace", [True, False])
@pytest.mark.parametrize("nc", [0, 1, 2, 3, 4])
def test_constraints(cuda, nc, kspace, dtype, eps, tol):
    """Zero to four constraints (the fifth block sum), with and without the mesh, pairs
    and damping on: |r| < 60 eps over eigenvalues of 1 or more, of charges of 0.1 or more."""
    from admp_b200.qeq import QEqForceModule
    a = _water(cuda, dtype)
    n = a[0].shape[0]
    g = torch.Generator().manual_seed(nc)
    C = torch.rand(nc, n, dtype=torch.float64, generator=g).to(cuda, dtype) if nc else None
    b = torch.linspace(-1, 1, nc, dtype=dtype, device=cuda) if nc else None
    m = QEqForceModule(6.0, 5e-4, kmesh=14, kspace=kspace)
    _, err, size = _against_frames(cuda, a[:7] + (a[7].to(dtype),), m, eps, C, b)
    assert err < tol * max(size, 0.1)


@pytest.mark.parametrize("kspace", [True, False])
def test_more_iterations_than_one_launch(cuda, kspace):
    """The state carried from one launch of 128 iterations to the next, several times."""
    from admp_b200.qeq import QEqForceModule
    a = _spread_out(cuda)
    n = a[0].shape[0]
    m = QEqForceModule(6.0, 5e-4, kmesh=16, kspace=kspace, rspace=False, damping=False)
    C, b = torch.ones(1, n, dtype=torch.float64, device=cuda), torch.tensor([0.5], dtype=torch.float64, device=cuda)
    it, err, size = _against_frames(cuda, a, m, 1e-12, C, b)
    assert it > 256
    assert err < 1e-8 * size  # 2 n eps over the smallest eigenvalue 12: 1e-10, of charges of 0.02 or more
    if not kspace:
        w = 1 / (2 * a[3])
        lam = -((a[2] * w).sum() + 0.5) / w.sum()
        q = m._solve(torch.zeros_like(a[2]), *a, C, b, True, 1e-12, 4000)[0]
        assert rel(q, -(a[2] + lam) * w) < 1e-8
