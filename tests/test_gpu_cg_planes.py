"""Charges of one system's solve (one persistent kernel, whole x planes or single
lines in its z and y transforms) against the same system as one of two frames,
which takes a kernel per transform: odd and prime planes, the largest plane a
block takes by itself, the first above it, more planes than blocks.

Either solve stops at |r| < N eps, so the charges differ by 2 N eps over the
smallest eigenvalue (1 eV / e^2 or more) at most, of 0.2 e or more."""
import pytest
import torch

from _gpu_helpers import T, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmesh", [[14, 15, 17], [14, 64, 64], [14, 63, 128], [14, 64, 130], [150, 14, 15]])
@pytest.mark.parametrize("dtype,eps,tol", [(torch.float64, 1e-12, 1e-8), (torch.float32, 1e-6, 1e-3)])
def test_planes_and_lines(cuda, kmesh, dtype, eps, tol):
    from admp_b200 import synthetic
    from admp_b200.nblist import frame_pair_lists
    from admp_b200.qeq import QEqForceModule, pgrad_optimize, qeq_solve_frames
    pos, box, chi, hard, eta, _ = synthetic.water_frames(2, 3, n_mol=20, box_len=13.0, jitter=0.0)
    p, b = T(pos, cuda, dtype), T(box, cuda, dtype)
    chi, hard, eta = (T(v, cuda, dtype) for v in (chi, hard, eta))
    C = torch.ones(1, p.shape[1], dtype=dtype, device=cuda)
    m = QEqForceModule(6.0, 5e-4, kmesh=kmesh, eps=eps, max_iter=500)
    pairs, ds, bs = frame_pair_lists(p, b, 6.0)
    q = qeq_solve_frames(m, p, b, chi, hard, eta, pairs, ds, bs, C)
    _, one = pgrad_optimize(m, None, p[0], b[0], chi, hard, eta, pairs[0], ds[0], bs[0], C, T([0.0], cuda, dtype))[:2]
    assert rel(one, q[0]) < tol
