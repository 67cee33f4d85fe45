"""One system whose planes are transformed by lines (z and y apart) and the first
one still taken plane by plane: prime and odd lengths, a triclinic cell, energy,
forces, dE/dq and dE/dbox against the oracle, and a product of the charge
Hessian (cached Green's function) against the energy's own gradient."""
import numpy as np
import pytest
import torch

from _gpu_helpers import T, rel

pytestmark = pytest.mark.gpu

MESHES = [[15, 64, 71], [13, 67, 71], [12, 73, 79], [17, 59, 83], [16, 80, 97], [149, 64, 73], [299, 64, 73]]


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-11), (torch.float32, 2e-5)])
@pytest.mark.parametrize("kmesh", MESHES)
def test_energy_and_gradients(cuda, kmesh, dtype, tol):
    from admp_b200.ops import coulomb_pbc
    from oracle import admp_oracle as O
    rng = np.random.default_rng(kmesh[1])
    npdt = np.float64 if dtype == torch.float64 else np.float32
    box = np.array([[11.0, 0, 0], [1.5, 12.0, 0], [-1.0, 0.5, 13.0]]).astype(npdt)
    n = 33
    pos = (rng.random((n, 3)) * 1.5 @ box.astype(np.float64)).astype(npdt)
    q = rng.uniform(-1, 1, n).astype(npdt)
    none = torch.zeros(1, 0, 2, dtype=torch.long, device=cuda)
    empty = torch.zeros(1, 0, dtype=dtype, device=cuda)
    _, comps, g = coulomb_pbc(T(pos[None], cuda, dtype), T(box[None], cuda, dtype), none, empty, empty,
                              T(q[None], cuda, dtype), 0.4, [kmesh], O.DIELECTRIC, False, True, False, 2, True)
    p64, b64, q64 = pos.astype(np.float64), box.astype(np.float64), q.astype(np.float64)
    want = O.pme_recip(p64, b64, q64, 0.4, np.array(kmesh))
    es, en = O.pme_self(q64, 0.4), O.pme_non_neutral(q64, b64, 0.4)
    # FP32: as in the stencil tests, sums of 216 single-precision terms and transforms: ~1e-5
    assert abs(float(comps[0, 1]) - want["E"]) <= tol * max(abs(want["E"]), 1.0)
    ref = {"pos": want["dpos"], "q": want["dq"] + es[1] + en[1], "box": want["dbox"] + en[2]}
    for name, r in ref.items():
        err = np.abs(g[name][0].double().cpu().numpy() - r).max()
        assert err < 10 * tol * max(np.abs(r).max(), 1.0), (name, err)


@pytest.mark.parametrize("kmesh", MESHES)
def test_hessian_product(cuda, kmesh):
    """H q of the reciprocal, self and non-neutral parts is dE/dq (E is quadratic in q)."""
    from admp_b200 import _lib as L
    from admp_b200.ops import coulomb_pbc
    rng = np.random.default_rng(kmesh[2])
    n = 40
    p, b = T(rng.random((n, 3)) * 12, cuda), T(np.diag([12.0, 13.0, 12.5]), cuda)
    q = T(rng.normal(size=n), cuda)
    none, empty = torch.zeros(1, 0, 2, dtype=torch.long, device=cuda), torch.zeros(1, 0, dtype=torch.float64, device=cuda)
    _, _, g = coulomb_pbc(p[None], b[None], none, empty, empty, q[None], 0.4, [kmesh], 14.4, False, True, False, 2, True)
    lib = L.load()
    kp, _k = L.int3(kmesh)
    out, hard = torch.empty_like(q), torch.zeros_like(q)
    ws = L.workspace(lib.admp_qeq_workspace_size(L.F64, n, 0, kp, 0), cuda)
    L.check(lib.admp_qeq_hvp(L.F64, L.QEQ_KSPACE, n, kp, L.ptr(p), L.ptr(b), 0, None, None, None, L.ptr(hard), None, 0.4,
                             14.4, L.ptr(q), L.ptr(out), L.ptr(ws), ws.numel(), L.stream_of(cuda)))
    assert rel(out, g["q"][0]) < 1e-12
