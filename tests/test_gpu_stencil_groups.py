"""Spread and gather at the edges of their eight-atom groups and of the rule
that lets a gather's warp take several groups: energies, forces, dE/dq and
dE/dbox of batches of small systems against the oracle."""
import numpy as np
import pytest
import torch

from _gpu_helpers import T, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-11), (torch.float32, 2e-5)])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 32, 33, 65])
def test_recip_energy_and_gradients(cuda, n, dtype, tol):
    from admp_b200.ops import coulomb_pbc
    from oracle import admp_oracle as O
    rng = np.random.default_rng(n)
    npdt = np.float64 if dtype == torch.float64 else np.float32
    box = np.array([[11.0, 0, 0], [1.5, 12.0, 0], [-1.0, 0.5, 13.0]]).astype(npdt)
    pos = (rng.random((n, 3)) * 1.5 @ box.astype(np.float64)).astype(npdt)
    q = rng.uniform(-1, 1, n).astype(npdt)
    none = torch.zeros(1, 0, 2, dtype=torch.long, device=cuda)
    empty = torch.zeros(1, 0, dtype=dtype, device=cuda)
    E, comps, g = coulomb_pbc(T(pos[None], cuda, dtype), T(box[None], cuda, dtype), none, empty, empty,
                              T(q[None], cuda, dtype), 0.4, [[13, 16, 15]], O.DIELECTRIC, False, True, False, 2, True)
    p64, b64, q64 = pos.astype(np.float64), box.astype(np.float64), q.astype(np.float64)
    want = O.pme_recip(p64, b64, q64, 0.4, np.array([13, 16, 15]))
    es, en = O.pme_self(q64, 0.4), O.pme_non_neutral(q64, b64, 0.4)
    # FP32: sums of 216 terms of order ke kappa with single-precision weights and a 3,120-point transform: ~1e-5
    assert abs(float(comps[0, 1]) - want["E"]) <= tol * max(abs(want["E"]), 1.0)
    ref = {"pos": want["dpos"], "q": want["dq"] + es[1] + en[1], "box": want["dbox"] + en[2]}
    for name, r in ref.items():
        err = np.abs(g[name][0].double().cpu().numpy() - r).max()
        assert err < 10 * tol * max(np.abs(r).max(), 1.0), (name, err)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 2e-5)])
@pytest.mark.parametrize("slab", [False, True])
def test_hessian_equals_hessian_vector_products(cuda, slab, dtype, tol):
    """The dense matrix (chunks of 7, 60 and all columns) against unit-vector
    products, which go through the matvec kernels."""
    import ctypes  # noqa: F401
    from admp_b200 import _lib as L, synthetic
    from admp_b200.nblist import TorchNeighborList
    from admp_b200.qeq import QEqForceModule, _hessian
    pos, box, chi, hard, eta, _ = synthetic.water_system(30, 13.0, 3)
    n = len(pos)
    m = QEqForceModule(6.0, 5e-4, kmesh=15, slab_corr=slab)
    nb = TorchNeighborList(6.0)
    p, b = T(pos, cuda, dtype), T(box, cuda, dtype)
    h, e = T(hard, cuda, dtype), T(eta, cuda, dtype)
    pairs = nb(p, b)
    ds, bs = nb.get_ds(), nb.get_buffer_scales().to(dtype)
    lib = L.load()
    kp, _k = L.int3([15, 15, 15])
    c = m.submodels["coulomb"]
    ws = L.workspace(lib.admp_qeq_workspace_size(L.dtype_code(dtype), n, pairs.shape[0], kp, 0), cuda)
    ref = torch.empty(n, n, dtype=dtype, device=cuda)
    for k in range(n):
        v, out = torch.zeros(n, dtype=dtype, device=cuda), torch.empty(n, dtype=dtype, device=cuda)
        v[k] = 1
        L.check(lib.admp_qeq_hvp(L.dtype_code(dtype), m._flags(), n, kp, L.ptr(p), L.ptr(b), pairs.shape[0],
                                 L.ptr(pairs), L.ptr(ds), L.ptr(bs), L.ptr(h), L.ptr(e), c.kappa,
                                 m.const_lib.dielectric, L.ptr(v), L.ptr(out), L.ptr(ws), ws.numel(),
                                 L.stream_of(cuda)))
        ref[:, k] = out
    for cols in (7, 60, 256):
        got = _hessian(m, p, b, h, e, pairs, ds, bs, max_cols=cols)
        # the same terms in another order (FP32: two different single-precision transforms, ~1e-6 of the largest)
        assert rel(got, 0.5 * (ref + ref.T)) < tol, cols


@pytest.mark.parametrize("frames", [63, 64, 65])
def test_hessian_products_on_both_sides_of_the_gather_rule(cuda, frames):
    """63,000 and 64,000 atoms take one group a warp, 65,000 several: the products
    of equal frames agree with each other and across the rule."""
    from admp_b200 import _lib as L
    rng = np.random.default_rng(5)
    n, K = 1000, 12
    pos = rng.random((n, 3)) * 22.0
    v = rng.normal(size=n)
    lib = L.load()

    def product(nf):
        kp, _k = L.int3([K] * 3 * nf)
        rep = lambda x: T(np.repeat(x[None], nf, 0), cuda)  # noqa: E731
        p, b, h, q = rep(pos), rep(np.diag([22.0] * 3)), rep(np.full(n, 10.0)), rep(v)
        out = torch.empty(nf, n, dtype=torch.float64, device=cuda)
        ws = L.workspace(lib.admp_qeq_frames_workspace_size(L.F64, nf, n, 0, kp, 0), cuda)
        L.check(lib.admp_qeq_hvp_frames(L.F64, L.QEQ_KSPACE, nf, n, kp, L.ptr(p), L.ptr(b), 0, None, None, None,
                                        L.ptr(h), None, 0.4, 14.4, L.ptr(q), L.ptr(out), L.ptr(ws), ws.numel(),
                                        L.stream_of(cuda)))
        return out

    one, many = product(1), product(frames)
    assert float((many - one).abs().max() / one.abs().max()) < 1e-12


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 1e-4)])
@pytest.mark.parametrize("definite", [True, False])
@pytest.mark.parametrize("m", [None, 0, 1, 2])
def test_kkt_solves_definite_and_indefinite_systems(cuda, m, definite, dtype, tol):
    """Every route of the dense solve against numpy's solution of the bordered system."""
    from admp_b200.qeq import _kkt
    rng = np.random.default_rng(11)
    n = 37
    a = rng.normal(size=(n, n))
    h = a @ a.T / n + 3 * np.eye(n)
    if not definite:
        h[5, 5] -= 20.0
    chi, k = rng.normal(size=n), m or 0
    c, b = np.abs(rng.normal(size=(k, n))), rng.normal(size=k)
    full = np.block([[h, c.T], [c, np.zeros((k, k))]])
    want = np.linalg.solve(full, np.concatenate([-chi, b]))[:n]
    got = _kkt(T(h, cuda, dtype), T(chi, cuda, dtype), None if m is None else T(c, cuda, dtype), T(b, cuda, dtype))
    # condition numbers below 100: a few hundred ulp
    assert rel(got, want) < tol
