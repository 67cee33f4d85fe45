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


@pytest.mark.parametrize("frames", [63, 64, 65])
def test_hessian_products_on_both_sides_of_the_gather_rule(cuda, frames):
    """1,000 atoms a frame: 63,000 and 64,000 atoms take one group a warp, 65,000 several;
    equal frames have equal products either way."""
    from admp_b200 import synthetic
    from admp_b200.nblist import TorchNeighborList
    from admp_b200.qeq import QEqForceModule, _hessian
    pos, box, chi, hard, eta, _ = synthetic.water_system(20, 13.0, 3)
    m = QEqForceModule(6.0, 5e-4, kmesh=14)
    nb = TorchNeighborList(6.0)
    p, b = T(pos, cuda), T(box, cuda)
    pairs = nb(p, b)
    one = _hessian(m, p, b, T(hard, cuda), T(eta, cuda), pairs, nb.get_ds(), nb.get_buffer_scales(), max_cols=1)
    many = _hessian(m, p, b, T(hard, cuda), T(eta, cuda), pairs, nb.get_ds(), nb.get_buffer_scales(), max_cols=frames)
    assert rel(many, one) < 1e-12
