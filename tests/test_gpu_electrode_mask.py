"""Electrode masks of bytes give the charges and forces of boolean ones."""
import numpy as np
import pytest
import torch

from conftest import golden
from _gpu_helpers import T, rel

pytestmark = pytest.mark.gpu


@pytest.mark.filterwarnings("ignore")
def test_byte_mask(cuda):
    from admp_b200.electrode import LAMMPSElectrodeConstraint, PolarizableElectrode, infer, setup_from_lammps
    from admp_b200.nblist import TorchNeighborList
    d = golden("electrode_conp_slab_2d")
    calc = PolarizableElectrode(rcut=float(d["rcut"]), kappa=float(d["kappa"]), slab_corr=bool(d["slab_corr"]),
                                eps=1e-6, ls_eps=1e-6, max_iter=100, ethresh=float(d["ethresh"]))
    pos, box, q = T(d["pos"], cuda, grad=True), T(d["box"], cuda), T(d["q_lammps"], cuda, grad=True)
    nb = TorchNeighborList(float(d["rcut"]))
    pairs = nb(pos, box)
    cons = [LAMMPSElectrodeConstraint(indices=np.arange(int(a), int(z)), value=float(v),
                                      mode="conp" if int(md) == 0 else "conq", eta=float(d["lammps_eta"]),
                                      ffield=bool(d["ffield"])) for a, z, v, md in d["cons"]]
    mask, *rest = setup_from_lammps(len(d["q_lammps"]), cons, bool(d["symm"]), device=cuda)
    one, two = (infer(calc, pos, box, q, pairs, nb.get_ds(), nb.get_buffer_scales(), m, *rest)
                for m in (mask, mask.to(torch.uint8)))
    for x, y in zip(one, two):
        assert rel(x, y) < 1e-10  # atomics in another order
