"""The workloads this framework's speed is judged by.

Each case is one pass of what a user's program does through the public entry
points: a molecular-dynamics step (neighbour list, PME energy, forces), a QEq
charge solve with forces, a constant-potential electrode evaluation, the
differentiation batch, the image neighbour list of small cells, the dense KKT
solve, and continuous-batching serving from device-resident or host arrays.

``listed()`` names the fixed sizes, ``draw(rng)`` gives more of the same
ranges, ``prepare`` makes what the program holds before the call, ``run`` is
one pass, ``work`` counts the bytes and operations a pass cannot do without
and ``exact`` is the result in plain FP64 torch, without the package.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("torch-admp_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

RC = 6.0          # real-space cutoff of every workload of this repository (Angstrom)
ETHRESH = 5e-4    # Ewald accuracy of the benchmark workloads
DENSITY = 0.1     # atoms per cubic Angstrom of the serving stream
KE = 14.399645468667817  # e^2 / (4 pi eps0) in eV Angstrom
KAPPA = math.sqrt(-math.log(2 * ETHRESH)) / RC
DEV = "cuda:0"
DTYPES = {"f32": torch.float32, "f64": torch.float64}
CG_TOL = {"f32": 1e-7, "f64": 1e-12}  # ||P grad E|| / N: the benchmark's, and a tight one where double precision is asked for


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest system of the stream, one MD step in the reference's precision: launches and host time
        {"name": "md_200_f64", "kind": "md", "n": 200, "dtype": "f64", "mesh": 0, "tilt": False, "virial": False},
        # the plain PME configuration: 1,536 charges, 25 A box, 32^3 mesh
        {"name": "md_1536_f64", "kind": "md", "n": 1536, "dtype": "f64", "mesh": 32, "tilt": False, "virial": False},
        # an ordinary constant-pressure step: triclinic cell, forces and virial, automatic (odd) mesh
        {"name": "md_tilt_6007_f64", "kind": "md", "n": 6007, "dtype": "f64", "mesh": 0, "tilt": True, "virial": True},
        # the largest system of the stream in single precision
        {"name": "md_20000_f32", "kind": "md", "n": 20000, "dtype": "f32", "mesh": 0, "tilt": False, "virial": False},
        # the QEq configuration: 1,000 waters, 31 A box, 48^3 mesh
        {"name": "qeq_water_3000_f32", "kind": "qeq", "nmol": 1000, "dtype": "f32", "mesh": 48},
        # a larger charge solve in the reference's precision, automatic mesh
        {"name": "qeq_water_10701_f64", "kind": "qeq", "nmol": 3567, "dtype": "f64", "mesh": 0},
        # the constant-potential configuration: 2 x 1,152 electrode atoms, 3,000 ions, 64 x 64 x 160 mesh
        {"name": "electrode_5304_f32", "kind": "electrode", "side": 24, "ions": 3000, "dtype": "f32",
         "k0": 64, "k1": 64, "k2": 160},
        # the differentiation batch: 64 jittered frames, gradients through the implicit adjoint
        {"name": "frames_64x3000_f32", "kind": "frames", "frames": 64, "nmol": 1000, "dtype": "f32", "mesh": 48},
        # a cell smaller than twice the cutoff: pairs over periodic images, energy and forces
        {"name": "image_280_f64", "kind": "image", "n": 280, "rc": 9.0, "dtype": "f64"},
        # the dense path (Hessian and KKT solve) of a small system
        {"name": "dense_429_f64", "kind": "dense", "nmol": 143, "dtype": "f64"},
        # serving: a backlog of mixed requests from device arrays, single precision (the benchmark's stream)
        {"name": "serve_240_f32", "kind": "serve", "requests": 240, "nmin": 200, "nmax": 20000, "dtype": "f32",
         "host": False},
        # serving from host arrays in double precision, results to the host
        {"name": "serve_host_60_f64", "kind": "serve", "requests": 60, "nmin": 200, "nmax": 20000, "dtype": "f64",
         "host": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above."""
    kind = rng.choice(["md", "md", "md", "qeq", "qeq", "electrode", "frames", "image", "dense", "serve"])
    dtype = rng.choice(["f32", "f64"])
    if kind == "md":
        n = _log_int(rng, 200, 20000)
        length = (n / DENSITY) ** (1.0 / 3.0)
        mesh = rng.choice([0, 0, int(length * rng.uniform(1.1, 1.4))])
        return {"kind": "md", "n": n, "dtype": dtype, "mesh": mesh, "tilt": rng.random() < 0.4,
                "virial": rng.random() < 0.4}
    if kind == "qeq":
        nmol = _log_int(rng, 67, 4500)
        length = (3 * nmol / DENSITY) ** (1.0 / 3.0)
        return {"kind": "qeq", "nmol": nmol, "dtype": dtype,
                "mesh": rng.choice([0, 0, int(length * rng.uniform(1.1, 1.5))])}
    if kind == "electrode":
        side = 2 * rng.randint(6, 12)
        k = rng.randint(2 * side, int(2.7 * side))
        return {"kind": "electrode", "side": side, "ions": int(3000 * (side / 24.0) ** 2 * rng.uniform(0.6, 1.0)),
                "dtype": dtype, "k0": k, "k1": k + rng.randint(-2, 2), "k2": rng.randint(120, 160)}
    if kind == "frames":
        nmol = _log_int(rng, 67, 1000)
        return {"kind": "frames", "frames": _log_int(rng, 2, 64), "nmol": nmol, "dtype": dtype,
                "mesh": int((3 * nmol / DENSITY) ** (1.0 / 3.0) * rng.uniform(1.2, 1.5))}
    if kind == "image":
        return {"kind": "image", "n": _log_int(rng, 60, 400), "rc": round(rng.uniform(7.5, 10.0), 2), "dtype": dtype}
    if kind == "dense":
        return {"kind": "dense", "nmol": _log_int(rng, 67, 240), "dtype": "f64"}
    return {"kind": "serve", "requests": _log_int(rng, 12, 60 if dtype == "f64" else 200), "nmin": 200, "nmax": 20000,
            "dtype": dtype, "host": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _t(x, dtype, grad=False):
    return torch.tensor(np.asarray(x), dtype=dtype, device=DEV, requires_grad=grad)


def _box_length(n):
    return (n / DENSITY) ** (1.0 / 3.0)


def _md_arrays(case, seed):
    """Uniform random charges at the stream's density (25 A for the 1,536-charge configuration, which has it too).
    The lists these cases return have as many rows as there are pairs, so every seed takes the same points: in another
    order of the atoms, mirrored, with the axes of a cubic cell exchanged, and with other charges."""
    n = case["n"]
    length = 25.0 if n == 1536 else _box_length(n)
    box = np.diag([length] * 3)
    if case.get("tilt"):
        box[1, 0], box[2, 0], box[2, 1] = 0.15 * length, -0.1 * length, 0.2 * length
        box[0, 0] *= 1.06
        box *= (length ** 3 / np.linalg.det(box)) ** (1.0 / 3.0)
    pos = np.random.default_rng(n).random((n, 3)) @ box
    rng = np.random.default_rng(seed)
    pos = pos[rng.permutation(n)] * rng.choice([-1.0, 1.0])
    if not case.get("tilt"):
        pos = pos[:, rng.permutation(3)]
    q = rng.uniform(-1.0, 1.0, n)
    return pos, box, q - q.mean()


def _water_arrays(nmol, seed):
    from admp_b200 import synthetic
    length = 31.0 if nmol == 1000 else _box_length(3 * nmol)
    pos, box, chi, hard, eta, _ = synthetic.water_system(nmol, length, seed)
    return pos, box, chi, hard, eta


def _requests(case, seed):
    """Atom counts at the quantiles of the stream's log-uniform law, 60% PME / 40% QEq, in mixed order; positions,
    charges and orientations from the seed."""
    from admp_b200 import synthetic
    nreq, lo, hi = case["requests"], math.log(case["nmin"]), math.log(case["nmax"])
    order = np.random.default_rng(nreq).permutation(nreq)
    out = []
    for rid, k in enumerate(order):
        n = int(round(math.exp(lo + (hi - lo) * (int(k) + 0.5) / nreq)))
        s = (seed * 100003 + rid) % (2 ** 31)
        if int(k) % 5 in (0, 2, 4):
            n += n % 2
            pos, box, q = synthetic.random_charges_system(n, _box_length(n), s, balanced=True)
            out.append(synthetic.Request(rid, "pme", 0.0, pos, box, charges=q))
        else:
            nmol = max(67, n // 3)
            pos, box, chi, hard, eta, _ = synthetic.water_system(nmol, _box_length(3 * nmol), s)
            out.append(synthetic.Request(rid, "qeq", 0.0, pos, box, chi=chi, hardness=hard, eta=eta))
    return out


def _on_device(req, dtype):
    from admp_b200 import synthetic
    t = lambda x, d: None if x is None else torch.as_tensor(x, dtype=d, device=DEV)  # noqa: E731
    r = synthetic.Request(req.rid, req.kind, req.arrival, t(req.pos, torch.float64), t(req.box, torch.float64),
                          charges=t(req.charges, dtype), chi=t(req.chi, dtype), hardness=t(req.hardness, dtype),
                          eta=t(req.eta, dtype))
    r.box_host = req.box
    return r


def _electrode_arrays(case, seed):
    from admp_b200 import synthetic
    return synthetic.electrode_system(seed, n_side=case["side"], n_ions=case["ions"])


def _mesh(case):
    return case["mesh"] if case.get("mesh") else None


def prepare(case, seed):
    kind = case["kind"]
    dt = DTYPES[case["dtype"]]
    s = {"case": case, "kind": kind, "dt": dt}
    if kind == "md":
        from admp_b200.nblist import TorchNeighborList
        from admp_b200.pme import CoulombForceModule
        pos, box, q = _md_arrays(case, seed)
        s.update(pos=_t(pos, dt, True), box=_t(box, dt, bool(case["virial"])), q=_t(q, dt), nb=TorchNeighborList(RC),
                 model=CoulombForceModule(RC, ETHRESH, kmesh=_mesh(case)))
    elif kind in ("qeq", "dense"):
        from admp_b200.nblist import TorchNeighborList
        from admp_b200.qeq import QEqForceModule
        pos, box, chi, hard, eta = _water_arrays(case["nmol"], seed)
        n = len(pos)
        s.update(pos=_t(pos, dt, True), box=_t(box, dt), chi=_t(chi, dt), hard=_t(hard, dt), eta=_t(eta, dt),
                 q0=torch.zeros(n, dtype=dt, device=DEV), C=torch.ones(1, n, dtype=dt, device=DEV),
                 b=torch.zeros(1, dtype=dt, device=DEV), nb=TorchNeighborList(RC),
                 model=QEqForceModule(RC, ETHRESH, kmesh=_mesh(case), eps=CG_TOL[case["dtype"]], max_iter=1000))
    elif kind == "electrode":
        from admp_b200.electrode import LAMMPSElectrodeConstraint, PolarizableElectrode, setup_from_lammps
        from admp_b200.nblist import TorchNeighborList
        pos, box, q, top, bot = _electrode_arrays(case, seed)
        cons = [LAMMPSElectrodeConstraint(indices=top, value=1.0, mode="conp", eta=math.sqrt(2.0)),
                LAMMPSElectrodeConstraint(indices=bot, value=0.0, mode="conp", eta=math.sqrt(2.0))]
        s.update(pos=_t(pos, dt, True), box=_t(box, dt), q=_t(q, dt), nb=TorchNeighborList(RC),
                 data=setup_from_lammps(len(q), cons, True, device=DEV, dtype=dt),
                 model=PolarizableElectrode(RC, ETHRESH, kmesh=[case["k0"], case["k1"], case["k2"]], slab_corr=True,
                                            eps=CG_TOL[case["dtype"]], max_iter=1000))
    elif kind == "frames":
        from admp_b200.qeq import QEqForceModule
        pos, box, chi, hard, eta, w = _frames_arrays(case, seed)
        s.update(pos=_t(pos, dt, True), box=_t(box, dt, True), chi=_t(chi, dt, True), hard=_t(hard, dt, True),
                 eta=_t(eta, dt, True), w=_t(w, dt), C=torch.ones(1, pos.shape[1], dtype=dt, device=DEV),
                 model=QEqForceModule(RC, ETHRESH, kmesh=case["mesh"], eps=CG_TOL[case["dtype"]], max_iter=1000))
    elif kind == "image":
        from admp_b200.pme import CoulombForceModule
        pos, box, q = _md_arrays(case, seed)
        s.update(pos=_t(pos, dt, True), box=_t(box, dt), q=_t(q, dt),
                 model=CoulombForceModule(case["rc"], ETHRESH))
    else:
        from admp_b200.serving import ServingEngine
        reqs = _requests(case, seed)
        mesh = sum(int(np.prod(_auto_mesh(np.diagonal(r.box), KAPPA))) for r in reqs)
        s["engine"] = ServingEngine(device=DEV, dtype=dt, max_atoms=int(1.1 * sum(r.natoms for r in reqs)) + 65536,
                                    max_slots=case["requests"] + 8, mesh_budget=mesh + 4_000_000, rcut=RC,
                                    ethresh=ETHRESH, tol=CG_TOL[case["dtype"]], max_iter=300)
        s["engine"].results_to_host = bool(case["host"])
        s["reqs"] = reqs if case["host"] else [_on_device(r, dt) for r in reqs]
    return s


def _frames_arrays(case, seed):
    from admp_b200 import synthetic
    nmol = case["nmol"]
    length = 31.0 if nmol == 1000 else _box_length(3 * nmol)
    pos, box, chi, hard, eta, _ = synthetic.water_frames(case["frames"], seed, n_mol=nmol, box_len=length)
    w = np.random.default_rng(seed + 7).normal(size=pos.shape[:2])
    return pos, box, chi, hard, eta, w


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_md(s):
    """Neighbour list, PME energy, forces (and dE/dbox): the loop body of an MD program."""
    nb = s["nb"]
    pairs = nb(s["pos"], s["box"])
    e = s["model"](s["pos"], s["box"], pairs, nb.get_ds(), nb.get_buffer_scales(), {"charge": s["q"]})
    wrt = [s["pos"], s["box"]] if s["case"]["virial"] else [s["pos"]]
    grads = torch.autograd.grad(e.sum(), wrt)
    return {"pairs": pairs, "ds": nb.get_ds().detach(), "energy": e.detach(), "forces": -grads[0],
            "dE_dbox": grads[1] if s["case"]["virial"] else None}


def _run_qeq(s):
    """Neighbour list, charge solve from zero charges, energy and forces at the solved charges."""
    from admp_b200.qeq import pgrad_optimize
    nb = s["nb"]
    pairs = nb(s["pos"], s["box"])
    e, q = pgrad_optimize(s["model"], s["q0"], s["pos"], s["box"], s["chi"], s["hard"], s["eta"], pairs, nb.get_ds(),
                          nb.get_buffer_scales(), s["C"], s["b"], reinit_q=True, method="quadratic")
    return {"energy": e.detach(), "q": q.detach(), "forces": -torch.autograd.grad(e.sum(), s["pos"])[0]}


def _run_dense(s):
    """As _run_qeq with the dense Hessian and KKT solve."""
    from admp_b200.qeq import matinv_optimize
    nb = s["nb"]
    pairs = nb(s["pos"], s["box"])
    e, q = matinv_optimize(s["model"], s["pos"], s["box"], s["chi"], s["hard"], s["eta"], pairs, nb.get_ds(),
                           nb.get_buffer_scales(), s["C"], s["b"])
    return {"energy": e.detach(), "q": q.detach(), "forces": -torch.autograd.grad(e.sum(), s["pos"])[0]}


def _run_electrode(s):
    from admp_b200.electrode import infer
    nb = s["nb"]
    pairs = nb(s["pos"], s["box"])
    e, f, q = infer(s["model"], s["pos"], s["box"], s["q"], pairs, nb.get_ds(), nb.get_buffer_scales(), *s["data"])
    return {"energy": e.detach(), "forces": f.detach(), "q": q.detach()}


def _run_frames(s):
    """Charges of all frames, energies, and the gradients of energies + w.q through the implicit adjoint."""
    from admp_b200.nblist import frame_pair_lists
    from admp_b200.qeq import qeq_solve_frames
    m, pos, box, chi, hard, eta = s["model"], s["pos"], s["box"], s["chi"], s["hard"], s["eta"]
    nf, n = pos.shape[0], pos.shape[1]
    pairs, ds, bs = frame_pair_lists(pos, box, RC)
    q = qeq_solve_frames(m, pos, box, chi, hard, eta, pairs, ds, bs, s["C"])
    e = m(pos, box, pairs, ds, bs, {"charge": q, "chi": chi.expand(nf, n), "hardness": hard.expand(nf, n),
                                    "eta": eta.expand(nf, n)})
    g = torch.autograd.grad(e.sum() + (s["w"] * q).sum(), [pos, box, chi, hard, eta])
    return {"energy": e.detach(), "q": q.detach(), "pos": g[0], "box": g[1], "chi": g[2], "hard": g[3], "eta": g[4]}


def _run_image(s):
    from admp_b200.nblist import dp_nblist
    pairs, ds, bs = dp_nblist(s["pos"], s["box"], 4000, s["case"]["rc"])
    e = s["model"](s["pos"], s["box"], pairs, ds, bs, {"charge": s["q"]})
    f = -torch.autograd.grad(e.sum(), s["pos"])[0]
    return {"pairs": pairs, "scales": bs, "ds": ds.detach(), "energy": e.detach(), "forces": f}


def _run_serve(s):
    """Every request of a backlog; energies, forces and solved charges in request order."""
    eng = s["engine"]
    eng.results = []
    res = sorted(eng.run(s["reqs"], arrivals=False), key=lambda r: r.rid)
    cat = np.concatenate if s["case"]["host"] else torch.cat
    return {"energy": np.array([r.energy for r in res]), "forces": cat([r.forces for r in res]),
            "q": cat([r.charges for r in res if r.kind == "qeq"]), "status": np.array([r.status for r in res])}


# ---------------------------------------------------------------------------
# bytes and operations a pass cannot do without
# ---------------------------------------------------------------------------
def _auto_mesh(diag, kappa):
    return [int(math.ceil(2 * kappa * float(x) / (3.0 * ETHRESH ** 0.2))) for x in diag]


def _pme_flops(n, mesh, pairs, matvec=False):
    """Spread and gather of 216 mesh points per atom, two real 3-D FFTs, the pair terms (half list)."""
    fft = 2 * 2.5 * mesh * math.log2(max(mesh, 2))
    return n * 216 * (4 if matvec else 10) + fft + pairs / 2 * (4 if matvec else 60)


def work(case):
    kind, sz = case["kind"], 4 if case["dtype"] == "f32" else 8
    per_atom = DENSITY * 4.0 / 3.0 * math.pi * RC ** 3  # neighbours within the cutoff
    if kind == "md":
        n = case["n"]
        mesh = case["mesh"] ** 3 if case["mesh"] else int(np.prod(_auto_mesh([_box_length(n)] * 3, KAPPA)))
        p = n * per_atom
        # positions and charges in; full pair list, distances, forces out
        return {"bytes": 7 * n * sz + p * (16 + 8 + sz), "flops": _pme_flops(n, mesh, p) + 30 * p}
    if kind in ("qeq", "dense"):
        n = 3 * case["nmol"]
        mesh = case["mesh"] ** 3 if case.get("mesh") else int(np.prod(_auto_mesh([_box_length(n)] * 3, KAPPA)))
        p = n * per_atom
        its = 20 if kind == "qeq" else n
        dense = n ** 3 * 2.0 / 3.0 if kind == "dense" else 0.0
        return {"bytes": 10 * n * sz + p * (16 + 8 + sz),
                "flops": its * _pme_flops(n, mesh, p, True) + _pme_flops(n, mesh, p) + dense}
    if kind == "electrode":
        ne, n = 4 * case["side"] ** 2, 4 * case["side"] ** 2 + case["ions"]
        mesh, p = case["k0"] * case["k1"] * case["k2"], n * 60
        return {"bytes": 10 * n * sz + p * (16 + 8 + sz),
                "flops": 36 * _pme_flops(ne, mesh, ne * 60, True) + 2 * _pme_flops(n, mesh, p)}
    if kind == "frames":
        n, mesh = 3 * case["nmol"], case["mesh"] ** 3
        p = n * per_atom
        return {"bytes": case["frames"] * (14 * n * sz + p * (16 + 8 + 2 * sz)),
                "flops": case["frames"] * (2 * 20 * _pme_flops(n, mesh, p, True) + 3 * _pme_flops(n, mesh, p))}
    if kind == "image":
        n, rc = case["n"], case["rc"]
        kap = math.sqrt(-math.log(2 * ETHRESH)) / rc
        mesh = int(np.prod(_auto_mesh([_box_length(n)] * 3, kap)))
        p = n * DENSITY * 4.0 / 3.0 * math.pi * rc ** 3 / 2
        return {"bytes": 7 * n * sz + p * (16 + 12 + 4 + sz), "flops": _pme_flops(n, mesh, 2 * p) + 30 * p}
    b = f = 0.0
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    for k in range(case["requests"]):
        n = math.exp(lo + (hi - lo) * (k + 0.5) / case["requests"])
        mesh, p = float(np.prod(_auto_mesh([_box_length(n)] * 3, KAPPA))), n * per_atom
        qeq = k % 5 not in (0, 2, 4)
        b += n * (8 * 3 + 3 * sz + (4 * sz if qeq else sz))
        f += _pme_flops(n, mesh, p) + 30 * p + (20 * _pme_flops(n, mesh, p, True) if qeq else 0.0)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# results in plain FP64 torch
# ---------------------------------------------------------------------------
def _dev():
    return DEV if torch.cuda.is_available() else "cpu"


def _f64(x, dtype):
    """The value the program's tensor of `dtype` holds, in FP64."""
    return torch.tensor(np.asarray(x), dtype=dtype, device=_dev()).double()


def _erfc(x):
    return torch.erfc(x)


class _Exact:
    """One periodic system: PME with order-6 B-splines, real-space and damping sums over minimum images."""

    def __init__(self, pos, box, mesh, kappa, eta=None, slab=False, images=None):
        self.pos, self.box, self.mesh, self.kappa, self.eta, self.slab = pos, box, mesh, kappa, eta, slab
        self.rc = RC
        if images is None:
            self._min_image_pairs()
        else:
            self.i, self.j, self.shift, self.scale = images

    def _min_image_pairs(self):
        """Half list (i < j) in (i, j) order and the integer image shifts."""
        pos, box = self.pos.detach(), self.box.detach()
        n = pos.shape[0]
        frac = pos @ torch.linalg.inv(box)
        ii, jj, nn = [], [], []
        step = max(1, 20_000_000 // n)
        for a in range(0, n, step):
            df = frac[a:a + step, None] - frac[None]
            sh = torch.floor(df + 0.5)
            r2 = (((df - sh) @ box) ** 2).sum(-1)
            hit = (r2 < self.rc ** 2) & (r2 > 1e-4)
            i, j = hit.nonzero(as_tuple=True)
            keep = i + a < j
            i, j = i[keep], j[keep]
            ii.append(i + a)
            jj.append(j)
            nn.append(-sh[i, j])
        self.i, self.j, self.shift = torch.cat(ii), torch.cat(jj), torch.cat(nn)
        self.scale = torch.ones(self.i.numel(), dtype=torch.float64, device=pos.device)

    def full_list(self):
        """Both orders, sorted by (i, j): rows and their distances."""
        d = self.distances(self.pos.detach(), self.box.detach())
        a, b = torch.cat([self.i, self.j]), torch.cat([self.j, self.i])
        order = torch.argsort(a * self.pos.shape[0] + b)
        return torch.cat([d, d])[order]

    def distances(self, pos, box):
        return torch.linalg.norm(pos[self.i] - pos[self.j] + self.shift @ box, dim=1)

    def stencil(self, pos, box):
        """Flat mesh indices [N, 216] and B-spline weights [N, 216]."""
        dev = pos.device
        k = torch.tensor(self.mesh, dtype=torch.float64, device=dev)
        x = (pos @ torch.linalg.inv(box)) * k
        m0 = torch.ceil(x.detach())
        t = m0 - x
        m = [t, 1.0 - t]
        for order in range(3, 7):
            new = []
            for c in range(order):
                cur = m[c] if c < order - 1 else torch.zeros_like(t)
                prev = m[c - 1] if c > 0 else torch.zeros_like(t)
                new.append(((t + c) * cur + (order - t - c) * prev) / (order - 1))
            m = new
        w = torch.stack(m, -1)
        steps = torch.arange(6, device=dev)
        idx = (m0.long()[:, :, None] - 3 + steps) % torch.tensor(self.mesh, device=dev)[None, :, None]
        n, (_, k1, k2) = pos.shape[0], self.mesh
        flat = ((idx[:, 0, :, None, None] * k1 + idx[:, 1, None, :, None]) * k2 + idx[:, 2, None, None, :])
        wt = w[:, 0, :, None, None] * w[:, 1, None, :, None] * w[:, 2, None, None, :]
        return flat.reshape(n, 216), wt.reshape(n, 216)

    def green(self, box):
        """G(k) with E = sum G |S|^2 over the full spectrum (zero at k = 0)."""
        dev = box.device
        lab, th = [], []
        for size in self.mesh:
            i = torch.arange(size, device=dev)
            lb = torch.where(i <= (size - 1) // 2, i, i - size).double()
            lab.append(lb)
            th.append(66 / 120 + 52 / 120 * torch.cos(2 * math.pi * lb / size)
                      + 2 / 120 * torch.cos(4 * math.pi * lb / size))
        n = torch.stack(torch.meshgrid(*lab, indexing="ij"), -1)
        theta = th[0][:, None, None] * th[1][None, :, None] * th[2][None, None, :]
        # k = 2 pi n B^-1, the convention of the modules (rows of the box are the lattice vectors)
        ksq = ((2 * math.pi * (n @ torch.linalg.inv(box))) ** 2).sum(-1)
        zero = torch.zeros_like(ksq, dtype=torch.bool)
        zero[0, 0, 0] = True
        ksq = torch.where(zero, torch.ones_like(ksq), ksq)
        g = KE * 2 * math.pi / torch.linalg.det(box) / ksq * torch.exp(-ksq / (4 * self.kappa ** 2)) / theta ** 2
        return torch.where(zero, torch.zeros_like(g), g)

    def coefficients(self, pos, box, eta):
        """Pair matrix entries of the real-space and damping sums (half list)."""
        d = self.distances(pos, box)
        c = _erfc(self.kappa * d)
        if eta is not None:
            e = torch.sqrt((eta[self.i] ** 2 + eta[self.j] ** 2) / 2)
            e = torch.where(e == 0, torch.full_like(e, 1e-10), e)
            c = c - _erfc(d / (2 * e))
        return KE * self.scale * c / d

    def energy(self, q, pos=None, box=None, eta=None):
        """The part quadratic in q (Coulomb and damping), differentiable in every argument."""
        pos = self.pos if pos is None else pos
        box = self.box if box is None else box
        eta = self.eta if eta is None else eta
        idx, wt = self.stencil(pos, box)
        mesh = torch.zeros(int(np.prod(self.mesh)), dtype=torch.float64, device=pos.device)
        mesh = mesh.index_add(0, idx.reshape(-1), (wt * q[:, None]).reshape(-1)).reshape(self.mesh)
        spec = torch.fft.fftn(mesh)
        e = (self.green(box) * (spec.real ** 2 + spec.imag ** 2)).sum()
        e = e + (self.coefficients(pos, box, eta) * q[self.i] * q[self.j]).sum()
        e = e - KE * self.kappa / math.sqrt(math.pi) * (q ** 2).sum()
        vol = torch.linalg.det(box)
        e = e - math.pi / (2 * vol * self.kappa ** 2) * KE * q.sum() ** 2
        if eta is not None:
            inv = torch.where(eta.abs() > 1e-4, 1 / torch.where(eta == 0, torch.ones_like(eta), eta),
                              torch.zeros_like(eta))
            e = e + KE * (inv * q ** 2).sum() / (2 * math.sqrt(math.pi))
        if self.slab:
            z, lz2 = pos[:, 2], (box[2] ** 2).sum()
            e = e + 2 * math.pi / vol * KE * ((q * z).sum() ** 2 - q.sum() * (q * z * z).sum() - q.sum() ** 2 * lz2 / 12)
        return e

    def operator(self):
        """q -> dE/dq of ``energy`` (a linear map), with the stencils and coefficients kept."""
        with torch.no_grad():
            pos, box, eta = self.pos.detach(), self.box.detach(), None if self.eta is None else self.eta.detach()
            idx, wt = self.stencil(pos, box)
            flat, green = idx.reshape(-1), self.green(box)
            total = green.numel()
            coef = self.coefficients(pos, box, eta)
            vol = float(torch.linalg.det(box))
            diag = torch.full((pos.shape[0],), -2 * KE * self.kappa / math.sqrt(math.pi), dtype=torch.float64,
                              device=pos.device)
            if eta is not None:
                diag = diag + torch.where(eta.abs() > 1e-4, KE / (math.sqrt(math.pi) * torch.where(eta == 0, torch.ones_like(eta), eta)),
                                          torch.zeros_like(eta))
            z, lz2 = pos[:, 2], float((box[2] ** 2).sum())

        def apply(q):
            with torch.no_grad():
                mesh = torch.zeros(total, dtype=torch.float64, device=q.device)
                mesh.index_add_(0, flat, (wt * q[:, None]).reshape(-1))
                phi = torch.fft.ifftn(torch.fft.fftn(mesh.reshape(self.mesh)) * green).real.reshape(-1) * (2 * total)
                out = (phi[idx] * wt).sum(1) + diag * q - math.pi / (vol * self.kappa ** 2) * KE * q.sum()
                out.index_add_(0, self.i, coef * q[self.j])
                out.index_add_(0, self.j, coef * q[self.i])
                if self.slab:
                    out = out + 2 * math.pi / vol * KE * (2 * z * (q * z).sum() - (q * z * z).sum() - z * z * q.sum()
                                                          - lz2 / 6 * q.sum())
                return out

        return apply


def _solve(apply, rhs, iterations=400):
    """H x = rhs with sum(x) = 0: projected conjugate gradient to rounding error."""
    proj = lambda v: v - v.mean()  # noqa: E731
    x = torch.zeros_like(rhs)
    r = proj(rhs)
    p, rr = r.clone(), torch.dot(r, r)
    stop = 1e-28 * float(rr)
    for _ in range(iterations):
        hp = proj(apply(p))
        a = rr / torch.dot(p, hp)
        x, r = x + a * p, r - a * hp
        new = torch.dot(r, r)
        if float(new) <= stop:
            break
        p, rr = r + new / rr * p, new
    return proj(x)


def _exact_qeq(ref, chi, hard):
    """Solved charges, then (energy, charges, forces) at them."""
    apply = ref.operator()
    q = _solve(lambda v: apply(v) + 2 * hard * v, -chi)
    pos = ref.pos.detach().clone().requires_grad_(True)
    e = ref.energy(q, pos=pos) + (chi * q + hard * q * q).sum()
    return e.detach(), q, -torch.autograd.grad(e, pos)[0]


def exact(case, seed):
    kind, dt = case["kind"], DTYPES[case["dtype"]]
    if kind in ("md", "image"):
        pos, box, q = (_f64(x, dt) for x in _md_arrays(case, seed))
        rc = case.get("rc", RC)
        kappa = math.sqrt(-math.log(2 * ETHRESH)) / rc
        mesh = [case["mesh"]] * 3 if case.get("mesh") else _auto_mesh(torch.diagonal(box).tolist(), kappa)
        ref = _Exact(pos, box, mesh, kappa, images=_all_images(pos, box, rc) if kind == "image" else None)
        p, b = pos.clone().requires_grad_(True), box.clone().requires_grad_(True)
        e = ref.energy(q, pos=p, box=b)
        gp, gb = torch.autograd.grad(e, [p, b])
        if kind == "image":
            return {"pairs": None, "scales": None, "ds": ref.distances(pos, box), "energy": e.detach().reshape(1),
                    "forces": -gp}
        return {"pairs": None, "ds": ref.full_list(), "energy": e.detach().reshape(1), "forces": -gp,
                "dE_dbox": gb if case["virial"] else None}
    if kind in ("qeq", "dense"):
        pos, box, chi, hard, eta = (_f64(x, dt) for x in _water_arrays(case["nmol"], seed))
        mesh = [case["mesh"]] * 3 if case.get("mesh") else _auto_mesh(torch.diagonal(box).tolist(), KAPPA)
        e, q, f = _exact_qeq(_Exact(pos, box, mesh, KAPPA, eta=eta), chi, hard)
        return {"energy": e.reshape(1), "q": q, "forces": f}
    if kind == "electrode":
        pos, box, qin, top, bot = _electrode_arrays(case, seed)
        n, ne = len(qin), len(top) + len(bot)
        eta, chi = np.zeros(n), np.zeros(n)
        eta[:ne] = 1 / math.sqrt(2.0) * math.sqrt(2.0) / 2.0
        chi[:len(top)] = -1.0
        pos, box, qin, eta, chi = (_f64(x, dt) for x in (pos, box, qin, eta, chi))
        ref = _Exact(pos, box, [case["k0"], case["k1"], case["k2"]], KAPPA, eta=eta, slab=True)
        apply = ref.operator()

        def restricted(v):
            full = torch.zeros(n, dtype=torch.float64, device=v.device)
            full[:ne] = v
            return apply(full)[:ne]

        q = qin.clone()
        q[:ne] = _solve(restricted, -(chi + apply(qin))[:ne])
        p = pos.clone().requires_grad_(True)
        e = ref.energy(q, pos=p)
        return {"energy": e.detach(), "forces": -torch.autograd.grad(e, p)[0], "q": q}
    if kind == "frames":
        return _exact_frames(case, seed, dt)
    energies, forces, charges = [], [], []
    for r in _requests(case, seed):
        pos, box = _f64(r.pos, torch.float64), _f64(r.box, torch.float64)
        mesh = _auto_mesh(np.diagonal(r.box), KAPPA)
        if r.kind == "qeq":
            chi, hard, eta = (_f64(x, dt) for x in (r.chi, r.hardness, r.eta))
            e, q, f = _exact_qeq(_Exact(pos, box, mesh, KAPPA, eta=eta), chi, hard)
            charges.append(q)
        else:
            p = pos.clone().requires_grad_(True)
            e = _Exact(pos, box, mesh, KAPPA).energy(_f64(r.charges, dt), pos=p)
            f = -torch.autograd.grad(e, p)[0]
        energies.append(e.item())
        forces.append(f)
    return {"energy": np.array(energies), "forces": torch.cat(forces), "q": torch.cat(charges), "status": None}


def _exact_frames(case, seed, dt):
    pos, box, chi, hard, eta, w = (_f64(x, dt) for x in _frames_arrays(case, seed))
    energy, charges, gpos, gbox = [], [], [], []
    gchi, ghard, geta = torch.zeros_like(chi), torch.zeros_like(hard), torch.zeros_like(eta)
    for f in range(case["frames"]):
        ref = _Exact(pos[f], box[f], [case["mesh"]] * 3, KAPPA, eta=eta)
        apply = ref.operator()
        op = lambda v: apply(v) + 2 * hard * v  # noqa: E731
        q, lam = _solve(op, -chi), _solve(op, w[f])
        args = [x.detach().clone().requires_grad_(True) for x in (pos[f], box[f], chi, hard, eta)]
        p, b, c, h, t = args
        e = ref.energy(q, p, b, t) + (c * q + h * q * q).sum()
        # dL/dtheta = dE/dtheta - lam . d(dE/dq)/dtheta, lam . J q by polarisation
        cross = 0.5 * (ref.energy(q + lam, p, b, t) - ref.energy(q - lam, p, b, t)) + (c * lam + 2 * h * q * lam).sum()
        g = torch.autograd.grad(e - cross, args)
        energy.append(e.detach())
        charges.append(q)
        gpos.append(g[0])
        gbox.append(g[1])
        gchi += g[2]
        ghard += g[3]
        geta += g[4]
    return {"energy": torch.stack(energy), "q": torch.stack(charges), "pos": torch.stack(gpos),
            "box": torch.stack(gbox), "chi": gchi, "hard": ghard, "eta": geta}


def _all_images(pos, box, rc):
    """Pairs over periodic images: i < j by (i, j, image) with scale 1, then self images with scale 1/2."""
    n = pos.shape[0]
    inv = torch.linalg.inv(box)
    heights = 1.0 / torch.linalg.norm(inv, dim=0)
    m = [int(math.ceil(rc / float(h))) for h in heights]
    cell = torch.floor(pos @ inv)
    frac = pos @ inv - cell
    ax = [torch.arange(-k, k + 1, device=pos.device, dtype=torch.float64) for k in m]
    img = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    df = frac[None, :, None] - frac[:, None, None] + img[None, None]
    r2 = ((df @ box) ** 2).sum(-1)
    idx = torch.arange(n, device=pos.device)
    hit = r2 <= rc * rc
    self_zero = (idx[:, None, None] == idx[None, :, None]) & (img == 0).all(-1)[None, None]
    hit &= ~self_zero & (idx[None, :, None] >= idx[:, None, None])
    i, j, c = hit.nonzero(as_tuple=True)
    shift = img[c] + cell[i] - cell[j]
    order = torch.cat([(i != j).nonzero()[:, 0], (i == j).nonzero()[:, 0]])
    i, j, shift = i[order], j[order], shift[order]
    scale = torch.where(i == j, 0.5, 1.0).double()
    # distances() takes r_i - r_j + shift.B: the opposite orientation, same length
    return i, j, -shift, scale
