"""The charge solves refuse arrays with fewer values than atoms, pairs or frames,
and arrays on another device, before anything of them reaches a kernel (so the
first test needs no GPU)."""
import pytest
import torch

N, P, NF = 6, 10, 3
ONE = {"positions": (N, 3), "box": (3, 3), "chi": (N,), "hardness": (N,), "eta": (N,), "pairs": (P, 2), "ds": (P,),
       "scales": (P,)}
MANY = {k: (NF,) + s for k, s in ONE.items()}
WRONG = [("chi", (N - 1,)), ("hardness", (N - 1,)), ("eta", (1,)), ("ds", (P - 1,)), ("scales", (P - 1,)),
         ("pairs", (P, 1)), ("positions", (N, 2)), ("box", (2, 3))]


def _call(dev, frames, elsewhere=None, **wrong):
    from admp_b200.qeq import QEqForceModule, pgrad_optimize, qeq_solve_frames
    g = torch.Generator().manual_seed(1)
    a = {}
    for k, s in dict(MANY if frames else ONE, **wrong).items():
        x = torch.zeros(s, dtype=torch.long) if k == "pairs" else torch.rand(s, dtype=torch.float64, generator=g) + 5
        if k == "box":
            x = torch.eye(3, dtype=torch.float64).expand(NF, 3, 3) * 12 if frames and s == MANY["box"] else x
            x = torch.eye(3, dtype=torch.float64) * 12 if s == ONE["box"] else x
        a[k] = x.to(dev if k != elsewhere else "cpu")
    m = QEqForceModule(4.0, 1e-4, kmesh=8, max_iter=200)
    C = torch.ones(1, N, dtype=torch.float64, device=dev)
    if frames:
        return qeq_solve_frames(m, a["positions"], a["box"], a["chi"], a["hardness"], a["eta"], a["pairs"], a["ds"],
                                a["scales"], C)
    return pgrad_optimize(m, None, a["positions"], a["box"], a["chi"], a["hardness"], a["eta"], a["pairs"], a["ds"],
                          a["scales"], C, torch.zeros(1, dtype=torch.float64, device=dev))[1]


@pytest.mark.parametrize("name,shape", WRONG)
def test_short_arrays_are_refused(name, shape):
    with pytest.raises(ValueError, match="are needed"):
        _call("cpu", False, **{name: shape})


@pytest.mark.parametrize("name,shape", [("ds", (NF, P - 1)), ("scales", (NF - 1, P)), ("pairs", (NF, P, 1)),
                                        ("box", (NF - 1, 3, 3)), ("positions", (NF, N, 2))])
def test_short_arrays_of_frames_are_refused(name, shape):
    with pytest.raises(ValueError, match="are needed"):
        _call("cpu", True, **{name: shape})


@pytest.mark.gpu
@pytest.mark.parametrize("frames", [False, True])
@pytest.mark.parametrize("name", ["box", "chi", "hardness", "eta", "pairs", "ds", "scales"])
def test_arrays_elsewhere_are_refused(cuda, frames, name):
    with pytest.raises(RuntimeError, match="positions on cuda"):
        _call(cuda, frames, elsewhere=name)
    assert _call(cuda, frames).numel() == (NF * N if frames else N)


@pytest.mark.gpu
def test_arrays_that_nothing_reads_may_be_short(cuda):
    """Without damping the widths are not read, without pair terms the pair list."""
    from admp_b200 import _lib as L
    from admp_b200.qeq import QEqForceModule
    r = lambda *s: torch.rand(*s, dtype=torch.float64, device=cuda)  # noqa: E731
    pos, box, chi, hard = r(N, 3) * 10, torch.eye(3, dtype=torch.float64, device=cuda) * 12, r(N), r(N) + 10
    pairs = torch.tensor([[0, 1], [2, 3]], device=cuda)
    for rspace, ds in ((True, r(2) + 2), (False, r(1))):
        m = QEqForceModule(4.0, 1e-4, kmesh=8, damping=False, rspace=rspace)
        for eta in (r(1), torch.zeros(1, dtype=torch.float64), None):
            q, _, _, st = m._solve(torch.zeros_like(chi), pos, box, chi, hard, eta, pairs, ds, torch.ones_like(ds), None,
                                   None, False, 1e-10, 100)
            assert st == L.OK and bool(torch.isfinite(q).all())
