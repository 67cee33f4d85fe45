"""Rows of the warp-per-atom neighbour search against brute force: both cell
builds (one block, several launches), rows that outgrow the shared-memory
ordering buffer (256 neighbours), one, two and many cells per axis, a
triclinic cell, open boundaries, unwrapped positions, and both precisions."""
import numpy as np
import pytest
import torch

from _gpu_helpers import T

pytestmark = pytest.mark.gpu


def brute(pos, box, rc):
    """Pairs (i, j) sorted, with the FP64 minimum-image test of the list."""
    n, out = len(pos), []
    frac = pos @ np.linalg.inv(box) if box is not None else None
    for a in range(0, n, 512):
        if box is None:
            d2 = ((pos[None] - pos[a:a + 512, None]) ** 2).sum(-1)
        else:
            df = frac[None] - frac[a:a + 512, None]
            d2 = (((df - np.floor(df + 0.5)) @ box) ** 2).sum(-1)
        hit = d2 < rc * rc
        if box is not None:
            hit &= d2 > 1e-4
        hit[np.arange(hit.shape[0]), a + np.arange(hit.shape[0])] = False
        i, j = np.nonzero(hit)
        out.append(np.stack([i + a, j], 1))
    return np.concatenate(out)


CASES = [  # atoms, box length (None: open), rc, triclinic
    (33, 12.5, 6.0, False),      # two cells per axis
    (1, 12.5, 6.0, False),
    (700, 13.0, 6.0, False),     # ~285 neighbours a row: past the ordering buffer
    (257, 7.0, 3.4, False),      # two cells per axis, dense
    (900, 30.0, 4.0, True),      # seven cells per axis, triclinic
    (2048, 28.0, 5.0, False),    # the largest frame of the one-block build
    (2049, 28.0, 5.0, True),     # the smallest of the other
    (8192, 44.0, 5.0, False),
    (8193, 44.0, 5.0, True),
    (500, None, 4.0, False),
    (600, None, 30.0, False),    # everything within the cutoff: rows of 599
    (9000, None, 3.0, False),
]


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,length,rc,tilt", CASES)
def test_rows_match_brute_force(cuda, n, length, rc, tilt, dtype):
    from admp_b200.nblist import TorchNeighborList
    rng = np.random.default_rng(n)
    size = length if length is not None else 20.0
    box = np.diag([size, 1.05 * size, 1.1 * size])
    if tilt:
        box[1, 0], box[2, 0], box[2, 1] = 0.2 * size, -0.15 * size, 0.1 * size
    # unwrapped: some atoms sit one or two cells away
    shift = rng.integers(-2, 3, (n, 3)) if length is not None else np.zeros((n, 3))
    npdt = np.float64 if dtype == torch.float64 else np.float32
    pos = ((rng.random((n, 3)) + shift) @ box).astype(npdt)
    bx = box.astype(npdt) if length is not None else None
    nb = TorchNeighborList(rc)
    pairs = nb(T(pos, cuda, dtype), None if bx is None else T(bx, cuda, dtype))
    want = brute(pos.astype(np.float64), None if bx is None else bx.astype(np.float64), rc)
    assert np.array_equal(pairs.cpu().numpy(), want)  # the set and its (i, j) order
    assert np.array_equal(nb.get_buffer_scales().cpu().numpy(), (want[:, 0] < want[:, 1]).astype(np.int64))
    d = pos[want[:, 0]].astype(np.float64) - pos[want[:, 1]].astype(np.float64)
    if bx is not None:
        f = d @ np.linalg.inv(bx.astype(np.float64))
        d = (f - np.floor(f + 0.5)) @ bx.astype(np.float64)
    ref = np.linalg.norm(d, axis=1)
    # FP64: the inverse box and three products, a few ulp of the (unwrapped) coordinates; FP32 results round once
    tol = 1e-12 if dtype == torch.float64 else 2e-7
    assert len(ref) == 0 or np.abs(nb.get_ds().cpu().numpy() - ref).max() < tol * max(ref.max(), 1.0)


def test_nonfinite_position_is_refused_and_the_next_call_runs(cuda):
    from admp_b200 import _lib as L
    from admp_b200.nblist import TorchNeighborList
    pos = torch.rand(300, 3, dtype=torch.float64, device=cuda) * 13
    box = torch.eye(3, dtype=torch.float64, device=cuda) * 13
    bad = pos.clone()
    bad[7, 1] = float("nan")
    with pytest.raises(L.AdmpError):
        TorchNeighborList(5.0)(bad, box)
    assert TorchNeighborList(5.0)(pos, box).shape[0] > 0


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [1, 40, 8300])
def test_frames_equal_single_lists(cuda, n, dtype):
    """Frames with different pair counts (different boxes) against one list per
    frame: rows, padding, distances and their gradients."""
    from admp_b200.nblist import TorchNeighborList, frame_pair_lists
    rng = np.random.default_rng(n)
    sizes = [13.0, 15.0, 14.0] if n < 8000 else [44.0, 46.0, 45.0]
    box = T(np.stack([np.diag([s] * 3) + np.array([[0, 0, 0], [0.3, 0, 0], [0, 0.2, 0]]) for s in sizes]), cuda, dtype,
            grad=True)
    pos = T(rng.random((3, n, 3)) * 40.0, cuda, dtype, grad=True)
    pairs, ds, bs = frame_pair_lists(pos, box, 5.0)
    w = torch.linspace(0.5, 1.5, max(ds.shape[1], 1), dtype=dtype, device=cuda)[:ds.shape[1]]
    gpos, gbox = torch.autograd.grad((ds * w).sum(), [pos, box])
    counts = []
    for f in range(3):
        nb = TorchNeighborList(5.0)
        p1, b1 = pos[f].detach().requires_grad_(True), box[f].detach().requires_grad_(True)
        one = nb(p1, b1)
        k = one.shape[0]
        counts.append(k)
        assert torch.equal(pairs[f, :k], one) and torch.equal(bs[f, :k], nb.get_buffer_scales())
        assert torch.equal(ds[f, :k], nb.get_ds())
        assert not pairs[f, k:].any() and not bs[f, k:].any() and bool((ds[f, k:] == 1).all())
        if k:
            g1, g2 = torch.autograd.grad((nb.get_ds() * w[:k]).sum(), [p1, b1])
            # the same terms summed by atomics in another order: 1e-15 (FP64) / 1e-6 (FP32) of ~100 terms
            tol = 1e-12 if dtype == torch.float64 else 1e-4
            assert float((gpos[f] - g1).abs().max()) < tol * max(1.0, float(g1.abs().max()))
            assert float((gbox[f] - g2).abs().max()) < tol * max(1.0, float(g2.abs().max()))
    assert pairs.shape[1] == max(counts)
