"""Frame lists in several calls: the rows of one call, and a bounded scratch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,atoms", [(4096, 100), (2, 4 << 20), (4096, 50)])  # 2, 2 and 1 frames a call
def test_calls_of_a_few_frames_equal_one_call(cuda, monkeypatch, frames, atoms):
    from admp_b200 import nblist
    pos = torch.rand(5, 50, 3, dtype=torch.float64, device=cuda).mul(12).requires_grad_(True)
    box = (torch.eye(3, dtype=torch.float64, device=cuda) * torch.linspace(12, 14, 5, device=cuda)[:, None, None]).double()
    want = nblist.frame_pair_lists(pos, box, 5.0)
    monkeypatch.setattr(nblist, "_MAX_FRAMES", frames)
    monkeypatch.setattr(nblist, "_MAX_ATOMS", atoms)
    got = nblist.frame_pair_lists(pos, box, 5.0)
    for x, y in zip(got, want):
        assert torch.equal(x, y)
    g = [torch.autograd.grad(d.sum(), pos)[0] for d in (got[1], want[1])]
    assert float((g[0] - g[1]).abs().max()) < 1e-12


def test_scratch_of_many_atoms_is_bounded(cuda):
    """6 M atoms with next to no neighbours: the scratch is that of 4 M."""
    from admp_b200 import _lib as L
    from admp_b200.nblist import TorchNeighborList, frame_pair_lists
    nf, n = 300, 20000
    pos = torch.rand(nf, n, 3, dtype=torch.float32, device=cuda) * 200
    box = (torch.eye(3, device=cuda) * 200).expand(nf, 3, 3)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    pairs, ds, bs = frame_pair_lists(pos, box, 1.5)
    kept = sum(t.numel() * t.element_size() for t in (pairs, ds, bs)) + pos.numel() * 4
    peak = torch.cuda.max_memory_allocated() - before
    assert peak < L.load().admp_nblist_frames_workspace_size(4 * 2**20 // n, n) + 4 * kept
    for f in (0, 208, 209, 299):
        one = TorchNeighborList(1.5)(pos[f], box[f])
        assert torch.equal(pairs[f, :one.shape[0]], one)
