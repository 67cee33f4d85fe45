"""The list operator indexes a box a frame and three coordinates an atom: calls
with fewer of either are refused before any pointer is taken (so these run
without a GPU; with one, the same through frame_pair_lists)."""
import pytest
import torch

CASES = [((6, 3), (1, 3, 3), 3), ((6, 3), (2, 3, 3), 3), ((6, 3), (4, 3, 3), 3), ((6, 3), (2, 3), 1), ((6, 3), (0,), 1),
         ((7, 3), (3, 3, 3), 3), ((6, 2), (3, 3, 3), 3), ((6,), (3, 3), 1)]


@pytest.mark.parametrize("pos,box,nf", CASES)
def test_operator_refuses_missing_boxes_and_coordinates(pos, box, nf):
    from admp_b200 import nblist  # noqa: F401  (loads the operators)
    with pytest.raises(IndexError):
        torch.ops.admp_b200.neighbor_list(torch.rand(pos, dtype=torch.float64), torch.rand(box, dtype=torch.float64), 1.0,
                                          nf)


@pytest.mark.gpu
@pytest.mark.parametrize("boxes", [1, 2])
def test_frames_need_a_box_each(cuda, boxes):
    from admp_b200.nblist import TorchNeighborList, frame_pair_lists
    pos = torch.rand(3, 20, 3, dtype=torch.float64, device=cuda) * 13
    box = torch.eye(3, dtype=torch.float64, device=cuda) * 13
    with pytest.raises(IndexError):
        frame_pair_lists(pos, box.expand(boxes, 3, 3), 5.0)
    with pytest.raises(RuntimeError):
        TorchNeighborList(5.0)(pos[0], box.cpu())
    pairs, ds, _ = frame_pair_lists(pos, box.expand(4, 3, 3), 5.0)  # a box more than frames, as before
    assert pairs.shape[0] == 3 and ds.shape[0] == 3
