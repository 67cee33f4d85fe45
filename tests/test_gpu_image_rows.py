"""Image neighbour list with a block per atom: the order of the pairs, cells of
one atom, more images than the shared table, more images within the cutoff than
the shared buffer of the nnei cut, and open boundaries, against the oracle."""
import numpy as np
import pytest
import torch

from _gpu_helpers import T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,size,rc,nnei", [
    (1, 4.0, 9.0, -1), (1, 4.0, 9.0, 20), (2, 3.0, 3.1, -1), (40, 8.0, 9.0, -1), (40, 8.0, 9.0, 100),
    (33, 30.0, 4.0, 0),
    (3, 1.5, 9.0, -1),       # 13^3 images: past the table
    (3, 1.5, 9.0, 1600),     # and thousands within the cutoff: past the buffer of the cut
    (300, None, 4.0, -1), (300, None, 8.0, 12)])
def test_image_rows_match_oracle(cuda, n, size, rc, nnei):
    from admp_b200.ops import image_neighbor_pairs
    from oracle import admp_oracle as O
    rng = np.random.default_rng(n)
    box = None
    pos = rng.random((n, 3)) * 12.0
    if size is not None:
        box = np.diag([size, 1.1 * size, 0.9 * size])
        box[1, 0], box[2, 1] = 0.2 * size, -0.1 * size
        pos = (rng.random((n, 3)) * 3 - 1) @ box  # unwrapped
    pairs, shifts, n_ij, ntr = image_neighbor_pairs(T(pos, cuda), None if box is None else T(box, cuda), rc, nnei)
    want = O.image_nblist(pos, box, rc, nnei)
    p, s = pairs.cpu().numpy(), shifts.cpu().numpy()
    got = {tuple(map(int, (*a, *b))) for a, b in zip(p, s)}
    ref = {tuple(map(int, (*a, *b))) for a, b in zip(want[0], want[1])}
    assert len(got) == len(p) and got == ref
    assert np.all(p[:n_ij, 0] < p[:n_ij, 1]) and np.all(p[n_ij:, 0] == p[n_ij:, 1])
    # i-major, then j within each block
    for blk in (p[:n_ij], p[n_ij:]):
        assert np.all(np.diff(blk[:, 0] * n + blk[:, 1]) >= 0)
