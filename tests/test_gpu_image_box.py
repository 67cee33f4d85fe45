"""Image lists of boxes whose images cannot be counted (singular, or far thinner
than the cutoff) are refused; thin boxes within the range are not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("diag,rc", [((9.0, 9.0, 0.0), 5.0), ((9.0, 1e-4, 9.0), 500.0), ((1e-3, 1e-3, 1e-3), 5.0)])
def test_uncountable_images_are_refused(cuda, diag, rc):
    from admp_b200.nblist import dp_nblist, vesin_nblist
    pos = torch.rand(4, 3, dtype=torch.float64, device=cuda)
    box = torch.diag(torch.tensor(diag, dtype=torch.float64, device=cuda))
    with pytest.raises(ValueError):
        dp_nblist(pos, box, 100, rc)
    with pytest.raises(ValueError):
        vesin_nblist(pos, box, rc)
    assert dp_nblist(pos, torch.eye(3, dtype=torch.float64, device=cuda) * 9, 100, 5.0)[0].shape[1] == 2


def test_thin_box_counts_its_self_images(cuda):
    """One atom, a 0.01 A thin box: 2 x 500 images along it within 5 A, none across."""
    from admp_b200.nblist import dp_nblist
    box = torch.diag(torch.tensor([20.0, 20.0, 0.01], dtype=torch.float64, device=cuda))
    pairs, ds, _ = dp_nblist(torch.zeros(1, 3, dtype=torch.float64, device=cuda), box, 5000, 5.005)
    assert pairs.shape[0] == 1000
    assert abs(float(ds.max()) - 5.0) < 1e-12
