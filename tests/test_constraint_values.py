"""Constraint values of a charge solve from host and device memory: missing ones
are zero, more than there are constraints raise, wherever they lie."""
import pytest
import torch


def _values(b, n):
    from admp_b200 import _lib as L
    flag, ptr, keep = L.constraint_values(b, n, b.device)
    if flag:
        return keep.tolist()
    return [ptr[k] for k in range(n)]


def _check(dev):
    for n, given, want in [(1, [0.5], [0.5]), (2, [0.5], [0.5, 0.0]), (3, [], [0.0] * 3), (2, [[1.0], [2.0]], [1.0, 2.0])]:
        for dt in (torch.float64, torch.float32):
            assert _values(torch.tensor(given, dtype=dt, device=dev), n) == want
    for n, k in [(1, 2), (2, 5)]:
        with pytest.raises(IndexError):
            _values(torch.ones(k, dtype=torch.float64, device=dev), n)


def test_host_values():
    _check("cpu")


@pytest.mark.gpu
def test_device_values(cuda):
    _check(cuda)
