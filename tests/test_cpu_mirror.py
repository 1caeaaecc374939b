"""Host logic of the Python mirror that needs no GPU."""
import pytest
import torch

import orq_b200


@pytest.mark.parametrize("shape", [(2, 5), (1, 5), (0, 5), (2, 5, 2)])
def test_fewer_than_three_share_rows_are_refused(shape):
    """the share pointers come from the base and the row stride: a tensor
    without three rows must not give pointers past its end"""
    t = torch.zeros(shape, dtype=torch.int64)
    with pytest.raises(IndexError):
        orq_b200._rows3(t)
    with pytest.raises(IndexError):
        orq_b200._flat([orq_b200.BSharedVector(None, torch.zeros((3, 4), dtype=torch.int64)),
                        orq_b200.BSharedVector(None, t)])


@pytest.mark.parametrize("make", [
    lambda: torch.zeros((3, 7), dtype=torch.int32),
    lambda: torch.zeros((4, 7), dtype=torch.int8),
    lambda: torch.zeros((3, 9), dtype=torch.int64)[:, 2:],
    lambda: torch.zeros((6, 5), dtype=torch.int16)[::2],
    lambda: torch.zeros((3, 5, 2), dtype=torch.int64),
    lambda: torch.zeros((3, 1), dtype=torch.int64).expand(3, 4),
    lambda: torch.zeros((3, 0), dtype=torch.int64),
])
def test_share_rows_are_the_tensors_rows(make):
    t = make()
    assert orq_b200._rows3(t) == tuple(t[j].data_ptr() for j in range(3))
