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


@pytest.mark.parametrize("other", [torch.zeros((3, 4), dtype=torch.int64), torch.zeros((3, 5), dtype=torch.int32),
                                   torch.zeros((3, 5, 2), dtype=torch.int64)])
def test_vectors_of_another_size_or_width_are_refused(other):
    """before anything is allocated or launched (there is no runtime here)"""
    A, B = orq_b200.ASharedVector, orq_b200.BSharedVector
    t = torch.zeros((3, 5), dtype=torch.int64)
    x, y, xa, ya = B(Lib(), t), B(Lib(), other), A(Lib(), t), A(Lib(), other)
    calls = [lambda: x & y, lambda: x.__iand__(y), lambda: x == y, lambda: x > y, lambda: x + y,
             lambda: x.extend_lsb(y), lambda: xa * ya, lambda: xa.__iadd__(ya)]
    for call in calls:
        with pytest.raises(ValueError):
            call()


class Lib:
    """a runtime whose library has entry points that nothing may call"""

    def __getattr__(self, name):
        return self if name == "lib" else None
