"""Admission estimates of the serving loop (host arithmetic)."""
import pytest

import orq_b200
from orq_b200 import serve

pytestmark = pytest.mark.usefixtures("cuda_lib")  # (built)


# the arithmetic of the generator's buffers: permutations and accepted offsets,
# and from 2^16 rows on (few: 2^15) three rings of four times the buffers, of 4
# MiB, that an eighth of the permutations is expected to use
@pytest.mark.parametrize("n,count,ring_buffers", [(1000, 3, 0), (32768, 3, 8), (65536, 66, 60), (262144, 66, 200),
                                                  (1 << 22, 44, 200)])
def test_permutation_bytes_cover_the_generator(n, count, ring_buffers):
    assert orq_b200.permutation_bytes(n, count) >= 24 * n * count + 3 * ring_buffers * (4 << 20)
    assert orq_b200.permutation_bytes(n, 0) == 0


def test_permutation_bytes_refuses_what_the_generator_refuses():
    for n, count, sms in ((1 << 31, 1, 148), (5, 1, 0)):
        with pytest.raises(orq_b200.OrqError):
            orq_b200.permutation_bytes(n, count, sms)


@pytest.mark.parametrize("kind,perms", [("sort", {"quick": 3, "radix": 66}), ("groupby", {"quick": 12, "radix": 75}),
                                        ("join", {"quick": 18, "radix": 81})])
@pytest.mark.parametrize("n", [1000, 20000, 32768, 65535, 65536, 100003, 262144, 1 << 20])
def test_estimates_hold_the_reserved_permutations(kind, perms, n):
    rows = 5 * n if kind == "join" else n
    for protocol in ("quick", "radix"):
        assert serve.estimate_bytes(kind, n, protocol) > orq_b200.permutation_bytes(rows, perms[protocol]) + 200 * rows
