"""Prefix sums without allocation of two runtimes at the same time."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1 << 24) + 5, 4097])
def test_noalloc_prefix_sums_of_two_runtimes_overlap(cuda_lib, n):
    """each runtime has tile sums of its own: calls on two streams, not
    waited for in between, give what single calls give"""
    import torch

    import orq_b200 as orq

    data, want, rts, streams, got = [], [], [], [], []
    for k in range(2):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            rt = orq.Runtime(seed=5 + k)
            v = rt.secret_share_a((np.arange(n, dtype=np.uint64) * np.uint64(3 + k)).astype(np.uint64), 0)
            w = v.clone()
            orq.prefix_sum(w)
            s.synchronize()
        data.append(v)
        want.append(w)
        rts.append(rt)
        streams.append(s)
    for rep in range(4):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                got.append((k, data[k].clone()))
        torch.cuda.synchronize()
        for k, v in got[-2:]:
            ptrs = (ctypes.c_void_p * 3)(*[v.shares[j].data_ptr() for j in range(3)])
            assert cuda_lib.orqcu_prefix_sum_a_noalloc(rts[k].h, 8, ctypes.c_size_t(n), ptrs) == 0
    torch.cuda.synchronize()
    for k, v in got:
        assert torch.equal(v.shares, want[k].shares)
