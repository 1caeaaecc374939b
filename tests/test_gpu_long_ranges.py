"""Primitives over ranges long enough that a CTA goes chunk by chunk with the
constant parts of AES rounds 1 and 2 (4096 blocks a CTA, 64 passes in a
compare), across the end of a 1 MiB chunk and its last two blocks, whose counter
has a third byte."""
import numpy as np
import pytest

from replay import GpuBackend, OracleBackend, compare_inputs, prim_inputs, same

pytestmark = pytest.mark.gpu
U = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}


def backend(seed, sms):
    be = GpuBackend(seed)
    be.rt.set_sm_limit(sms)
    return be


# on 4 SMs, and on all of them
SIZES = [(1, 4800001, 4), (2, 2400003, 4), (4, 1200003, 4), (8, 600001, 4), (4, (1 << 23) + 1025, 0), (8, 3000017, 0)]


@pytest.mark.parametrize("w,n,sms", SIZES)
def test_and_multiply_and_b2a_match_restatement(cuda_lib, oracle_lib, w, n, sms):
    x, y = prim_inputs(n, 3, U[w])

    def run(be):
        xb, yb, xa, ya = (be.share(v, arith, p) for v, arith, p in ((x, False, 0), (y, False, 1), (x, True, 2), (y, True, 0)))
        return [be.np(v) for v in (xa, be.and_b(xb, yb), be.mul_a(xa, ya), be.b2a_bit(xb))]

    for name, a, b in zip(("share", "and", "multiply", "b2a"), run(backend(33, sms)), run(OracleBackend(33))):
        assert same(a, b), name


@pytest.mark.parametrize("w,n,sms", [(4, 1200003, 4), (8, 600001, 4), (4, 2000003, 0), (8, 1000003, 0)])
def test_compare_and_equality_match_restatement(cuda_lib, oracle_lib, w, n, sms):
    x, y = compare_inputs(n, 5, U[w])

    def run(be):
        xb, yb = be.share(x, False, 0), be.share(y, False, 1)
        eq, gt = be.compare(xb, yb)
        return [be.np(v) for v in (eq, gt, be.relops(xb, yb)[0])]

    for name, a, b in zip(("eq", "gt", "=="), run(backend(35, sms)), run(OracleBackend(35))):
        assert same(a, b), name


def test_16_byte_shares_do_not_depend_on_the_range_a_cta_takes(cuda_lib):
    """300001 elements on 4 SMs are long ranges, on 148 short ones"""
    import torch

    import orq_b200 as orq

    g = torch.Generator().manual_seed(1)
    x, y = (torch.randint(-(1 << 62), 1 << 62, (3, 300001, 2), generator=g).cuda() for _ in range(2))
    y[:, ::3] = x[:, ::3]
    out = []
    for sms in (4, 0):
        rt = orq.Runtime(seed=7)
        rt.set_sm_limit(sms)
        xb, yb, xa, ya = (rt.from_shares(v, a) for a in (False, True) for v in (x, y))
        out.append([(xb & yb).shares, (xa * ya).shares, (xb == yb).shares, (xb > yb).shares])
    for a, b in zip(*out):
        assert torch.equal(a, b)
