"""Aggregation levels without min / max, which run in kernels of their own."""
import numpy as np
import pytest

from replay import BIT_OR, COPY, COUNT, SUM, VALID, GpuBackend, OracleBackend, same

pytestmark = pytest.mark.gpu


def replay(be, n, w, nkeys, boolean, reverse):
    from oracle.oracle import splitmix64_fast

    dt = {4: np.uint32, 8: np.uint64}[w]
    st = splitmix64_fast(77, 8 * n)
    keys = [be.share((np.sort(st[:n] % np.uint64(n // 4 + 1)) >> np.uint64(k)).astype(dt), False, k) for k in range(nkeys)]
    b = [be.share((st[(2 + i) * n:(3 + i) * n] & m).astype(dt), False, 0)
         for i, m in enumerate((np.uint64(0xFFFFFFFF), np.uint64(1), np.uint64(0xFFFFFFFF)))]
    sel = be.share((st[5 * n:6 * n] & np.uint64(1)).astype(dt), False, 1)
    a = be.share((st[6 * n:7 * n] & np.uint64(0xFFFF)).astype(dt), True, 0)
    bs = list(zip(b, (COPY, VALID, BIT_OR)))
    bo, ao = be.aggregate(keys, bs, [] if boolean else [(a, SUM), (a, COUNT)], reverse, sel if nkeys > 1 else None)
    return {**{f"b{i}": be.np(x) for i, x in enumerate(bo)}, **{f"a{i}": be.np(x) for i, x in enumerate(ao)}}


SIZES = [(4, 2), (4, 256), (4, 512), (4, 1024), (4, 1 << 14), (8, 128), (8, 256), (8, 1 << 13)]


# a unit is 16 bytes: fewer than 128 of them, a CTA, a few for each of 148 CTAs,
# and more than one for every thread of 148 CTAs of 256
@pytest.mark.parametrize("w,n,nkeys,reverse,boolean",
                         [(w, n, k, k > 1, b) for w, n in SIZES for k in (1, 3) for b in (True, False)]
                         + [(4, 1 << 18, 1, False, True), (8, 1 << 17, 1, False, True)])
def test_levels_without_minmax_match_restatement(cuda_lib, oracle_lib, w, n, nkeys, reverse, boolean):
    gpu = replay(GpuBackend(61), n, w, nkeys, boolean, reverse)
    cpu = replay(OracleBackend(61), n, w, nkeys, boolean, reverse)
    assert gpu.keys() == cpu.keys()
    for k in gpu:
        assert same(gpu[k], cpu[k]), k
