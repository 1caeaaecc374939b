"""The permutation generator's corrections: what it does when its first guess
is wrong. The permutations and the nonces must be those of the C restatement
whatever was guessed first."""
import pytest

from replay import same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def orq(cuda_lib, oracle_lib):
    import orq_b200

    return orq_b200


def check_permutations(orq, rt, n, count, seed):
    from oracle.oracle import G01, Oracle

    o = Oracle(seed)
    rt.reserve_permutations(n, count)
    for m in range(count):
        got = rt.next_permutation(n).cpu().numpy()
        for g in range(3):
            want, _ = o.gen_perm(G01 + g, n)
            assert same(got[g], want), (m, g)
    for g in range(3):
        assert rt.nonce(orq.STREAM_G01 + g) == o.nonce(G01 + g)


# wrong predicted starts (the second of 70 permutations on: a pass verifies one
# more of each group, more passes than 64), and room for too few draws in the
# first pass, at the smallest sizes, at a chunk's 8192 draws and at the largest
@pytest.mark.parametrize("n,count,buffers,chunks", [(1, 70, 1, 0), (300, 70, 2, 0), (1000, 3, -1, 0), (32767, 4, 1, 0),
                                                    (1, 1, 0, 1), (63, 2, 0, 1), (2000, 3, 0, 1), (5000, 2, 1, 1),
                                                    (32767, 3, 0, 3)])
def test_small_permutations_from_wrong_first_guesses(orq, n, count, buffers, chunks):
    rt = orq.Runtime(seed=17)
    rt.tune_permutations(buffers=buffers, chunks=chunks)
    check_permutations(orq, rt, n, count, 17)


# windows too narrow for the thresholds: every chain starts over with wider ones
@pytest.mark.parametrize("n,count", [(65536, 4), (131071, 3), (262143, 2), (524288, 2), (1048577, 1)])
def test_chain_from_windows_too_narrow(orq, n, count):
    rt = orq.Runtime(seed=5)
    rt.tune_permutations(width=0.25)
    check_permutations(orq, rt, n, count, 5)


def test_the_environment_does_not_reach_the_generator(orq, monkeypatch):
    def launches():
        rt = orq.Runtime(seed=5)
        rt.reserve_permutations(100003, 2)  # (loads the kernels, fills the pool)
        rt.reseed(5)
        k = rt.kernels_launched()
        rt.reserve_permutations(100003, 2)
        return rt.kernels_launched() - k

    want = launches()
    monkeypatch.setenv("ORQ_FY_WIDTH", "none")
    assert launches() < 1.5 * want  # (a second chain doubles them)


@pytest.mark.parametrize("n,count", [(65536, 3), (300001, 2)])
def test_chain_after_lists_that_overflow(orq, n, count):
    """windows so wide that runs of the classification hold more uncertain
    draws than they keep: whatever becomes of that call, the next ones are right"""
    rt = orq.Runtime(seed=23)
    rt.tune_permutations(width=1000.0)
    try:
        rt.reserve_permutations(n, 1)
    except orq.OrqError:
        pass
    rt.reseed(23)
    rt.tune_permutations()
    check_permutations(orq, rt, n, count, 23)


@pytest.mark.parametrize("n,count,width", [(65536, 2, 1000.0), (100003, 3, 60.0), (524287, 1, 400.0)])
def test_chain_from_windows_too_wide(orq, n, count, width):
    """lists that overflow are answered with narrower windows"""
    rt = orq.Runtime(seed=29)
    rt.tune_permutations(width=width)
    check_permutations(orq, rt, n, count, 29)


# both sides of the rule that sends permutations of M = 2^16 to the path of the
# small ones; there, many take one launch a pass and one batch of finalizes
@pytest.mark.parametrize("n,count", [(32768, 17), (32768, 18), (65535, 18), (50001, 66)])
def test_many_permutations_of_medium_size(orq, n, count):
    rt = orq.Runtime(seed=31)
    check_permutations(orq, rt, n, count, 31)
    k = rt.kernels_launched()
    rt.reserve_permutations(n, count)
    assert count < 18 or rt.kernels_launched() - k < 60
