"""The serving loop's admission estimates against what requests take."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(1, 1), (1000, 70), (32768, 17), (32768, 18), (65535, 3), (65536, 66), (200000, 12),
                                     (1 << 20, 3)])
def test_permutation_bytes_are_what_the_pool_takes(cuda_lib, n, count):
    import torch

    import orq_b200 as orq

    rt = orq.Runtime(seed=5)
    rt.reserve_permutations(n, count)
    rt.reseed(5)  # (drops them)
    assert rt.trim() == orq.permutation_bytes(n, count, torch.cuda.get_device_properties(0).multi_processor_count)


@pytest.mark.parametrize("protocol", ["quick", "radix"])
@pytest.mark.parametrize("kind,n", [("sort", 20000), ("sort", 32768), ("sort", 65536), ("sort", 262144),
                                    ("groupby", 32768), ("groupby", 131072), ("join", 20000), ("join", 65536)])
def test_requests_stay_within_their_estimate(cuda_lib, kind, n, protocol):
    import torch

    import orq_b200 as orq
    from orq_b200.serve import Request, estimate_bytes, run_request

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_reserved()
    rt = orq.Runtime(seed=5)
    run_request(rt, Request(0, kind, n, 5), protocol)
    torch.cuda.synchronize()
    used = rt.trim() + torch.cuda.max_memory_reserved() - held
    rt.close()
    assert used <= estimate_bytes(kind, n, protocol) <= 2 * used + (128 << 20)
