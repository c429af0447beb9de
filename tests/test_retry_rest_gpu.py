"""The second pass 2 of overflowed collections (BF16 and FP8 scans): after a batch where it was in vain for most of
them, the next batches' overflowed queries go straight to the FP32 scan, and it is tried again later; where it
serves, it is run every time (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex
from test_reruns_gpu import on_device

pytestmark = pytest.mark.gpu

RETRY = 6  # kernels: the higher T (two), the gather, the scan, the rerank (two)


@pytest.mark.parametrize("buffers", ["host", "device"])
@pytest.mark.parametrize("precision", ["bf16", "fp8"])
def test_vain_retries_rest(precision, buffers):
    rng = np.random.default_rng(4)
    distinct = rng.standard_normal((4, 64), dtype=np.float32)
    m = distinct[rng.integers(0, 4, 60_000)]  # 15,000 equal rows each
    q = distinct[rng.integers(0, 4, 40)] + np.float32(0.1) * rng.standard_normal((40, 64), dtype=np.float32)
    index = NNdex(m, precision=precision, autotune=False)
    index.search(q, k=10)  # (the pass-1 stride rule settles)
    launches, first = [], None
    for _ in range(66):
        got = index.search(q, k=10) if buffers == "host" else on_device(index, q)
        st = index.last_search_stats()
        assert st["fp32_fallback_queries"] == 40, st
        launches.append(st["kernel_launches"])
        first = first or got
        np.testing.assert_array_equal(got[0], first[0])
        np.testing.assert_array_equal(got[1].view(np.uint32), first[1].view(np.uint32))
    base = min(launches[-40:])
    tries = [i for i, n in enumerate(launches) if n == base + RETRY]
    assert len(tries) == 2 and tries[1] - tries[0] == 32, launches


def test_serving_retries_stay():
    # FP8's wide bound over tight clusters of distinct rows: T from a sampled pass 1 collects a cluster, the second
    # T a part of it
    rng = np.random.default_rng(6)
    centres = rng.standard_normal((20, 128), dtype=np.float32)
    m = centres[rng.integers(0, 20, 200_000)] + np.float32(0.25) * rng.standard_normal((200_000, 128), dtype=np.float32)
    q = centres[rng.integers(0, 20, 256)] + np.float32(0.25) * rng.standard_normal((256, 128), dtype=np.float32)
    index = NNdex(m, precision="fp8", autotune=False)
    for _ in range(3):
        index.search(q, k=100)
    launches = []
    for _ in range(6):
        index.search(q, k=100)
        st = index.last_search_stats()
        launches.append((st["kernel_launches"], st["fp32_fallback_queries"]))
    assert len(set(launches)) == 1, launches
