"""Statistics that are read after a call belong to that call (needs a B200)."""
import numpy as np
import pytest
import torch

from nndex_b200 import NNdex, _lib
from test_reruns_gpu import COPIES, K, data, on_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,path", [(12, 6), (72, 7)])
def test_counts_of_an_earlier_device_call_are_not_read_into_a_later_one(nq, path):
    m, q = data(nq)
    index = NNdex(m, autotune=False)
    on_device(index, q, synchronize=0)
    index.search(q[0], k=K)
    st = index.last_search_stats()
    assert (st["path"], st["fp32_fallback_queries"], st["certified"]) == (1, 0, 0), st
    on_device(index, q, synchronize=0)
    st = index.last_search_stats()
    assert st["path"] == path and st["fp32_fallback_queries"] >= len(q[::5]), st
    on_device(index, q[1:2], synchronize=0)
    assert index.last_search_stats()["fp32_fallback_queries"] == 0


def test_device_time_outlives_a_wait_check():
    m, q = data(12)
    index = NNdex(m, autotune=False)
    index.search(q, k=K)
    assert _lib.lib().nndex_cuda_check_bounded_wait(index.handle, 100_000) == _lib.NNDEX_ERR_TIMEOUT
    assert index.last_search_stats()["device_ms"] > 0


def test_listed_queries_are_summed_over_the_pieces_of_a_large_call():
    # a call runs in pieces of 16,384 queries
    rng = np.random.default_rng(2)
    m = rng.standard_normal((20_000, 32), dtype=np.float32)
    m[3_000:3_000 + COPIES] = m[3_000]
    q = rng.standard_normal((16_384 + 400, 32), dtype=np.float32)
    q[:50] = m[3_000] + np.float32(1e-3) * rng.standard_normal((50, 32), dtype=np.float32)
    q[-10:] = q[:10]
    index = NNdex(m, autotune=False)
    counts = {}
    for name, part in (("first", q[:16_384]), ("rest", q[16_384:]), ("all", q)):
        on_device(index, part, synchronize=0)
        st = index.last_search_stats()
        assert st["path"] == 7
        counts[name] = st["fp32_fallback_queries"]
    assert counts["first"] >= 50 and counts["rest"] >= 10
    assert counts["all"] == counts["first"] + counts["rest"], counts
    index.search(q, k=K)
    st = index.last_search_stats()
    assert (st["fp32_fallback_queries"], st["certified"]) == (counts["all"], 0), st
