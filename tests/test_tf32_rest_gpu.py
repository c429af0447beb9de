"""Data on which most collections of the two-pass TF32 scan overflow: after such a batch the next ones take the
FP32 scan, on host and device buffers, and the two-pass scan is tried again later (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex
from test_reruns_gpu import on_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("buffers", ["host", "device"])
@pytest.mark.parametrize("nq", [40, 300])
def test_batches_after_a_vain_one_take_the_fp32_scan(nq, buffers):
    rng = np.random.default_rng(nq)
    distinct = rng.standard_normal((5, 128), dtype=np.float32)
    m = distinct[rng.integers(0, 5, 100_000)]
    q = (distinct[rng.integers(0, 5, nq)] + np.float32(0.2) * rng.standard_normal((nq, 128), dtype=np.float32))
    index = NNdex(m, autotune=False)
    paths, listed, first = [], [], None
    for _ in range(34):
        got = index.search(q, k=10) if buffers == "host" else on_device(index, q)
        st = index.last_search_stats()
        paths.append(st["path"])
        listed.append(st["fp32_fallback_queries"])
        first = first or got
        np.testing.assert_array_equal(got[0], first[0])
        np.testing.assert_array_equal(got[1].view(np.uint32), first[1].view(np.uint32))
    assert paths == [7] + 31 * [1] + [7, 1]
    assert listed == [nq] + 31 * [0] + [nq, 0]


@pytest.mark.parametrize("buffers", ["host", "device"])
def test_a_minority_that_overflows_changes_nothing(buffers):
    rng = np.random.default_rng(1)
    m = rng.standard_normal((60_000, 128), dtype=np.float32)
    m[:9_000] = m[0]
    q = rng.standard_normal((64, 128), dtype=np.float32)
    q[::3] = m[0] + np.float32(1e-3) * rng.standard_normal((22, 128), dtype=np.float32)
    index = NNdex(m, autotune=False)
    for _ in range(4):
        index.search(q, k=10) if buffers == "host" else on_device(index, q)
        st = index.last_search_stats()
        assert st["path"] == 7 and 22 <= st["fp32_fallback_queries"] <= 32, st
