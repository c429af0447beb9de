"""The second pass 2 of overflowed collections is weighed with its reading of the copy: where it serves one query, but
the copy is long and its rows are short, the FP32 scan of that query costs less (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex, _lib
from test_group_maxima_gpu import force

pytestmark = pytest.mark.gpu

RETRY, RERUN = 6, 2  # kernels: the higher T (two), the gather, the scan, the rerank (two); the FP32 scan and merge


def unit(x):
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def opened(seed):
    """Clusters of 6,500 rows each, some of them close together, and queries of theirs. FP8's bound takes in a
    cluster; a pass 1 on every 32nd tile leaves T low, so that a few collections overflow and the next T saves them."""
    rng = np.random.default_rng(seed)
    centres = rng.standard_normal((200, 8), dtype=np.float32)

    def points(n):
        return unit(centres[rng.integers(0, 200, n)] + np.float32(0.2) * rng.standard_normal((n, 8), dtype=np.float32))

    index = NNdex(points(1_300_000), normalized=True, precision="fp8")
    force(index, 0, 1, 5, _lib.NNDEX_PRECISION_FP8, 0, 3, 32)
    return index, points(400)


def saved_query():
    """An index, a query whose collection overflows and that the second pass serves, and the launches without either."""
    for seed in range(10):
        index, q = opened(seed)
        plain = None
        for x in q:
            index.search(x, k=5)
            st = index.last_search_stats()
            if st["pass2_rows"] < 8192:
                plain = st["kernel_launches"]
            elif plain and st["kernel_launches"] == plain + RETRY and st["fp32_fallback_queries"] == 0:
                return index, x, plain
    pytest.fail("no such query")


def test_a_costly_retry_rests():
    index, q, plain = saved_query()
    launches, want = [], None
    for _ in range(66):
        got = index.search(q, k=5)
        st = index.last_search_stats()
        assert st["fp32_fallback_queries"] == (0 if st["kernel_launches"] == plain + RETRY else 1), st
        launches.append(st["kernel_launches"])
        want = want or got
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    assert launches.count(plain + RETRY) == 2 and launches.count(plain + RERUN) == 64, launches
