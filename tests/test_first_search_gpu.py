"""The first search of an index: a small batch needs no pinned allocation (opening has room for it), larger
batches and small ones in turn use the right buffers (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("approx", [False, True])
@pytest.mark.parametrize("nq", [1, 12, 64])
def test_small_first_batches_allocate_no_pinned_memory(nq, approx):
    rng = np.random.default_rng(nq)
    m = rng.standard_normal((20_000, 64), dtype=np.float32)
    q = rng.standard_normal((nq, 64), dtype=np.float32)
    index = NNdex(m, approx=approx, autotune=False, seed=1)
    want, path = index.search(q, k=10), index.last_search_stats()["path"]
    L, failed = _lib.lib(), []
    try:
        for skip in range(40):  # fail each allocation of the first search in turn
            index = NNdex(m, approx=approx, autotune=False, seed=1)
            L.nndex_cuda_inject_alloc_failures_after(skip, 1)
            try:
                got = index.search(q, k=10)
            except RuntimeError as e:
                failed.append(str(e))
                continue
            finally:
                L.nndex_cuda_inject_alloc_failures(0)
            np.testing.assert_array_equal(got[0], want[0])
            if index.last_search_stats()["path"] == path:
                break  # no allocation was left to fail
        else:
            pytest.fail("every allocation failed the search")
    finally:
        L.nndex_cuda_inject_alloc_failures(0)
    assert failed and not [e for e in failed if "pinned" in e], failed


def test_batches_of_all_sizes_in_turn():
    rng = np.random.default_rng(3)
    m = rng.standard_normal((30_000, 100), dtype=np.float32)
    q = rng.standard_normal((400, 100), dtype=np.float32)
    index = NNdex(m, autotune=False)
    want = [np.vstack(p) for p in zip(*(index.search(q[a:a + 8], k=50) for a in range(0, 400, 8)))]
    # queries and results below, above and just at 64 KB (163 queries; 109 of 50 results with their counts)
    for n, k in ((8, 50), (163, 10), (164, 10), (400, 50), (5, 50), (108, 50), (109, 50), (110, 50), (400, 1), (8, 50)):
        for _ in range(3):
            got = index.search(q[:n], k=k)
            np.testing.assert_array_equal(got[0], want[0][:n, :k])
            np.testing.assert_array_equal(got[1].view(np.uint32), np.ascontiguousarray(want[1][:n, :k]).view(np.uint32))
