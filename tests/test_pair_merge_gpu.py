"""Small IVF batches are scanned pair by pair without a plan only where that leaves each query's merge few enough
keys: a slot of k for every chunk of the longest list, in each list that is probed (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu

ROWS, DIMS, NLIST, NPROBE = 200_000, 32, 512, 128
PAIRS, PLAN = 5, 7  # kernels: prep, two of the probe, scan, merge; with a plan two more


@pytest.fixture(scope="module")
def index():
    """A fifth of the rows in one list, 32 chunks of 1,280; the others even."""
    rng = np.random.default_rng(3)
    m = rng.standard_normal((ROWS, DIMS), dtype=np.float32)
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    member = rng.integers(1, NLIST, ROWS)
    member[:ROWS // 5] = 0
    off = np.zeros(NLIST + 1, dtype=np.uint64)
    off[1:] = np.cumsum(np.bincount(member, minlength=NLIST))
    index = NNdex(m, normalized=True, autotune=False)
    index.load_ivf({"centroids": m[-NLIST:], "cluster_offsets": off,
                    "original_indices": np.argsort(member, kind="stable").astype(np.uint64),
                    "init_rows": np.arange(NLIST, dtype=np.uint64)})
    index.set_nprobe(NPROBE)
    return index


@pytest.mark.parametrize("nq", [1, 4])
@pytest.mark.parametrize("k,kernels", [(1, PAIRS), (24, PAIRS), (25, PLAN), (256, PLAN)])  # 24: 98,304 keys
def test_large_merges_take_the_plan(index, k, kernels, nq):
    q = np.random.default_rng(k).standard_normal((64, DIMS), dtype=np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    idx, sim = index.search(q[:nq], k=k)
    st = index.last_search_stats()
    assert (st["path"], st["kernel_launches"]) == (4, kernels), st
    many, msim = index.search(q, k=k)  # with the plan
    np.testing.assert_array_equal(idx.reshape(nq, -1), many.reshape(64, -1)[:nq])
    np.testing.assert_array_equal(sim.reshape(nq, -1).view(np.uint32), msim.reshape(64, -1)[:nq].view(np.uint32))
