"""Small IVF batches are scanned pair by pair without a plan only where the lists are even enough: what the
longest lists cost every query has to stay below a plan's cost (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu

ROWS, DIMS, NLIST, NPROBE = 200_000, 128, 512, 16
PAIRS, PLAN = 5, 7  # kernels: prep, two of the probe, scan, merge; with a plan two more


@pytest.fixture(scope="module")
def rows():
    m = np.random.default_rng(3).standard_normal((ROWS, DIMS), dtype=np.float32)
    return m / np.linalg.norm(m, axis=1, keepdims=True)


def opened(m, share):
    """One list with that share of the rows, the others even."""
    rng = np.random.default_rng(5)
    member = rng.integers(0, NLIST, ROWS)
    member[:int(share * ROWS)] = 0
    off = np.zeros(NLIST + 1, dtype=np.uint64)
    off[1:] = np.cumsum(np.bincount(member, minlength=NLIST))
    index = NNdex(m, normalized=True, autotune=False)
    index.load_ivf({"centroids": m[-NLIST:], "cluster_offsets": off,
                    "original_indices": np.argsort(member, kind="stable").astype(np.uint64),
                    "init_rows": np.arange(NLIST, dtype=np.uint64)})
    index.set_nprobe(NPROBE)
    return index


@pytest.mark.parametrize("share,nq,kernels", [
    (0.0, 1, PAIRS), (0.0, 32, PAIRS), (0.0, 33, PLAN),
    (0.3, 1, PAIRS), (0.3, 32, PLAN),   # 60,000 rows that 32 queries may all probe
    (0.9, 1, PLAN),                     # 180,000 rows in 32 chunks would outlast the rest
])
def test_uneven_lists_take_the_plan(rows, share, nq, kernels):
    index = opened(rows, share)
    q = rows[-NLIST:-NLIST + 1] + np.float32(0.02) * np.random.default_rng(nq).standard_normal((nq, DIMS), dtype=np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)  # all beside list 0's centroid
    idx, sim = index.search(q, k=10)
    st = index.last_search_stats()
    assert (st["path"], st["kernel_launches"]) == (4, kernels), st
    many, msim = index.search(np.vstack([q, rows[:64]]), k=10)  # with the plan
    np.testing.assert_array_equal(idx.reshape(nq, -1), many[:nq])
    np.testing.assert_array_equal(sim.reshape(nq, -1).view(np.uint32), msim[:nq].view(np.uint32))
