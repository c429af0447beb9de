"""The one-block merge (k up to 256) against the split merge (k from 257): a search's first 256 results
do not depend on which of them ran (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


def alternating(rows, dims, period):
    """Rows along the first axis for every other run of `period` rows, against it for the others: the
    best keys crowd into half of the threads that read the lists, so the list above the cut overflows."""
    rng = np.random.default_rng(rows)
    m = rng.standard_normal((rows, dims), dtype=np.float32)
    m[:, 0] = np.where(np.arange(rows) // period % 2 == 0, 1.0, -1.0) * (3.0 + np.abs(m[:, 0]))
    return m, np.eye(1, dims, dtype=np.float32)


@pytest.mark.parametrize("rows,k", [(148 * 256, 256), (148 * 256, 255), (5_000, 256), (300, 256), (256, 256)])
def test_scan_merge(rows, k):
    m, q = alternating(rows, 32, 256)
    index = NNdex(m)
    long_i, long_s = index.search(q[0], k=257)
    i, s = index.search(q[0], k=k)
    n = min(k, rows)
    assert len(i) == n
    np.testing.assert_array_equal(i, long_i[:n])
    np.testing.assert_array_equal(s.view(np.uint32), long_s[:n].view(np.uint32))


@pytest.mark.parametrize("nprobe,k", [(64, 256), (64, 100), (3, 256), (1, 64)])
def test_list_merge(nprobe, k):
    m, q = alternating(40_000, 32, 256)
    index = NNdex(m, approx=True, nlist=64, kmeans_iters=2, seed=5, precision="fp32")
    index.set_nprobe(nprobe)
    long_i, long_s = index.search(np.repeat(q, 3, axis=0), k=257)
    i, s = index.search(np.repeat(q, 3, axis=0), k=k)
    np.testing.assert_array_equal(i, long_i[:, :i.shape[1]])
    np.testing.assert_array_equal(s.view(np.uint32), long_s[:, :i.shape[1]].view(np.uint32))
