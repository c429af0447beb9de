"""The probe among thousands of lists of which many have equal centroids (rows with few distinct values): the
reference's lists, and no quadratic work (needs a B200)."""
import time

import numpy as np
import pytest

from nndex_b200 import NNdex
from test_probe_gpu import probed_rows

pytestmark = pytest.mark.gpu


def opened(nlist, nprobe, distinct, dims, rows_each=3):
    rng = np.random.default_rng(nlist + nprobe + distinct)
    rows = rows_each * nlist
    m = rng.standard_normal((rows, dims), dtype=np.float32)
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    cent = rng.standard_normal((nlist, dims)).astype(np.float32)
    if distinct:
        cent = cent[rng.integers(0, distinct, nlist)]
    cent /= np.linalg.norm(cent, axis=1, keepdims=True)
    order = np.argsort(rng.permutation(np.arange(rows) % nlist), kind="stable")
    lay = {"centroids": cent, "cluster_offsets": np.arange(0, rows + 1, rows_each).astype(np.uint64),
           "original_indices": order.astype(np.uint64), "init_rows": np.zeros(nlist, dtype=np.uint64)}
    index = NNdex(m, normalized=True)
    index.load_ivf(lay)
    index.set_nprobe(nprobe)
    q = rng.standard_normal((40, dims), dtype=np.float32)
    return index, lay, q / np.linalg.norm(q, axis=1, keepdims=True)


@pytest.mark.parametrize("nlist,nprobe,distinct", [
    (8_192, 32, 3),     # thousands of lists share the best score
    (3_000, 500, 3),    # the largest block
    (3_000, 64, 40),    # the best score's lists are fewer than the probed ones
    (2_000, 10, 7),     # more equal lists than the band holds, fewer than the merge's list
    (5_000, 300, 1),    # every list ties
])
def test_probed_lists_among_equal_centroids(nlist, nprobe, distinct):
    index, lay, q = opened(nlist, nprobe, distinct, 64)
    k = min(3 * nprobe, 2_048)
    want = probed_rows(lay, q, nprobe, 3 * nlist)
    for batch in (q, q[:2]):
        idx, _ = index.search(batch, k=k)
        for i in range(len(batch)):
            assert set(idx[i].tolist()) == set(want[i].tolist()), i


def test_ties_cost_no_quadratic_time():
    def us(index, q):
        t = []
        for _ in range(25):
            a = time.perf_counter()
            index.search(q, k=5)
            t.append(time.perf_counter() - a)
        return np.median(t[5:])

    for n in (1, 40):
        spread, tied = (us(i, q[:n]) for i, _, q in (opened(8_192, 32, d, 64) for d in (0, 3)))
        assert tied < 10 * spread, (n, spread, tied)
