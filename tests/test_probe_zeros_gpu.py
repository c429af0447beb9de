"""The probe where most centroids have a zero dot with the query (empty lists, rows without a dimension in common):
the reference's lists, at little more than the time of lists without zeros (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex
from test_probe_gpu import probed_rows

pytestmark = pytest.mark.gpu

NLIST, NPROBE, DIMS = 1_500, 100, 256


def opened(kind):
    rng = np.random.default_rng(8)
    rows = 3 * NLIST
    m = rng.standard_normal((rows, DIMS), dtype=np.float32)
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    q = rng.standard_normal((60, DIMS), dtype=np.float32)
    cent = rng.standard_normal((NLIST, DIMS)).astype(np.float32)
    if kind == "empty":  # two thirds of the centroids are zero
        cent[rng.random(NLIST) < 0.67] = 0.0
    elif kind == "disjoint":  # three dimensions each, few of them in common
        for x in (cent, q):
            keep = rng.integers(0, DIMS, (len(x), 3))
            y = np.zeros_like(x)
            np.put_along_axis(y, keep, np.take_along_axis(x, keep, 1), 1)
            x[:] = y
    cent /= np.maximum(np.linalg.norm(cent, axis=1, keepdims=True), np.float32(1e-20))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    order = np.argsort(rng.permutation(np.arange(rows) % NLIST), kind="stable")
    lay = {"centroids": cent, "cluster_offsets": np.arange(0, rows + 1, 3).astype(np.uint64),
           "original_indices": order.astype(np.uint64), "init_rows": np.zeros(NLIST, dtype=np.uint64)}
    index = NNdex(m, normalized=True, autotune=False)
    index.load_ivf(lay)
    index.set_nprobe(NPROBE)
    return index, lay, q


def device_ms(index, q):
    t = []
    for _ in range(30):
        index.search(q, k=5)
        t.append(index.last_search_stats()["device_ms"])
    return np.median(t[8:])


@pytest.mark.parametrize("kind", ["empty", "disjoint"])
def test_zero_dots(kind):
    index, lay, q = opened(kind)
    want = probed_rows(lay, q, NPROBE, 3 * NLIST)
    idx, _ = index.search(q, k=3 * NPROBE)
    for i in range(len(q)):
        assert set(idx[i].tolist()) == set(want[i].tolist()), i
    plain = device_ms(opened("plain")[0], q)
    assert device_ms(index, q) < 2.0 * plain
