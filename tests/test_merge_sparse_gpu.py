"""One-block merges of lists that are filled only at their start (more results asked for than a list has rows), at
a k whose lists line up with the threads: about as fast as at one whose lists do not (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


def test_lists_that_line_up_with_the_threads():
    rng = np.random.default_rng(9)
    nlist, each, dims = 300, 60, 64
    rows = nlist * each
    m = rng.standard_normal((rows, dims), dtype=np.float32)
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    index = NNdex(m, normalized=True, autotune=False)
    index.load_ivf({"centroids": m[:nlist].copy(), "cluster_offsets": np.arange(0, rows + 1, each).astype(np.uint64),
                    "original_indices": rng.permutation(rows).astype(np.uint64),
                    "init_rows": np.arange(nlist, dtype=np.uint64)})
    index.set_nprobe(nlist)
    q = m[-1]
    ms = {}
    for k in (250, 256):
        t = []
        for _ in range(40):
            idx, sim = index.search(q, k=k)
            t.append(index.last_search_stats()["device_ms"])
        ms[k] = np.median(t[8:])
        s = m.astype(np.float64) @ q.astype(np.float64)
        assert np.all(np.abs(np.sort(s)[::-1][:k] - sim) < 1e-5) and len(set(idx.tolist())) == k
    assert ms[256] < 1.8 * ms[250], ms
