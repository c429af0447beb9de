"""The IVF merges at the largest k that one block merges: as fast as at half of it (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


def test_merge_time_does_not_jump_at_the_largest_k():
    rng = np.random.default_rng(1)
    rows, dims, nlist, nprobe = 400_000, 64, 512, 32
    m = rng.standard_normal((rows, dims), dtype=np.float32)
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    member = rng.integers(0, nlist, rows)
    off = np.zeros(nlist + 1, dtype=np.uint64)
    off[1:] = np.cumsum(np.bincount(member, minlength=nlist))
    index = NNdex(m, normalized=True)
    index.load_ivf({"centroids": m[:nlist], "cluster_offsets": off,
                    "original_indices": np.argsort(member, kind="stable").astype(np.uint64),
                    "init_rows": np.arange(nlist, dtype=np.uint64)})
    index.set_nprobe(nprobe)
    ms = {}
    for k in (128, 256):
        t = []
        for i in range(40):
            index.search(m[nlist + i], k=k)
            t.append(index.last_search_stats()["device_ms"])
        ms[k] = np.median(t[8:])
    assert ms[256] < 1.4 * ms[128], ms
