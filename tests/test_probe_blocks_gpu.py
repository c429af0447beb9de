"""The probe's pick kernel has large blocks for few queries over more than 1,024 lists, small ones for more queries:
both pick the same lists, also where most centroids are equal (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu

ROWS, DIMS = 20_000, 48


@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("nlist,nprobe", [(1024, 4), (1025, 1), (1025, 64), (2048, 16), (2049, 64)])
def test_block_sizes_agree(nlist, nprobe, equal):
    rng = np.random.default_rng(nlist + nprobe)
    m = rng.standard_normal((ROWS, DIMS), dtype=np.float32)
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    member = rng.integers(0, nlist, ROWS)
    off = np.zeros(nlist + 1, dtype=np.uint64)
    off[1:] = np.cumsum(np.bincount(member, minlength=nlist))
    index = NNdex(m, normalized=True, autotune=False)
    index.load_ivf({"centroids": m[rng.integers(0, 3, nlist)] if equal else m[:nlist], "cluster_offsets": off,
                    "original_indices": np.argsort(member, kind="stable").astype(np.uint64),
                    "init_rows": np.arange(nlist, dtype=np.uint64)})
    index.set_nprobe(nprobe)
    q = m[rng.integers(0, ROWS, 340)] + np.float32(0.1) * rng.standard_normal((340, DIMS), dtype=np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    idx, sim = index.search(q, k=5)  # small blocks
    for lo, hi in [(0, 1), (1, 38), (38, 76), (76, 300)]:  # 1, 37, 38 and 224 queries
        part, psim = index.search(q[lo:hi], k=5)
        np.testing.assert_array_equal(part.reshape(hi - lo, -1), idx[lo:hi])
        np.testing.assert_array_equal(psim.reshape(hi - lo, -1).view(np.uint32), sim[lo:hi].view(np.uint32))
