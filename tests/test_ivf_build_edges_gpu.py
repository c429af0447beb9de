"""The IVF build at the sizes where its kernels change shape, against the oracle (needs a B200): rows of
more than 256, 512 and 1,024 values (lanes and loads of the seeding's screen), more than 1,024 lists (sort
blocks, the offsets' scan), more rows than one pass of a seeding block, and rows whose INT8 copy says
little (one value far above the others), so that most distances are taken exactly. Everything is exact:
the same seeds, centroids, lists and row order.
"""
import numpy as np
import pytest

from nndex_b200 import NNdex
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def spiky(rng, rows, dims):
    m = 0.01 * rng.normal(size=(rows, dims))
    m[np.arange(rows), rng.integers(0, dims, size=rows)] = rng.choice([-1.0, 1.0], size=rows)
    return m.astype(np.float32)


@pytest.mark.parametrize("rows,dims,nlist,iters,data", [
    (1500, 256, 20, 2, "gauss"),
    (1500, 257, 20, 2, "gauss"),
    (700, 530, 12, 2, "gauss"),
    (500, 1100, 10, 2, "gauss"),
    (4000, 24, 1100, 1, "gauss"),
    (800_000, 16, 4, 1, "gauss"),
    (3000, 128, 40, 2, "spiky"),
    (257, 16, 2, 1, "gauss"),
])
def test_ivf_build_edges(rows, dims, nlist, iters, data):
    rng = np.random.default_rng(rows + dims)
    m = spiky(rng, rows, dims) if data == "spiky" else rng.normal(size=(rows, dims)).astype(np.float32)
    index = NNdex(m, approx=True, nlist=nlist, kmeans_iters=iters, seed=11)
    st, storage = O.prepare_index(m, False)
    assert st == 0
    ref = O.IvfIndex(storage, nlist=nlist, iters=iters, seed=11)
    lay = index.ivf_layout()
    assert np.array_equal(lay["init_rows"], ref.init_rows)
    assert np.array_equal(lay["cluster_offsets"], ref.offsets)
    assert np.array_equal(lay["original_indices"], ref.original_indices)
    assert np.array_equal(lay["centroids"].view(np.uint32), ref.centroids.view(np.uint32))
