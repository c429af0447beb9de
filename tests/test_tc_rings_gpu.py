"""The two-pass tensor-core scans at the row lengths where their ring of shared-memory stages changes
form (query slabs resident or streamed, three or four stages), flat and over lists (needs a B200): the
FP32 scan's rows and scores, bit for bit, with batches that leave query blocks and tiles partly filled.
"""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


def data(rows, dims, nq):
    rng = np.random.default_rng(rows + dims + nq)
    c = rng.normal(size=(64, dims)).astype(np.float32)
    base = c[rng.integers(0, 64, rows)] + 0.5 * rng.normal(size=(rows, dims)).astype(np.float32)
    q = c[rng.integers(0, 64, nq)] + 0.5 * rng.normal(size=(nq, dims)).astype(np.float32)
    return base.astype(np.float32), q.astype(np.float32)


def same(a, b):
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1].view(np.uint32), b[1].view(np.uint32))


@pytest.mark.parametrize("precision,dims", [("bf16", 320), ("bf16", 384), ("bf16", 448), ("bf16", 500), ("bf16", 576),
                                            ("bf16", 640), ("fp8", 768), ("fp8", 1000), ("fp8", 1152)])
@pytest.mark.parametrize("nq,k", [(130, 10), (257, 33)])
def test_flat_rings(precision, dims, nq, k):
    base, q = data(5011, dims, nq)
    index = NNdex(base, precision=precision, autotune=False)
    got = index.search(q, k=k)
    assert index.last_search_stats()["path"] == (2 if precision == "bf16" else 3)
    index.set_precision("fp32")
    same(got, index.search(q, k=k))


@pytest.mark.parametrize("dims", [384, 512, 600])
def test_list_rings(dims):
    base, q = data(20_011, dims, 300)
    index = NNdex(base, approx=True, precision="auto", nlist=20, kmeans_iters=2, seed=3, nprobe=6, autotune=False)
    got = index.search(q, k=10)
    assert index.last_search_stats()["path"] == 5
    index.set_precision("fp32")
    same(got, index.search(q, k=10))
