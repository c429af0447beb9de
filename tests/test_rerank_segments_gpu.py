"""The exact rerank of a two-pass batch's collected rows, at the collection sizes and batch sizes where its
work is dealt differently (needs a B200): below, at and past one round of segments, up to a full
collection. Rows and scores are the FP32 scan's, bit for bit.
"""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [20, 64, 65, 256, 257])
@pytest.mark.parametrize("near,k", [(31, 10), (512, 64), (513, 100), (3000, 128), (8000, 7)])
def test_collections_of_every_size(nq, near, k):
    # `near` rows lie within the scan's bound of each other around one point, so a query there collects
    # all of them or none
    rng = np.random.default_rng(near + nq)
    dims = 96
    m = rng.normal(size=(60_000, dims)).astype(np.float32)
    v = rng.normal(size=dims).astype(np.float32)
    at = rng.permutation(len(m))[:near]
    m[at] = v + 1e-5 * rng.normal(size=(near, dims)).astype(np.float32)
    q = (v + 0.05 * rng.normal(size=(nq, dims))).astype(np.float32)
    index = NNdex(m, precision="bf16", autotune=False)
    got = index.search(q, k=k)
    assert index.last_search_stats()["path"] == 2
    index.set_precision("fp32")
    # (never one query alone: the reference normalises a single vector with other roundings)
    want = [index.search(np.vstack([q[lo:lo + 7], q[:1]]), k=k) for lo in range(0, nq, 7)]
    assert np.array_equal(got[0], np.vstack([w[0][:-1] for w in want]))
    assert np.array_equal(got[1].view(np.uint32), np.vstack([w[1][:-1] for w in want]).view(np.uint32))
