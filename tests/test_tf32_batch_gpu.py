"""The two-pass TF32 scan (FP32 indexes, 17 queries and more) against the FP32 scan, which serves the
same queries eight at a time: rows and scores are equal bit for bit (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


def fp32_scan(index, q, k):
    parts = [index.search(np.vstack([q[lo:lo + 7], q[:1]]), k=k) for lo in range(0, len(q), 7)]
    assert index.last_search_stats()["path"] == 1
    return np.vstack([p[0][:-1] for p in parts]), np.vstack([p[1][:-1] for p in parts])


def equal(index, q, k, path=7):
    ti, ts = index.search(q, k=k)
    st = index.last_search_stats()
    assert st["path"] == path, st
    fi, fs = fp32_scan(index, q, k)
    np.testing.assert_array_equal(ti, fi)
    np.testing.assert_array_equal(ts.view(np.uint32), fs.view(np.uint32))
    return st


@pytest.mark.parametrize("rows,dims,nq,k,centres", [
    (300_007, 100, 37, 33, 257),    # rows, dims and queries off every tile
    (130_000, 128, 17, 1, 0),       # the smallest batch
    (200_000, 64, 129, 10, 64),     # one query in the second block
    (16_640, 768, 64, 100, 64),     # streamed query slabs, a whole number of tiles
    (100_001, 256, 300, 256, 0),    # the largest k
    (1_100, 1_000, 256, 5, 0),      # five tiles: every one scanned by pass 1
    (4_300_000, 32, 40, 10, 512),   # sampled at the largest stride, one slab
])
def test_equals_fp32_scan(rows, dims, nq, k, centres):
    rng = np.random.default_rng(rows + dims + nq + k)

    def draw(n):
        x = rng.standard_normal((n, dims), dtype=np.float32)
        if centres:
            c = np.random.default_rng(7).standard_normal((centres, dims), dtype=np.float32)
            x = np.float32(0.3) * x + c[rng.integers(0, centres, n)]
        return x

    st = equal(NNdex(draw(rows)), draw(nq), k)
    assert st["fp32_fallback_queries"] == 0, st


def test_bound_follows_row_and_query_norms():
    # normalized=true keeps the caller's norms: 0.01 to 100, then values whose products overflow FP32
    rng = np.random.default_rng(31)
    m = rng.standard_normal((60_000, 96), dtype=np.float32)
    m *= (10.0 ** rng.uniform(-2, 2, size=(60_000, 1))).astype(np.float32)
    q = rng.standard_normal((48, 96), dtype=np.float32)
    q *= (10.0 ** rng.uniform(-2, 2, size=(48, 1))).astype(np.float32)
    index = NNdex(m, normalized=True)
    equal(index, q, 50)
    q[3] *= np.float32(1e36)  # norm ~1e37: its scores reach the overflow limit, the FP32 scan answers it
    q[4] = 0.0
    q[5] *= np.float32(1e-36)
    st = equal(index, q, 50)
    assert 1 <= st["fp32_fallback_queries"] <= 3, st


def test_overflowing_collections_fall_back_to_the_fp32_scan():
    # 9,000 copies of one row tie at the k-th score: the queries next to them collect every copy, more
    # than a collection holds, and are re-run; the others are not
    rng = np.random.default_rng(41)
    m = rng.standard_normal((80_000, 64), dtype=np.float32)
    m[5_000:14_000] = m[5_000]
    q = rng.standard_normal((60, 64), dtype=np.float32)
    q[10:30] = m[5_000] + np.float32(1e-3) * rng.standard_normal((20, 64), dtype=np.float32)
    st = equal(NNdex(m), q, 20)
    assert st["fp32_fallback_queries"] == 20, st


def test_small_batches_and_large_k_keep_their_paths():
    rng = np.random.default_rng(5)
    index = NNdex(rng.standard_normal((2_000, 16), dtype=np.float32))
    equal(index, rng.standard_normal((17, 16), dtype=np.float32), 10, path=1)  # too little work
    index = NNdex(rng.standard_normal((30_000, 128), dtype=np.float32))
    equal(index, rng.standard_normal((64, 128), dtype=np.float32), 257, path=1)
