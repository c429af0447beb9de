"""The sampled first pass with group maxima (BF16 / FP8 and IVF list scans) returns the FP32 path's
results bit for bit, at the edges of its tiles, groups, spans and candidate lists (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


def mixture(rng, rows, dims, centers=64, sigma=0.25):
    c = np.random.default_rng(99).normal(size=(centers, dims)).astype(np.float32)
    return (c[rng.integers(0, centers, size=rows)] + np.float32(sigma) * rng.normal(size=(rows, dims))).astype(np.float32)


def force(index, ivf, nq, k, precision, nprobe, path, stride):
    """Installs the plan (path, pass-1 stride) for the shape, as a saved tuner cache would."""
    up = lambda v: 1 << (int(v) - 1).bit_length() if v > 1 else 1  # noqa: E731
    header = index.autotune_export().splitlines()[0]
    index.autotune_import(f"{header}\nshape ivf={ivf} nq={up(nq)} k={up(k)} precision={precision} nprobe={nprobe} "
                          f"plan path={path} stride={stride} qb=0 ms=1.0\n")


def fp32_scan(index, q, k):
    """The FP32 scan's results: it serves batches of up to eight queries."""
    index.set_precision("fp32")
    parts = [index.search(np.vstack([q[lo:lo + 7], q[:1]]), k=k) for lo in range(0, len(q), 7)]
    assert index.last_search_stats()["path"] == 1
    return np.vstack([p[0][:-1] for p in parts]), np.vstack([p[1][:-1] for p in parts])


@pytest.mark.parametrize("precision,rows,dims,nq,k,stride", [
    ("bf16", 16_384, 64, 1, 1, 8),         # the smallest sampled base, one query, one slab
    ("bf16", 16_641, 100, 129, 10, 8),     # one row in the last tile, one query in the last block
    ("bf16", 70_001, 256, 300, 10, 32),    # a part-empty last span, groups of 8 columns
    ("bf16", 400_003, 64, 200, 10, 8),     # groups of 32 columns, several tiles per span
    ("bf16", 60_000, 768, 130, 100, 8),    # streamed query slabs, four maxima per thread
    ("bf16", 120_000, 64, 70, 140, 8),     # the longest candidate lists the path takes at 64 dims
    ("bf16", 20_000, 128, 70, 100, 32),    # too few groups for k: heaps
    ("fp8", 16_385, 128, 64, 1, 8),
    ("fp8", 90_000, 512, 129, 100, 8),
    ("fp8", 300_001, 200, 257, 10, 32),
])
def test_sampled_pass_equals_fp32(precision, rows, dims, nq, k, stride):
    rng = np.random.default_rng(rows + dims + nq + k)
    m, q = mixture(rng, rows, dims), mixture(rng, nq, dims)
    if rows == 70_001:
        m[5_000:9_000] = m[4_999]  # mass ties: the listed words are truncated
    index = NNdex(m, precision=precision)
    force(index, 0, nq, k, {"bf16": 2, "fp8": 3}[precision], 0, {"bf16": 2, "fp8": 3}[precision], stride)
    ti, ts = index.search(np.vstack([q, q[:1]]) if nq == 1 else q, k=k)
    st = index.last_search_stats()
    assert st["path"] == {"bf16": 2, "fp8": 3}[precision]
    fi, fs = fp32_scan(index, np.vstack([q, q[:1]]) if nq == 1 else q, k)
    assert np.array_equal(ti, fi)
    assert np.array_equal(ts, fs)
    if nq > 1:
        assert st["pass1_tile_stride"] == stride


@pytest.mark.parametrize("rows,dims,nq,k,nlist,nprobe,stride", [
    (30_000, 64, 64, 10, 40, 8, 2),        # lists of a few tiles
    (50_000, 100, 300, 100, 50, 16, 4),    # more candidates than a list's groups
    (90_000, 128, 129, 10, 8, 4, 16),      # lists of several 4,096-row chunks
    (20_000, 256, 200, 1, 100, 3, 4),      # lists shorter than a tile: a query may have few groups
])
def test_sampled_list_scan_equals_fp32(rows, dims, nq, k, nlist, nprobe, stride):
    rng = np.random.default_rng(rows + dims + nq + k)
    m, q = mixture(rng, rows, dims, 300), mixture(rng, nq, dims, 300)
    index = NNdex(m, precision="auto", approx=True, nlist=nlist, kmeans_iters=4, seed=3)
    index.set_nprobe(nprobe)
    force(index, 1, nq, k, 0, nprobe, 5, stride)
    ti, ts = index.search(q, k=k)
    st = index.last_search_stats()
    assert st["path"] == 5 and st["pass1_tile_stride"] == stride
    index.set_precision("fp32")
    fi, fs = index.search(q, k=k)
    assert index.last_search_stats()["path"] == 4
    assert np.array_equal(ti, fi)
    assert np.array_equal(ts, fs)


@pytest.mark.parametrize("precision,nq", [("bf16", 70), ("fp8", 150)])
def test_overflowing_collection_gets_a_second_threshold(precision, nq):
    # One dense cluster of 30,000 rows the sample never meets (it sits in tiles that stride 32 skips)
    # next to unrelated rows: T is far too low, every query collects more than 8,192 rows, and the
    # k-th score of the rows it did collect finishes it without the FP32 scan.
    rng = np.random.default_rng(nq)
    dims = 128
    m = rng.normal(size=(256 * 80, dims)).astype(np.float32)
    v = rng.normal(size=(1, dims)).astype(np.float32)
    near = rng.uniform(0.2, 1.2, size=(256 * 62, 1)).astype(np.float32)
    cluster = v + near * rng.normal(size=(256 * 62, dims)).astype(np.float32)
    m[256:256 * 32] = cluster[:256 * 31]
    m[256 * 33:256 * 64] = cluster[256 * 31:]
    q = (v + np.float32(0.05) * rng.normal(size=(nq, dims))).astype(np.float32)
    index = NNdex(m, precision=precision)
    path = {"bf16": 2, "fp8": 3}[precision]
    force(index, 0, nq, 10, path, 0, path, 32)
    ti, ts = index.search(q, k=10)
    st = index.last_search_stats()
    assert st["path"] == path and st["fp32_fallback_queries"] == 0 and st["kernel_launches"] > 8, st
    fi, fs = fp32_scan(index, q, 10)
    assert np.array_equal(ti, fi)
    assert np.array_equal(ts, fs)
