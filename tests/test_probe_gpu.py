"""The probe's lists (TF32 scores, exact scores where they leave the choice open) are the reference's:
the nprobe best centroids by the f32 rounding of the FP64 dot, lower index on ties (needs a B200)."""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


def probed_rows(lay, q, nprobe, rows):
    """Rows of the nprobe best lists per query, from FP64 dots in numpy."""
    dims = lay["centroids"].shape[1]
    c = np.zeros((len(q), len(lay["centroids"])), dtype=np.float64)
    for d in range(dims):  # index order, as the reference adds
        if d < q.shape[1]:
            c += q[:, d:d + 1].astype(np.float64) * lay["centroids"][None, :, d].astype(np.float64)
    s = c.astype(np.float32)
    order = np.argsort(-s, axis=1, kind="stable")[:, :nprobe]
    out = []
    off = lay["cluster_offsets"].astype(np.int64)
    for lists in order:
        out.append(np.concatenate([lay["original_indices"][off[i]:off[i + 1]] for i in lists]))
    return out


@pytest.mark.parametrize("nlist,nprobe,dims,nq,kind", [
    (300, 1, 32, 1, "gauss"), (300, 64, 40, 5, "gauss"), (1000, 65, 100, 130, "gauss"), (1000, 512, 64, 3, "gauss"),
    (700, 600, 64, 4, "gauss"),      # more lists than the pick holds: exact scores of every pair
    (300, 300, 32, 3, "gauss"),      # every list
    (600, 20, 64, 9, "ties"),        # equal centroids at the cut: lower index first
    (1100, 40, 64, 6, "close"),      # more lists between the certain ones than fit shared memory
    (300, 10, 1_000, 70, "gauss"),   # streamed query slabs
])
def test_probed_lists(nlist, nprobe, dims, nq, kind):
    rng = np.random.default_rng(nlist + nprobe + dims)
    rows = 3 * nlist
    m = rng.standard_normal((rows, dims), dtype=np.float32)
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    cent = rng.standard_normal((nlist, dims)).astype(np.float32)
    if kind == "ties":
        cent[::2] = cent[0]
    if kind == "close":
        cent = (cent[:1] + np.float32(1e-4) * cent).astype(np.float32)
    cent /= np.linalg.norm(cent, axis=1, keepdims=True)
    q = rng.standard_normal((nq, dims), dtype=np.float32)
    if kind != "gauss":
        q = (cent[:1] + np.float32(0.02) * q).astype(np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    member = rng.permutation(np.arange(rows) % nlist)  # three rows each, whatever they hold
    order = np.argsort(member, kind="stable")
    dp = (dims + 7) // 8 * 8
    pad = np.zeros((nlist, dp), dtype=np.float32)
    pad[:, :dims] = cent
    lay = {"centroids": pad, "cluster_offsets": np.arange(0, rows + 1, 3).astype(np.uint64),
           "original_indices": order.astype(np.uint64), "init_rows": np.zeros(nlist, dtype=np.uint64)}
    index = NNdex(m, normalized=True)
    index.load_ivf(lay)
    index.set_nprobe(nprobe)
    k = min(3 * nprobe, 2_048)
    idx, _ = index.search(np.vstack([q, q[:1]]), k=k)
    want = probed_rows(lay, q, nprobe, rows)
    for i in range(nq):
        if k == 3 * nprobe:
            assert set(idx[i].tolist()) == set(want[i].tolist()), i
        else:
            assert set(idx[i].tolist()) <= set(want[i].tolist()), i


@pytest.mark.parametrize("rows,dims,nlist,nprobe,k,sizes", [
    (20_000, 40, 64, 8, 10, (1, 3)),         # lists of a few hundred rows, one chunk
    (120_000, 128, 300, 20, 100, (1, 9)),
    (60_000, 96, 40, 3, 256, (1, 13)),       # lists of several chunks, the longest merge
    (5_000, 1_100, 100, 60, 1, (1,)),
])
def test_small_batches_equal_large_ones(rows, dims, nlist, nprobe, k, sizes):
    # a few queries are scanned per (query, list, chunk) without a plan, a large batch by the plan's
    # items: the same rows and scores
    rng = np.random.default_rng(rows + dims)
    c = rng.standard_normal((37, dims), dtype=np.float32)
    w = np.arange(1, 38) ** -1.2
    pick = rng.choice(37, size=rows + 300, p=w / w.sum())  # uneven lists
    x = c[pick] + np.float32(0.4) * rng.standard_normal((rows + 300, dims), dtype=np.float32)
    index = NNdex(x[:rows], approx=True, nlist=nlist, kmeans_iters=3, seed=1, precision="fp32")
    index.set_nprobe(nprobe)
    q = x[rows:]
    bi, bs = index.search(q, k=k)
    streamed = index.last_search_stats()["ivf_rows_streamed"]
    for n in sizes:
        for lo in (0, 111):
            i, s = index.search(np.vstack([q[lo:lo + n], q[:1]]) if n == 1 else q[lo:lo + n], k=k)
            st = index.last_search_stats()
            assert st["path"] == 4 and 0 < st["ivf_rows_union"] <= st["ivf_rows_streamed"] <= st["rows_scanned"]
            np.testing.assert_array_equal(i[:n], bi[lo:lo + n])
            np.testing.assert_array_equal(s[:n].view(np.uint32), bs[lo:lo + n].view(np.uint32))
    assert streamed > 0
