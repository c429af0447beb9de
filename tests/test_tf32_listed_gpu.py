"""Listed queries of the TF32 scans' host-buffer batches (needs a B200): their re-run follows the batch,
call after call of one shape (direct, captured, replayed), small batches that the kernels write into
host memory and larger ones that are copied, and never touches the queries that were not listed.
"""
import numpy as np
import pytest

from nndex_b200 import NNdex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,k,dims,path", [(12, 10, 64, 6), (24, 10, 256, 7), (300, 40, 128, 7)])
def test_listed_queries_are_rerun_on_every_call(nq, k, dims, path):
    # a quarter of the rows are copies of one row: a query near it collects more than a batch holds
    # (path 7), or finds more equals than its lists (path 6); the others are certified at once
    rng = np.random.default_rng(nq)
    rows = 60_000
    m = rng.normal(size=(rows, dims)).astype(np.float32)
    m[::4] = m[0]
    index = NNdex(m, autotune=False)
    clean = rng.normal(size=(nq, dims)).astype(np.float32)
    near = clean.copy()
    near[::5] = m[0] + 1e-3 * rng.normal(size=(len(near[::5]), dims)).astype(np.float32)
    header = index.autotune_export().splitlines()[0]
    up = lambda n: 1 << (n - 1).bit_length()
    plan = lambda p: f"{header}\nshape ivf=0 nq={up(nq)} k={up(k)} precision=1 nprobe=0 plan path={p} stride=0 qb=0 ms=0\n"
    index.autotune_import(plan(1))
    index.set_autotune(True)
    want = [index.search(q, k=k) for q in (clean, near)]
    assert index.last_search_stats()["path"] == 1
    index.autotune_import(plan(path))
    listed = {0: set(), 1: set()}
    for which in (0, 1, 1, 0, 1, 0, 1):
        got = index.search((clean, near)[which], k=k)
        st = index.last_search_stats()
        assert st["path"] == path, st
        listed[which].add(st["fp32_fallback_queries"])
        assert np.array_equal(got[0], want[which][0])
        assert np.array_equal(got[1].view(np.uint32), want[which][1].view(np.uint32))
    # the same queries every time; a few of the random ones may lie near the copies too
    assert len(listed[0]) == len(listed[1]) == 1
    assert listed[1].pop() >= max(listed[0].pop(), len(near[::5]))
