"""A cached plan serves the batches of its bucket that it can run: a bucket's larger k, an index without
the TF32 scans' row norms or without the copy that an imported plan names take the rules' path."""
import ctypes as C

import numpy as np
import pytest

from nndex_b200 import NNdex, _lib

AUTO, FP32, BF16, FP8 = 0, 1, 2, 3


def up(n):
    return 1 << (n - 1).bit_length()


def plan(path, nq, k, precision):
    return f"shape ivf=0 nq={up(nq)} k={up(k)} precision={precision} nprobe=0 plan path={path} stride=0 qb=0 ms=0\n"


def path_of(planned, rows, dims, nq, k, precision=FP32, flags=0, norms=1):
    out = C.c_uint32(0)
    st = _lib.lib().nndex_cuda_autotune_path(("nndex-autotune v2 any\n" + plan(planned, nq, k, precision)).encode(),
                                             rows, dims, flags, precision, norms, nq, k, C.byref(out))
    assert st == 0, _lib.last_error()
    return out.value


@pytest.mark.parametrize("planned,nq,k", [(6, 12, 10), (7, 64, 10), (7, 300, 256)])
def test_tf32_plans_need_the_row_norms(planned, nq, k):
    assert path_of(planned, 200_000, 128, nq, k) == planned
    assert path_of(planned, 200_000, 128, nq, k, norms=0) == 1


@pytest.mark.parametrize("rows,k,path", [
    (1_000_000, 300, 6), (1_000_000, 448, 6), (1_000_000, 449, 1), (1_000_000, 512, 1),  # one bucket
    (1_000, 70, 6), (1_000, 100, 1),                                                      # k' of four rows each
])
def test_candidate_scan_plan_serves_the_k_it_holds(rows, k, path):
    assert path_of(6, rows, 768, 12, k) == path


def test_two_pass_plan_serves_the_batches_of_its_rule():
    assert path_of(7, 50_000, 128, 64, 10) == 7
    assert path_of(7, 50_000, 128, 33, 10) == 1  # too little work
    assert path_of(7, 50_000, 128, 64, 257, precision=FP32) == 1


def test_low_precision_plans_need_their_copy_and_room_for_k():
    bf16, fp8 = _lib.NNDEX_FLAG_BF16, _lib.NNDEX_FLAG_FP8
    assert path_of(2, 200_000, 128, 64, 10, precision=AUTO, flags=bf16) == 2
    assert path_of(2, 200_000, 128, 64, 10, precision=AUTO) != 2
    assert path_of(3, 200_000, 128, 64, 10, precision=AUTO, flags=bf16) == 2
    assert path_of(3, 200_000, 128, 64, 10, precision=AUTO, flags=fp8) == 3
    # the largest k that the heaps beside one FP8 slab hold lies inside a bucket
    held = [path_of(3, 200_000, 128, 64, k, precision=FP8, flags=fp8) == 3 for k in range(129, 257)]
    assert held[0] and not held[-1] and sorted(held, reverse=True) == held


@pytest.mark.parametrize("rows,dims,nq,k,path", [
    (1_200, 128, 1_628, 10, 1), (1_200, 512, 652, 10, 1), (2_500, 32, 5_001, 10, 1),   # few rows for many queries
    (20_000, 512, 25, 256, 1), (100_000, 512, 32, 256, 1), (10_000, 512, 79, 100, 1),  # few queries, much to gather
    (100_000, 512, 32, 10, 7), (100_000, 128, 63, 256, 7), (40_000, 128, 157, 100, 7), (5_000, 512, 626, 10, 7),
])
def test_two_pass_plan_weighs_its_own_costs(rows, dims, nq, k, path):
    assert path_of(7, rows, dims, nq, k) == path


@pytest.mark.gpu
def test_batches_outside_a_cached_plan_are_answered():
    rng = np.random.default_rng(0)
    index = NNdex(rng.normal(size=(20_000, 64)).astype(np.float32))
    q = rng.normal(size=(12, 64)).astype(np.float32)
    index.set_autotune(False)
    want = {k: index.search(q[:8], k=k) for k in (300, 500)}
    index.set_autotune(True)
    index.autotune_import(index.autotune_export().splitlines()[0] + "\n" + plan(6, 12, 300, FP32))
    for k, path, tuned in ((300, 6, 2), (500, 1, 0)):
        got = index.search(q, k=k)
        st = index.last_search_stats()
        assert (st["path"], st["tuned"]) == (path, tuned), st
        np.testing.assert_array_equal(got[0][:8], want[k][0])
        np.testing.assert_array_equal(got[1][:8].view(np.uint32), want[k][1].view(np.uint32))
