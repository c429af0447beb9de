"""The two-pass TF32 scan without memory for its collections (needs a B200): the batch and the next ones take
the FP32 scan, what the attempt had grown is given back, no captured graph of another index is dropped
again, and the scan is tried anew later."""
import numpy as np
import pytest
import torch

from nndex_b200 import NNdex, _lib

pytestmark = pytest.mark.gpu


# the scan grows up to 13 buffers: the first, one in the middle, the collections, the rerank's slots
@pytest.mark.parametrize("skip", [0, 5, 9, 11])
def test_batch_without_memory_takes_the_fp32_scan(skip):
    rng = np.random.default_rng(skip)
    m = rng.standard_normal((20_000, 64), dtype=np.float32)
    q = rng.standard_normal((4_096, 64), dtype=np.float32)
    index, other = NNdex(m, autotune=False), NNdex(m, autotune=False)
    want = other.search(q, k=10)
    assert other.last_search_stats()["path"] == 7
    index.search(q, k=300)  # the FP32 scan: sizes the buffers that it shares
    assert index.last_search_stats()["path"] == 1
    one = q[0]
    for _ in range(4):
        other.search(one, k=10)
    assert other.last_search_stats()["graph"] == 2
    free = torch.cuda.mem_get_info()[0]
    L = _lib.lib()
    try:
        L.nndex_cuda_inject_alloc_failures_after(skip, 1000)
        paths = []
        for _ in range(3):
            got = index.search(q, k=10)
            paths.append(index.last_search_stats()["path"])
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
    finally:
        L.nndex_cuda_inject_alloc_failures(0)
    assert paths == [1, 1, 1]
    assert torch.cuda.mem_get_info()[0] >= free - (8 << 20)  # the collections alone are 128 MB
    for _ in range(4):  # the first of them after the attempt captures again, and then nothing drops it
        other.search(one, k=10)
        index.search(q, k=10)
    assert other.last_search_stats()["graph"] == 2
    for _ in range(40):
        got = index.search(q, k=10)
    assert index.last_search_stats()["path"] == 7
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
