"""Queries that a tensor-core scan cannot finish (their collections overflow twice, or on the list scan and the
TF32 scans once) are re-run in FP32, on host batches that the kernels write in place, host batches that
are copied, and device buffers; a device wait that runs out in a re-run fails the call (needs a B200)."""
import ctypes as C

import numpy as np
import pytest
import torch

from nndex_b200 import NNdex, NNdexError, _lib

pytestmark = pytest.mark.gpu

ROWS, COPIES, DIMS, K = 60_000, 9_000, 64, 10
# path, precision, IVF, queries
CASES = [(2, "bf16", False, 64), (2, "bf16", False, 300), (3, "fp8", False, 64), (5, "auto", True, 64),
         (5, "auto", True, 300), (6, "fp32", False, 12), (7, "fp32", False, 72), (7, "fp32", False, 300)]


def data(nq):
    # more copies of one row than a collection holds, and a fifth of the queries beside them
    rng = np.random.default_rng(nq)
    m = rng.standard_normal((ROWS, DIMS), dtype=np.float32)
    m[20_000:20_000 + COPIES] = m[20_000]
    q = rng.standard_normal((nq, DIMS), dtype=np.float32)
    q[::5] = m[20_000] + np.float32(1e-3) * rng.standard_normal((len(q[::5]), DIMS), dtype=np.float32)
    return m, q


def opened(m, precision, ivf):
    return NNdex(m, precision=precision, autotune=False, **(dict(approx=True, nlist=16, nprobe=8, seed=1) if ivf else {}))


def on_device(index, q, k=K, synchronize=1):
    d = torch.as_tensor(q).cuda()
    out = (torch.zeros((len(q), k), dtype=torch.int64, device="cuda"), torch.zeros((len(q), k), device="cuda"),
           torch.zeros(len(q), dtype=torch.int32, device="cuda"))
    st = _lib.lib().nndex_cuda_search_batch_device(index.handle, d.data_ptr(), len(q), q.shape[1], k,
                                                   *(o.data_ptr() for o in out),
                                                   C.c_void_p(torch.cuda.current_stream().cuda_stream), synchronize)
    if st:
        raise NNdexError(st, _lib.last_error())
    torch.cuda.synchronize()
    return out[0].cpu().numpy().astype(np.uint64), out[1].cpu().numpy()


def in_fp32(index, q, k=K):
    """Eight queries at a time: the FP32 scan, or the FP32 list scan."""
    index.set_precision("fp32")
    parts = [index.search(np.vstack([q[a:a + 7], q[:1]]), k=k) for a in range(0, len(q), 7)]
    assert index.last_search_stats()["path"] in (1, 4)
    return np.vstack([p[0][:-1] for p in parts]), np.vstack([p[1][:-1] for p in parts])


@pytest.mark.parametrize("buffers", ["host", "device"])
@pytest.mark.parametrize("path,precision,ivf,nq", CASES)
def test_rerun_queries_equal_the_fp32_scan(path, precision, ivf, nq, buffers):
    m, q = data(nq)
    index = opened(m, precision, ivf)
    for _ in range(3):  # host batches: direct, captured, replayed
        got = index.search(q, k=K) if buffers == "host" else on_device(index, q)
        st = index.last_search_stats()
        assert st["path"] == path and st["fp32_fallback_queries"] >= len(q[::5]), st
    want = in_fp32(index, q)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


@pytest.mark.parametrize("buffers", ["host", "device"])
@pytest.mark.parametrize("path,precision,ivf,nq", CASES)
def test_wait_that_runs_out_in_a_rerun_fails_the_call(path, precision, ivf, nq, buffers):
    if path >= 6 and buffers == "device":
        pytest.skip("re-run behind the batch, before the call's own status check")
    m, q = data(nq)
    index = opened(m, precision, ivf)
    search = (lambda: index.search(q, k=K)) if buffers == "host" else (lambda: on_device(index, q))
    want = search()
    try:
        _lib.lib().nndex_cuda_inject_rerun_timeouts(1)
        with pytest.raises((NNdexError, RuntimeError), match="timed out"):
            search()
    finally:
        _lib.lib().nndex_cuda_inject_rerun_timeouts(0)
    got = search()
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
