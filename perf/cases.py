"""The searches, index builds and serving mixes this library is timed on.

A case is one thing a program does with an index, through the public entry points: the Python class
(`NNdex`, `Server`) on host arrays, or the C ABI on host or device buffers. Sizes follow the
repository's own workloads (50,000 x 128, 1M x 768, 10M x 256, 2M x 384, 5M x 512) and the odd sizes
between them; the data are what those workloads use: i.i.d. normal entries, or Gaussian mixtures with
unit rows (uniform or power-law cluster sizes).

An index lives long and answers many batches, so `prepare` opens it, installs its IVF and sends it a
few batches of the case's shape with other queries (the first batches of a shape choose a plan and
size the buffers). The cases "open_*" and "build_ivf" time the opposite: a new index and its first
answer.
"""
import ctypes as C
import math

import numpy as np
import torch

from nndex_b200 import NNdex, Server, _lib

NORMALIZED, APPROX, BF16, FP8 = (_lib.NNDEX_FLAG_NORMALIZED, _lib.NNDEX_FLAG_APPROX, _lib.NNDEX_FLAG_BF16,
                                 _lib.NNDEX_FLAG_FP8)
PRECISION = {"auto": _lib.NNDEX_PRECISION_AUTO, "fp32": _lib.NNDEX_PRECISION_FP32,
             "bf16": _lib.NNDEX_PRECISION_BF16, "fp8": _lib.NNDEX_PRECISION_FP8}
COPIES = {"auto": BF16, "fp32": 0, "bf16": BF16, "fp8": FP8}


def listed():
    return [
        # One user query against a small corpus held by a Python program: the latency of a call.
        dict(name="one_50k", kind="search", api="python", rows=50_000, dims=128, nq=1, k=10, precision="fp32",
             normalized=False, centers=0),
        # The same corpus asked by a small batch.
        dict(name="batch64_50k", kind="search", api="python", rows=50_000, dims=128, nq=64, k=10, precision="fp32",
             normalized=False, centers=0),
        # One embedding against a large corpus, asked from host memory: one pass over the base.
        dict(name="one_1m", kind="search", api="host", rows=1_000_000, dims=768, nq=1, k=100, precision="fp32",
             normalized=True, centers=1024),
        # Sixteen embeddings that a model left on the GPU, answered there.
        dict(name="batch16_1m", kind="search", api="device", rows=1_000_000, dims=768, nq=16, k=100,
             precision="fp32", normalized=True, centers=1024),
        # A batch of no particular size over a corpus of no particular shape, raw rows.
        dict(name="odd_batch", kind="search", api="host", rows=300_007, dims=100, nq=37, k=33, precision="fp32",
             normalized=False, centers=257),
        # The large offline batch (near-duplicate search, graph building), BF16 scoring copy.
        dict(name="batch4096_bf16", kind="search", api="device", rows=10_000_000, dims=256, nq=4096, k=10,
             precision="bf16", normalized=True, centers=4096),
        # A wide re-ranking stage: many results per query from the FP8 scoring copy.
        dict(name="batch1000_fp8", kind="search", api="host", rows=2_000_003, dims=512, nq=1000, k=100,
             precision="fp8", normalized=True, centers=2048),
        # Approximate search over uneven lists, a large batch.
        dict(name="ivf_1024", kind="ivf", api="device", rows=2_000_000, dims=384, nq=1024, k=10, precision="auto",
             nlist=1414, nprobe=32, centers=8192, zipf=1.1),
        # Approximate search for one user query.
        dict(name="ivf_one", kind="ivf", api="python", rows=400_000, dims=128, nq=1, k=10, precision="fp32",
             nlist=512, nprobe=16, centers=2048, zipf=0.0),
        # Opening an index over rows already on the GPU (a model's embeddings), to its first answer.
        dict(name="open_bf16", kind="open", rows=1_000_000, dims=256, nq=16, k=10, precision="auto",
             normalized=False, centers=1024),
        # Opening an approximate index over a matrix in host memory, and exporting its layout.
        dict(name="build_ivf", kind="build", rows=200_000, dims=256, normalized=False, centers=512),
        # A second of mixed traffic at once: ragged requests, k of 1, 10 and 100, exact and approximate.
        dict(name="serve_mixed", kind="serve", rows=1_000_000, dims=512, requests=24, nlist=512, nprobe=32,
             centers=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "small", "exact", "exact", "low", "low", "ivf", "ivf", "open", "build", "serve"])
    if kind in ("small", "exact"):
        rows = _log(rng, 1_000, 60_000) if kind == "small" else _log(rng, 60_000, 1_000_000)
        dims = _log(rng, 16, 768)
        nq = 1 if rng.random() < 0.3 else _log(rng, 1, 256)
        return dict(kind="search", api=rng.choice(["python", "device"] if kind == "small" else ["host", "device"]),
                    rows=rows, dims=dims, nq=nq, k=_log(rng, 1, 100), precision="fp32",
                    normalized=rng.random() < 0.5, centers=rng.choice([0, 1024]))
    if kind == "low":
        dims = _log(rng, 64, 512)
        rows = min(_log(rng, 100_000, 10_000_000), 2_560_000_000 // dims)
        return dict(kind="search", api=rng.choice(["host", "device"]), rows=rows, dims=dims,
                    nq=_log(rng, 64, 4096), k=rng.choice([1, 10, 100]), precision=rng.choice(["bf16", "fp8", "auto"]),
                    normalized=True, centers=4096)
    if kind == "ivf":
        rows = _log(rng, 20_000, 2_000_000)
        nlist = min(1414, math.isqrt(rows))
        return dict(kind="ivf", api=rng.choice(["python", "device"]) if rows <= 400_000 else "device", rows=rows,
                    dims=_log(rng, 32, 384), nq=1 if rng.random() < 0.3 else _log(rng, 1, 1024),
                    k=rng.choice([1, 10, 100]), precision=rng.choice(["fp32", "auto"]), nlist=nlist,
                    nprobe=rng.choice([8, 32, 64]), centers=2048, zipf=rng.choice([0.0, 1.1]))
    if kind == "open":
        return dict(kind="open", rows=_log(rng, 10_000, 1_000_000), dims=_log(rng, 32, 512), nq=_log(rng, 1, 256),
                    k=10, precision=rng.choice(["fp32", "auto", "fp8"]), normalized=rng.random() < 0.5, centers=1024)
    if kind == "build":
        return dict(kind="build", rows=_log(rng, 5_000, 200_000), dims=_log(rng, 32, 256),
                    normalized=rng.random() < 0.5, centers=512)
    rows = _log(rng, 50_000, 1_000_000)
    return dict(kind="serve", rows=rows, dims=_log(rng, 64, 512), requests=rng.randint(4, 24),
                nlist=min(512, math.isqrt(rows)), nprobe=rng.choice([8, 32]), centers=1024)


# ---- data -----------------------------------------------------------------------------------------


def _points(n, dims, centers, seed, center_seed, unit, zipf=0.0):
    """n x dims float32 on the GPU: N(0, 1), or centre + 0.3 N(0, 1) with uniform or power-law sizes."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((n, dims), generator=g, device="cuda")
    if centers:
        c = torch.randn((centers, dims), generator=torch.Generator(device="cuda").manual_seed(center_seed),
                        device="cuda")
        u = torch.rand(n, generator=g, device="cuda")
        if zipf:
            w = torch.arange(1, centers + 1, dtype=torch.float64, device="cuda") ** -zipf
            cdf = (w.cumsum(0) / w.sum()).float()
            pick = torch.searchsorted(cdf, u).clamp_(max=centers - 1)
        else:
            pick = (u * centers).long().clamp_(max=centers - 1)
        for a in range(0, n, 1 << 20):
            x[a:a + (1 << 20)].mul_(0.3).add_(c[pick[a:a + (1 << 20)]])
    if unit:
        for a in range(0, n, 1 << 20):
            x[a:a + (1 << 20)] /= x[a:a + (1 << 20)].norm(dim=1, keepdim=True)
    return x


def _unit_rows(case):
    return bool(case.get("normalized", True))


def _base(case, seed):
    return _points(case["rows"], case["dims"], case["centers"], 4 * seed + 1, 4 * seed + 3, _unit_rows(case),
                   case.get("zipf", 0.0))


def _queries(case, seed, n, which=2):
    """Queries of the base's own distribution (which = 2: the timed ones; 4: other ones, to warm up with)."""
    return _points(n, case["dims"], case["centers"], 4 * seed + which, 4 * seed + 3, _unit_rows(case),
                   case.get("zipf", 0.0))


def _layout(base, nlist):
    """A saved IVF layout: `nlist` rows spread over the matrix, one Lloyd step, the rows by list."""
    rows, dims = base.shape
    init = torch.arange(nlist, device=base.device) * (rows // nlist)
    cent = base[init]

    def assign(c):
        out = torch.empty(rows, dtype=torch.long, device=base.device)
        for a in range(0, rows, 1 << 18):
            out[a:a + (1 << 18)] = (base[a:a + (1 << 18)] @ c.t()).argmax(1)
        return out

    first, total = assign(cent), torch.zeros_like(cent)
    for a in range(0, rows, 1 << 18):
        part = first[a:a + (1 << 18)]
        total += torch.nn.functional.one_hot(part, nlist).to(base.dtype).t() @ base[a:a + (1 << 18)]
    cent = total / total.norm(dim=1, keepdim=True).clamp_min(1e-20)
    member = assign(cent)
    order = torch.sort(member, stable=True).indices
    off = torch.zeros(nlist + 1, dtype=torch.long, device=base.device)
    off[1:] = torch.bincount(member, minlength=nlist).cumsum(0)
    padded = torch.zeros((nlist, (dims + 7) // 8 * 8), device=base.device)
    padded[:, :dims] = cent
    arrays = {"centroids": padded.cpu().numpy(), "cluster_offsets": off.cpu().numpy().astype(np.uint64),
              "original_indices": order.cpu().numpy().astype(np.uint64),
              "init_rows": init.cpu().numpy().astype(np.uint64)}
    return arrays, member, cent


# ---- the program's side -----------------------------------------------------------------------------


def _check(status):
    if status != 0:
        raise RuntimeError(_lib.last_error())


class Opened:
    """An index opened through the C ABI over a matrix on the GPU."""

    def __init__(self, base, flags, precision):
        self.rows, self.dims = base.shape
        opts = _lib.Opts()
        opts.device = -1
        opts.precision = PRECISION[precision]
        self.handle = C.c_void_p()
        _check(_lib.lib().nndex_cuda_create_from_device(base.data_ptr(), base.numel(), self.rows, self.dims, flags,
                                                        C.byref(opts), C.byref(self.handle)))

    def load_ivf(self, lay):
        ptr = [lay[n].ctypes.data for n in ("centroids", "cluster_offsets", "original_indices", "init_rows")]
        _check(_lib.lib().nndex_cuda_ivf_restore(self.handle, len(lay["init_rows"]), *ptr))

    def set_nprobe(self, n):
        _check(_lib.lib().nndex_cuda_set_nprobe(self.handle, n))

    def search_host(self, q, k):
        nq, kk = q.shape[0], min(k, self.rows)
        idx = np.empty((nq, kk), dtype=np.int64)
        sim = np.empty((nq, kk), dtype=np.float32)
        cnt = np.empty(nq, dtype=np.int64)
        _check(_lib.lib().nndex_cuda_search_batch(self.handle, q.ctypes.data, q.size, nq, k, idx.ctypes.data,
                                                  sim.ctypes.data, cnt.ctypes.data))
        return idx, sim, cnt

    def search_device(self, q, k, idx, sim, cnt):
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _check(_lib.lib().nndex_cuda_search_batch_device(self.handle, q.data_ptr(), q.shape[0], q.shape[1], k,
                                                         idx.data_ptr(), sim.data_ptr(), cnt.data_ptr(), stream, 0))
        return idx, sim, cnt

    def __del__(self):
        if self.handle:
            _lib.lib().nndex_cuda_destroy(self.handle)
            self.handle = None


def _ask(state, q):
    case, index = state["case"], state["index"]
    if case["api"] == "python":
        idx, sim = index.search(q[0] if len(q) == 1 else q, k=case["k"])
        return idx.view(np.int64), sim
    if case["api"] == "host":
        return index.search_host(q, case["k"])
    return index.search_device(q, case["k"], *state["out"])


def _requests(case):
    r = np.random.default_rng(case["requests"])
    sizes = r.integers(1, 257, size=case["requests"])
    return [(int(n), int(r.choice([1, 10, 100])), bool(r.integers(0, 2))) for n in sizes]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "build":
        return {"case": case, "matrix": _base(case, seed).cpu().numpy()}
    base = _base(case, seed)
    if kind == "open":
        nq = case["nq"]
        return {"case": case, "base": base, "q": _queries(case, seed, nq),
                "out": (torch.empty((nq, case["k"]), dtype=torch.int64, device="cuda"),
                        torch.empty((nq, case["k"]), device="cuda"),
                        torch.empty(nq, dtype=torch.int32, device="cuda"))}
    flags = (NORMALIZED if _unit_rows(case) else 0)
    if kind == "serve":
        index = Opened(base, flags | BF16, "auto")
        index.load_ivf(_layout(base, case["nlist"])[0])
        del base
        requests, at = _requests(case), 0
        q = _queries(case, seed, sum(n for n, _, _ in requests)).cpu().numpy()
        work = []
        for n, k, approx in requests:
            work.append((q[at:at + n], k, approx))
            at += n
        state = {"case": case, "index": index, "server": Server(index, slots=3), "work": work}
        run(state)
        return state
    state = {"case": case}
    if case["api"] == "python":
        state["index"] = NNdex(base.cpu().numpy(), normalized=_unit_rows(case), approx=False,
                               precision=case["precision"])
    else:
        state["index"] = Opened(base, flags | COPIES[case["precision"]], case["precision"])
    if kind == "ivf":
        state["index"].load_ivf(_layout(base, case["nlist"])[0])
        state["index"].set_nprobe(case["nprobe"])
    del base
    nq = case["nq"]
    q, other = _queries(case, seed, nq), _queries(case, seed, nq, 4)
    if case["api"] == "device":
        kk = min(case["k"], case["rows"])
        state["out"] = (torch.empty((nq, kk), dtype=torch.int64, device="cuda"),
                        torch.empty((nq, kk), device="cuda"), torch.empty(nq, dtype=torch.int32, device="cuda"))
    else:
        q, other = q.cpu().numpy(), other.cpu().numpy()
    state["q"] = q
    for _ in range(3):
        _ask(state, other)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "open":
        index = Opened(state["base"], (NORMALIZED if _unit_rows(case) else 0) | COPIES[case["precision"]],
                       case["precision"])
        index.search_device(state["q"], case["k"], *state["out"])
        torch.cuda.current_stream().synchronize()  # the index goes away with this call
        return state["out"]
    if case["kind"] == "build":
        lay = NNdex(state["matrix"], normalized=_unit_rows(case), approx=True).ivf_layout()
        return {k: v if v.dtype == np.float32 else v.view(np.int64) for k, v in lay.items()}
    if case["kind"] == "serve":
        server = state["server"]
        tickets = [server.submit(q, k=k, approx=a, nprobe=case["nprobe"] if a else 0) for q, k, a in state["work"]]
        got = [server.result(t) for t in tickets]
        return [(idx.view(np.int64), sim) for idx, sim in got]
    return _ask(state, state["q"])


# ---- what a pass cannot do without ------------------------------------------------------------------


def work(case):
    rows, dims, kind = case["rows"], case["dims"], case["kind"]
    if kind == "build":
        nlist = min(max(math.isqrt(rows), 16), 512)
        # read the matrix, write the reordered rows, the layout; 12 assignments and the seeding
        return {"bytes": 8 * rows * dims + 12 * rows, "flops": 2 * rows * dims * nlist * 13}
    if kind == "open":
        extra = {"fp32": 0, "auto": 2, "fp8": 1}[case["precision"]]
        return {"bytes": rows * dims * (8 + extra), "flops": 2 * rows * dims * (case["nq"] + 1)}
    width = {"fp32": 4, "bf16": 2, "fp8": 1, "auto": 2}
    if kind == "serve":
        q = 128 * case["requests"]
        share = case["nprobe"] / case["nlist"]
        # half of the requests score every row, half the rows of their lists; one pass over the copy
        return {"bytes": 2 * rows * dims + 4 * q * dims, "flops": rows * dims * q * (1 + share)}
    nq, k, w = case["nq"], case["k"], width[case["precision"]]
    io = nq * (4 * dims + 16 * k)
    if kind == "ivf":
        per_query = rows * case["nprobe"] / case["nlist"]
        union = min(rows, per_query * nq)
        return {"bytes": union * dims * w + 4 * case["nlist"] * dims + io,
                "flops": 2 * dims * nq * (per_query + case["nlist"])}
    return {"bytes": rows * dims * w + io, "flops": 2 * rows * dims * nq}


# ---- the same in 64 bits ----------------------------------------------------------------------------


def _unit64(x):
    x = x.double()
    return x / x.norm(dim=1, keepdim=True)


def _top_scores(base, q, k, unit, member=None, probed=None):
    """The k largest FP64 scores of each query (unit: rows and queries are taken as they are)."""
    q = q.double() if unit else _unit64(q)
    best = None
    step = max(1 << 10, min(1 << 20, (1 << 28) // max(1, len(q))))
    for a in range(0, len(base), step):
        part = base[a:a + step].double() if unit else _unit64(base[a:a + step])
        s = q @ part.t()
        if member is not None:
            s.masked_fill_(~probed[:, member[a:a + step]], -math.inf)
        s = s.topk(min(k, s.shape[1]), dim=1).values
        best = s if best is None else torch.cat([best, s], 1).topk(min(k, best.shape[1] + s.shape[1]), dim=1).values
    return best


def exact(case, seed):
    kind, unit = case["kind"], _unit_rows(case)
    if kind == "build":
        return None  # k-means: a chain of decisions, whose outputs no plain restatement reproduces
    base = _base(case, seed)
    if kind == "serve":
        _, member, cent = _layout(base, case["nlist"])
        requests, out, at = _requests(case), [], 0
        q = _queries(case, seed, sum(n for n, _, _ in requests))
        for n, k, approx in requests:
            part = q[at:at + n]
            at += n
            probed = _probed(part, cent, case["nprobe"], unit) if approx else None
            out.append((None, _top_scores(base, part, k, unit, member if approx else None, probed).cpu().numpy()))
        return out
    q = _queries(case, seed, case["nq"])
    if kind == "ivf":
        _, member, cent = _layout(base, case["nlist"])
        probed = _probed(q, cent, case["nprobe"], unit)
        lists = torch.bincount(member, minlength=case["nlist"])
        if float((probed.double() @ lists.double()).min()) < case["k"]:
            return None  # fewer probed rows than results: padded outputs
        sim = _top_scores(base, q, case["k"], unit, member, probed)
    else:
        sim = _top_scores(base, q, min(case["k"], case["rows"]), unit)
    if kind == "open" or case["api"] == "device":
        return None, sim, None
    sim = sim.cpu().numpy()
    if case["api"] == "host":
        return None, sim, None
    return None, sim[0] if case["nq"] == 1 else sim


def _probed(q, cent, nprobe, unit):
    q = q.double() if unit else _unit64(q)
    near = (q @ cent.double().t()).topk(min(nprobe, len(cent)), dim=1).indices
    return torch.zeros((len(q), len(cent)), dtype=torch.bool, device=q.device).scatter_(1, near, True)
