// index.cu — the CUDA backend object (CudaIndex) and the C ABI declared in include/nndex_cuda.h.
//
// Mirrors nndex's backend contract: GpuIndex::new / search / search_batch / adapter info
// (src/gpu.rs:138-309, 321-430, 974-1010) behind NNdex::new / search / search_batch
// (src/lib.rs:185-402), with the reference's validation order and error variants
// (src/lib.rs:107-145, 433-450). The device holds the whole normalised base; queries are
// normalised on the device (K1) and scored by the fused scan (K2) + merge.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <sys/mman.h>

#include <algorithm>
#include <chrono>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "common.cuh"
#include "index.h"
#include "internal.h"

namespace nndex {

static std::atomic<uint64_t> g_launches{0};
static std::atomic<uint64_t> g_alloc_epoch{0};
static std::atomic<uint32_t> g_fail_skip{0}, g_fail_allocs{0};  // host-side fault injection: allocations to fail
bool take_injected_alloc_failure() {
    uint32_t n = g_fail_skip.load(std::memory_order_relaxed);
    while (n > 0 && !g_fail_skip.compare_exchange_weak(n, n - 1, std::memory_order_relaxed)) {
    }
    if (n > 0) return false;
    n = g_fail_allocs.load(std::memory_order_relaxed);
    while (n > 0 && !g_fail_allocs.compare_exchange_weak(n, n - 1, std::memory_order_relaxed)) {
    }
    return n > 0;
}
void inject_alloc_failures(uint32_t skip, uint32_t n) {
    g_fail_skip.store(n ? skip : 0, std::memory_order_relaxed);
    g_fail_allocs.store(n, std::memory_order_relaxed);
}
static std::atomic<uint32_t> g_rerun_timeouts{0};
bool take_injected_rerun_timeout() {
    uint32_t n = g_rerun_timeouts.load(std::memory_order_relaxed);
    while (n > 0 && !g_rerun_timeouts.compare_exchange_weak(n, n - 1, std::memory_order_relaxed)) {
    }
    return n > 0;
}
void inject_rerun_timeouts(uint32_t n) { g_rerun_timeouts.store(n, std::memory_order_relaxed); }
static thread_local cudaStream_t t_scratch_stream = nullptr;
void set_scratch_stream(cudaStream_t s) { t_scratch_stream = s; }
cudaStream_t scratch_stream() { return t_scratch_stream; }
static void release_raw(void** p) {
    if (*p && t_scratch_stream) cudaFreeAsync(*p, t_scratch_stream);
    else if (*p) cudaFree(*p);
    *p = nullptr;
}
cudaError_t regrow_raw(void** p, size_t bytes) {
    if (bytes == 0) bytes = 1;
    cudaStream_t s = t_scratch_stream;
    if (!s) {
        if (*p) cudaFree(*p);
        *p = nullptr;
        return cudaMalloc(p, bytes);
    }
    // never inside a stream capture: the allocation would become a node of a graph that may be
    // discarded (the caller then runs the batch without a graph)
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
        return cudaErrorStreamCaptureUnsupported;
    if (*p) cudaFreeAsync(*p, s);
    *p = nullptr;
    return cudaMallocAsync(p, bytes, s);
}
uint64_t alloc_epoch() { return g_alloc_epoch.load(std::memory_order_acquire); }
void bump_alloc_epoch() { g_alloc_epoch.fetch_add(1, std::memory_order_acq_rel); }
bool sync_check_enabled() {
    static const bool on = [] {
        const char* v = getenv("NNDEX_SYNC_CHECK");
        return v && v[0] == '1';
    }();
    return on;
}
static thread_local char t_launch_note[256];
void set_launch_note(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(t_launch_note, sizeof(t_launch_note), fmt, ap);
    va_end(ap);
}
void count_launch_at(const char* file, int line, uint32_t n) {
    g_launches.fetch_add(n, std::memory_order_relaxed);
    if (!sync_check_enabled()) return;
    static std::atomic<bool> reported{false};
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess && !reported.exchange(true))
        std::fprintf(stderr, "nndex: %s (%d) after the launch at %s:%d [%s]\n", cudaGetErrorString(e),
                     static_cast<int>(e), file, line, t_launch_note);
    t_launch_note[0] = 0;
}
uint64_t kernel_launches_total() { return g_launches.load(std::memory_order_relaxed); }

static thread_local std::string t_error;

int set_error(int code, const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    t_error = buf;
    return code;
}
void clear_error() { t_error.clear(); }
const char* last_error() { return t_error.c_str(); }

int cuda_error(cudaError_t e, const char* what) {
    if (e == cudaErrorMemoryAllocation)
        return set_error(NNDEX_ERR_OUT_OF_MEMORY, "cuda execution error: %s: out of device memory", what);
    return set_error(NNDEX_ERR_CUDA, "cuda execution error: %s: %s", what, cudaGetErrorString(e));
}

// NNdexError Display strings (src/lib.rs:109-138).
int err_shape(uint64_t rows, uint64_t dims, uint64_t values) {
    return set_error(NNDEX_ERR_SHAPE_MISMATCH, "matrix shape mismatch: rows=%llu, dims=%llu, values=%llu",
                     (unsigned long long)rows, (unsigned long long)dims, (unsigned long long)values);
}
int err_query_dims(uint64_t expected, uint64_t found) {
    return set_error(NNDEX_ERR_QUERY_DIMS, "query dimensionality mismatch: expected %llu, found %llu",
                     (unsigned long long)expected, (unsigned long long)found);
}
int err_topk() { return set_error(NNDEX_ERR_INVALID_TOPK, "top-k must be greater than zero"); }
int err_code(int code) {
    switch (code) {
        case NNDEX_ERR_NON_FINITE: return set_error(code, "all input values must be finite");
        case NNDEX_ERR_ZERO_NORM: return set_error(code, "encountered a zero-norm vector");
        default: return set_error(code, "cuda execution error: device status %d", code);
    }
}

// src/lib.rs:433-442 validate_matrix_shape (saturating multiply).
bool shape_ok(uint64_t n_values, uint64_t rows, uint64_t dims) {
    if (rows == 0 || dims == 0) return false;
    unsigned __int128 p = static_cast<unsigned __int128>(rows) * dims;
    const uint64_t sat = p > UINT64_MAX ? UINT64_MAX : static_cast<uint64_t>(p);
    return sat == n_values;
}

static thread_local int t_encode_result = 0;  // the last encode's CUresult on this thread

static PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

bool encode_tmap_2d(CUtensorMap* map, CUtensorMapDataType dtype, uint32_t elem_bytes, const void* base,
                    uint64_t inner, uint64_t outer, uint64_t row_stride_bytes, uint32_t box_inner,
                    uint32_t box_outer, CUtensorMapSwizzle swizzle) {
    auto fn = get_encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_stride_bytes};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t es[2] = {1, 1};
    (void)elem_bytes;
    CUresult r = fn(map, dtype, 2, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    t_encode_result = static_cast<int>(r);
    return r == CUDA_SUCCESS;
}
int last_encode_result() { return t_encode_result; }

// ---- device buffers ------------------------------------------------------------------------

template <class T>
static int grow_device(T*& p, size_t& cap, size_t n, const char* what) {
    if (n <= cap && p) return NNDEX_OK;
    bump_alloc_epoch();
    cap = 0;
    void* raw = p;
    cudaError_t e = take_injected_alloc_failure() ? cudaErrorMemoryAllocation
                                                  : regrow_raw(&raw, std::max<size_t>(n, 1) * sizeof(T));
    if (e == cudaErrorMemoryAllocation && raw) cudaFree(raw);  // an injected failure frees it too
    if (e != cudaSuccess) {
        p = nullptr;
        return cuda_error(e, what);
    }
    p = static_cast<T*>(raw);
    cap = n;
    return NNDEX_OK;
}
// Pinned buffers grow geometrically from 4,096 elements: releasing one (cudaFreeHost) waits for
// the device, which in a serving slot means waiting for the other slots' batches too, so they are
// replaced as rarely as possible.
template <class T>
static int grow_host(T*& p, size_t& cap, size_t n, const char* what) {
    if (n <= cap && p) return NNDEX_OK;
    bump_alloc_epoch();
    if (p) cudaFreeHost(p);
    p = nullptr;
    const size_t want = std::max<size_t>({n, cap * 2, 4096});
    cap = 0;
    cudaError_t e = take_injected_alloc_failure()
                        ? cudaErrorMemoryAllocation
                        : cudaMallocHost(reinterpret_cast<void**>(&p), want * sizeof(T));
    if (e != cudaSuccess) {
        p = nullptr;
        return cuda_error(e, what);
    }
    cap = want;
    return NNDEX_OK;
}

void CudaIndex::scan_event_begin(cudaStream_t s, cudaEvent_t& a) {
    a = nullptr;
    if (!scan_timing) return;
    if (scan_events_used == scan_events.size()) {
        cudaEvent_t x, y;
        if (cudaEventCreate(&x) != cudaSuccess) return;
        if (cudaEventCreate(&y) != cudaSuccess) {
            cudaEventDestroy(x);
            return;
        }
        scan_events.emplace_back(x, y);
    }
    a = scan_events[scan_events_used].first;
    cudaEventRecord(a, s);
}

void CudaIndex::scan_event_end(cudaStream_t s, cudaEvent_t a) {
    if (!a) return;
    cudaEventRecord(scan_events[scan_events_used].second, s);
    ++scan_events_used;
}

void CudaIndex::drop_graphs() {
    for (auto& g : graphs) cudaGraphExecDestroy(g.exec);
    graphs.clear();
}

// The host's words and the small batches' queries and results (kHostBytes, pinned). Memory of our own,
// registered, takes a third of the time that a pinned allocation does (0.3 to 0.5 ms; the driver maps 2 MB for
// the first one of a process: 0.9 to 2.9). With the words alone in it the first search of an index paid that
// for its queries: 3 ms against 0.3 now (50k × 128, one query). It is kept out of forked children, as the
// driver's own pinned memory is: copy-on-write would leave the parent another page than the one that the GPU
// writes.
cudaError_t CudaIndex::alloc_words() {
    void* page = mmap(nullptr, kHostBytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (page != MAP_FAILED) {
        void* seen = nullptr;  // the kernels are given the host's address
        if (madvise(page, kHostBytes, MADV_DONTFORK) == 0 &&
            cudaHostRegister(page, kHostBytes, cudaHostRegisterMapped) == cudaSuccess) {
            if (cudaHostGetDevicePointer(&seen, page, 0) == cudaSuccess && seen == page)
                words_page = page;
            else
                cudaHostUnregister(page);
        }
        if (!words_page) munmap(page, kHostBytes);
    }
    if (words_page) {
        h_flags = static_cast<uint64_t*>(words_page);
    } else {
        cudaGetLastError();
        const cudaError_t e = cudaMallocHost(&h_flags, kHostBytes);
        if (e != cudaSuccess) return e;
    }
    uint8_t* const at = reinterpret_cast<uint8_t*>(h_flags);
    h_fbn = reinterpret_cast<uint32_t*>(at + kFbnAt);
    ivf_scratch.h_probed = reinterpret_cast<unsigned long long*>(at + kProbedAt);
    h_q = reinterpret_cast<float*>(at + kHostWordBytes);
    cap_hq = kMappedIoBytes / sizeof(*h_q);
    h_res = at + kHostWordBytes + kMappedIoBytes;
    cap_hres = kMappedIoBytes;
    return cudaSuccess;
}

void CudaIndex::free_words() {
    if (words_page) {
        cudaHostUnregister(words_page);
        munmap(words_page, kHostBytes);
    } else {
        cudaFreeHost(h_flags);
    }
}

CudaIndex::~CudaIndex() {
    cudaSetDevice(device);
    cudaStreamSynchronize(stream);
    drop_graphs();
    for (auto& p : scan_events) {
        cudaEventDestroy(p.first);
        cudaEventDestroy(p.second);
    }
    cudaFree(d_mem);  // an owner's rows and copies, and the device words; a view's words
    cudaFree(d_qraw);
    cudaFree(d_qn);
    cudaFree(d_ws);
    cudaFree(d_res);
    cudaFree(d_part_keys);
    cudaFree(d_part_done);
    if (!in_words(h_q)) cudaFreeHost(h_q);
    if (!in_words(h_res)) cudaFreeHost(h_res);
    free_words();
    cudaFree(d_q_bf16);
    cudaFree(d_q_fp8);
    cudaFree(d_q_scale);
    cudaFree(d_q_resid);
    cudaFree(d_serr);
    cudaFree(d_serr_acc);
    cudaFreeHost(h_serr_acc);
    cudaFree(d_fbq);
    cudaFree(d_thr);
    cudaFree(d_cand_idx);
    cudaFree(d_cand_sim);
    cudaFree(d_cand_cnt);
    cudaFree(d_cert);
    cudaFree(d_qsub);
    cudaFree(d_fb_idx);
    cudaFree(d_fb_sim);
    cudaFree(d_fb_cnt);
    cudaFree(d_kth);
    cudaFree(d_floor);
    cudaFree(d_rslots);
    cudaFree(d_ids);
    cudaFree(d_q2_lp);
    cudaFree(d_q2_resid);
    cudaFree(d_q2_scale);
    cudaFree(d_q2_thr);
    cudaFree(d_rows2);
    cudaFree(d_cnt2);
    cudaFree(d_ok2);
    cudaFreeHost(h_ids);
    cudaFreeHost(h_ok2);
    cudaFreeHost(h_cert);
    if (done_ev) cudaEventDestroy(done_ev);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (stream) cudaStreamDestroy(stream);
}

int CudaIndex::ensure_query_capacity(uint64_t nq) {
    int st;
    if ((st = grow_device(d_qraw, cap_qraw, nq * dims, "query buffer"))) return st;
    if ((st = grow_device(d_qn, cap_qn, nq * ds, "query buffer"))) return st;
    if (nq * dims > cap_hq && in_words(h_q)) {  // a larger batch: a buffer of its own from here on
        h_q = nullptr;
        cap_hq = 0;
    }
    if ((st = grow_host(h_q, cap_hq, nq * dims, "pinned query buffer"))) return st;
    return NNDEX_OK;
}

int CudaIndex::ensure_result_capacity(uint64_t nq, uint64_t kcap) {
    int st;
    const size_t bi = nq * kcap * sizeof(uint64_t), bs = nq * kcap * sizeof(float), bc = nq * sizeof(uint32_t);
    res_bytes = bi + bs + bc;
    if ((st = grow_device(d_res, cap_res, res_bytes, "result buffer"))) return st;
    if (res_bytes > cap_hres && in_words(h_res)) {
        h_res = nullptr;
        cap_hres = 0;
    }
    if ((st = grow_host(h_res, cap_hres, res_bytes, "pinned result buffer"))) return st;
    d_idx = reinterpret_cast<uint64_t*>(d_res);
    d_sim = reinterpret_cast<float*>(d_res + bi);
    d_cnt = reinterpret_cast<uint32_t*>(d_res + bi + bs);
    h_idx = reinterpret_cast<uint64_t*>(h_res);
    h_sim = reinterpret_cast<float*>(h_res + bi);
    h_cnt = reinterpret_cast<uint32_t*>(h_res + bi + bs);
    return NNDEX_OK;
}

// Workspace of the split merge (merge_parts(per_query, k, nq) blocks per query), into m.
int CudaIndex::merge_workspace(uint64_t per_query, uint32_t nq, uint32_t k, MergeArgs& m, cudaStream_t s) {
    const uint32_t parts = merge_parts(per_query, k, nq);
    if (parts <= 1) return NNDEX_OK;
    int st;
    if ((st = grow_device(d_part_keys, cap_part_keys, static_cast<size_t>(nq) * parts * k, "merge workspace")))
        return st;
    // counters start at zero: clear them whenever the buffer is (re)allocated (a new allocation
    // may return the old address, so compare capacities, not pointers)
    const size_t cap_before = cap_part_done;
    if ((st = grow_device(d_part_done, cap_part_done, nq, "merge workspace"))) return st;
    if (cap_part_done != cap_before) cudaMemsetAsync(d_part_done, 0, cap_part_done * sizeof(uint32_t), s);
    m.part_keys = d_part_keys;
    m.part_done = d_part_done;
    return NNDEX_OK;
}

// Enqueue the exact FP32 top-k of `nq` normalised queries (d_queries, stride ds) into the
// device outputs. Workspace is the index's own (grown on demand).
int CudaIndex::enqueue_exact_fp32(const float* d_queries, uint32_t nq, uint32_t k, uint32_t out_stride,
                                  uint64_t* o_idx, float* o_sim, uint32_t* o_cnt, cudaStream_t s) {
    ScanPlan plan;
    if (!plan_scan_fp32(nq, static_cast<uint32_t>(ds), k, rows, sm_count, smem_optin, plan))
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: k=%u above the fused top-k limit %u", k,
                         kMaxFusedK);
    const uint64_t per_query = static_cast<uint64_t>(plan.ctas_per_group) * k;
    int st = grow_device(d_ws, cap_ws, per_query * nq, "scan workspace");
    if (st) return st;
    ScanArgs a;
    a.tmap = &tmap_f32;
    a.tmap_tile = &tmap_f32_176;
    a.tmap_112 = &tmap_f32_112;
    a.queries = d_queries;
    a.nq = nq;
    a.dq = static_cast<uint32_t>(ds);
    a.rows = rows;
    a.k = k;
    a.ws_keys = d_ws;
    a.status = w_status;
    cudaEvent_t ev_a = nullptr;
    scan_event_begin(s, ev_a);
    cudaError_t e = launch_scan_fp32(a, plan, s);
    scan_event_end(s, ev_a);
    if (e != cudaSuccess) return cuda_error(e, "scan launch");
    MergeArgs m;
    m.ws_keys = d_ws;
    m.nq = nq;
    m.per_query = per_query;
    m.k = k;
    m.out_stride = out_stride;
    m.idx_out = o_idx;
    m.sim_out = o_sim;
    m.count_out = o_cnt;
    if ((st = merge_workspace(per_query, nq, k, m, s))) return st;
    e = launch_merge_topk(m, s);
    if (e != cudaSuccess) return cuda_error(e, "merge launch");
    stats.kernel_launches += 2;
    stats.path = 1;
    stats.rows_scanned += rows * nq;
    stats.scan_qb = plan.qb;
    stats.scan_wide = plan.wide;
    return NNDEX_OK;
}

// Prepare `nq` raw queries already in d_qraw (mode per K1) into d_qn.
int CudaIndex::enqueue_query_prep(uint64_t nq, int mode, cudaStream_t s) {
    PrepArgs p;
    p.src = d_qraw;
    p.rows = nq;
    p.dims = static_cast<uint32_t>(dims);
    p.out = d_qn;
    p.out_stride = static_cast<uint32_t>(ds);
    p.mode = mode;
    p.err = w_err;
    p.sm_count = sm_count;
    launch_prep_rows(p, s);
    stats.kernel_launches += 1;
    return NNDEX_OK;
}

int CudaIndex::check_device_words() {
    // h_flags[0] = err word, h_flags[1] = status word (copied with the results).
    const uint64_t err = h_flags[0];
    const uint32_t status = static_cast<uint32_t>(h_flags[1]);
    if (err != 0) return err_code(static_cast<int>(~err & 0xFF));
    if (status == kStatusTimeout)
        return set_error(NNDEX_ERR_TIMEOUT, "cuda execution error: a bounded device wait timed out");
    if (status != 0) return set_error(NNDEX_ERR_CUDA, "cuda execution error: device status %u", status);
    return NNDEX_OK;
}

// ---- path choice (rules by batch size, k and the index's copies) ----------------------------

// The tensor-core scan of the BF16 or FP8 copy holds k results (and there is such a copy).
bool CudaIndex::tc_fits(uint64_t kcap, bool fp8) const {
    if (fp8 ? !d_base_fp8 : !d_base_bf16) return false;
    const TcPlan p1 = plan_tc(kcap, fp8);
    return p1.stages > 0 && p1.kp >= kcap && p1.kp > 0 && plan_tc(0, fp8).stages > 0;
}

int CudaIndex::choose_path(uint64_t nq, uint64_t kcap) const {
    auto tc_ok = [&](bool fp8) { return tc_fits(kcap, fp8); };
    // Small batches (plan_tf32's range): the TF32 candidate scan, which reads the same FP32 base and
    // returns the same bits as the FP32 scan at the HBM rate, where the FP32 scan is bound by its
    // FMA issue.
    const int fp32_path = plan_tf32(nq, kcap).kp ? 6 : plan_tf32_batch(nq, kcap).kp ? 7 : 1;
    switch (precision) {
        case NNDEX_PRECISION_FP32: return fp32_path;
        case NNDEX_PRECISION_BF16: return tc_ok(false) ? 2 : 1;
        case NNDEX_PRECISION_FP8: return tc_ok(true) ? 3 : 1;
        default:
            // FP32 streaming is HBM-bound at small batches; the tensor cores win from a few dozen
            // queries per batch (the scan becomes compute-bound in FP32).
            if (nq >= 64) {
                if (tc_ok(false)) return 2;
                if (tc_ok(true)) return 3;
            }
            return fp32_path;
    }
}

CudaIndex::Tf32Plan CudaIndex::plan_tf32(uint64_t nq, uint64_t kcap) const {
    Tf32Plan p;
    static const uint32_t min_q = [] {
        const char* v = getenv("NNDEX_TF32_MIN_QUERIES");  // measurement override of the batch rule
        return v ? static_cast<uint32_t>(atoi(v)) : 9u;
    }();
    static const bool off = [] {
        const char* v = getenv("NNDEX_TF32_SCAN");  // 0: small batches always take the FP32 scan
        return v && v[0] == '0';
    }();
    if (off || !d_tfnorm || nq < std::max<uint32_t>(min_q, 1) || nq > 16 || kcap == 0 || kcap > 448) return p;
    // k′: 2.5 k rounded up to 32, at least k + 64 and at most 512, so that the exact k-th score
    // clears the k′-th bound on clustered data (on a 1,024-centre mixture of 1M × 768 rows the
    // 100th and 256th scores of a query are ≈ 2.4e-3 apart, twice the bound's typical ε)
    const uint64_t kp = std::min<uint64_t>(512, (std::max<uint64_t>(kcap * 5 / 2, kcap + 64) + 31) / 32 * 32);
    if (rows < 4 * kp || rows > 0xFFFFFFFFull) return p;
    // Each CTA lists a quarter of k′ (at least 32): the k′ best of a query come from all 148 CTAs,
    // and the rows a full list left out score below the largest full-list minimum (the floor),
    // which the certificate then also has to clear.
    const uint32_t kp_cta = static_cast<uint32_t>(std::max<uint64_t>(32, (kp / 4 + 31) / 32 * 32));
    // Room for three tiles of survivors above the list: a selection runs once ≥ 256 keys have
    // accumulated since the last one, not after every tile.
    const uint32_t cap = kp_cta + 3 * 128;
    const uint32_t stages = tf32_stages_for(cap, smem_optin);
    if (!stages) return p;
    p.kp = static_cast<uint32_t>(kp);
    p.kp_cta = kp_cta;
    p.cap = cap;
    p.stages = stages;
    return p;
}

// Batches of 17 queries and more of an FP32 index: the FP32 scan is bound by its FMAs there, the
// tensor cores read the same base at the HBM rate.
CudaIndex::Tf32BatchPlan CudaIndex::plan_tf32_batch(uint64_t nq, uint64_t kcap) const {
    Tf32BatchPlan p;
    static const bool off = [] {
        const char* v = getenv("NNDEX_TF32_SCAN");  // 0: FP32 batches always take the FP32 scan
        return v && v[0] == '0';
    }();
    if (off || !d_tfnorm || nq < 17 || kcap == 0 || kcap > kMaxGroupCandidates / 2) return p;
    const uint64_t kp = std::min<uint64_t>(rows, std::max<uint64_t>(32, 2 * kcap));
    // Pass 1 on every stride-th tile: few enough that the groups of 8 rows are at least 16 per
    // candidate, and that pass 2 collects about stride × k ≤ 2,048 rows per query.
    const uint64_t tiles = (rows + 255) / 256;
    uint32_t stride = 32;
    while (stride > 1 && ((tiles + stride - 1) / stride * 32 < 16 * kp || stride * kcap > 2048 ||
                          (stride > 8 && tiles < 16384)))
        stride /= 2;
    if (tiles * 32 < 4 * kp) return p;
    if (rows * nq * (ds + 64) < tf32_batch_costs(rows, ds, nq, kcap, stride, host_fallback)) return p;
    const uint32_t nchunks = static_cast<uint32_t>(ds / 32);
    bool stream_a = false;
    const uint32_t stages = tc_tf32_stages_for(nchunks, smem_optin, &stream_a);
    if (!stages) return p;
    plan_groups(static_cast<uint32_t>((nq + 127) / 128), static_cast<uint32_t>(kp), stride, p.group, p.span, p.gm_tiles,
                p.nranges, p.range_rows);
    if (!p.group) return p;
    p.stride = stride;
    p.stages = stages;
    p.stream_a = stream_a;
    p.kp = static_cast<uint32_t>(kp);
    return p;
}

// C of K12's bound, per unit ‖q‖‖x‖:
//   the tensor core's FP32 accumulation of ds exact TF32 products (each added with up to one FP32
//   rounding, 4× margin, as for the BF16 scan):                              4·ds·2⁻²³
//   the FP32 scan's own rounding (eight chains of ds/8 FMAs, then 3 adds):  (ds/8 + 3)·2⁻²⁴
//   the rounding of u = s̃ + ε:                                             2⁻²²
float CudaIndex::tf32_c_norm() const {
    const double d = static_cast<double>(ds);
    return static_cast<float>((4.0 * d * std::ldexp(1.0, -23) + (d / 8.0 + 3.0) * std::ldexp(1.0, -24) +
                               std::ldexp(1.0, -22)) * 1.01);
}

// For unit rows and queries ‖d_v‖ < 2⁻¹⁰: ε < 2·2⁻¹⁰ + 2⁻²⁰ + C.
float CudaIndex::tf32_eps() const {
    return static_cast<float>((2.0 * std::ldexp(1.0, -10) + std::ldexp(1.0, -20) + tf32_c_norm()) * 1.01);
}

// IVF batches: the tensor-core list scan (5) from a few dozen queries, when the index's precision
// allows low-precision scoring and k fits its pass-1 heaps; else the FP32 list scan (4).
int CudaIndex::ivf_path(uint64_t nq, uint64_t kcap) const {
    if (precision == NNDEX_PRECISION_FP32 || nq < 64 || !ivf || !ivf->d_reordered16) return 4;
    // The tensor-core list scan scores 128-query blocks per list chunk (≤ 4096 rows). With few
    // queries per probed list and short lists its items are small and their fixed cost dominates:
    // on 2M × 384 (nlist 1414, lists of ≈ 1,400 rows) with 1024 queries, nprobe 8 (≈ 6 queries per
    // list) runs faster on the FP32 list scan (489k vs 350k q/s), nprobe 32 (≈ 23) and 64 (≈ 46)
    // on the tensor cores (345k vs 269k, 324k vs 174k). With long lists (5M × 512, nlist 512, lists
    // of ≈ 9,800 rows) the tensor cores win from 64 queries on (serving at saturation: 157k vs 132k
    // q/s). So: the FP32 list scan when a probed list serves fewer than 12 queries on average and
    // the average list is shorter than one 4096-row chunk.
    const uint64_t np0 = ivf_scratch.nprobe ? ivf_scratch.nprobe : ivf_choose_nprobe(ivf->nlist, kcap, rows);
    const double per_list = static_cast<double>(nq) * static_cast<double>(std::min<uint64_t>(np0, ivf->nlist)) /
                            static_cast<double>(ivf->nlist);
    static const double min_per_list = [] {
        const char* v = getenv("NNDEX_IVF_TC_MIN_PER_LIST");  // measurement override of the rule
        return v ? atof(v) : 12.0;
    }();
    if (per_list < min_per_list && rows / ivf->nlist < 4096) return 4;
    const TcPlan p1 = plan_tc(kcap, false);
    return (p1.kp >= kcap && p1.kp > 0 && plan_tc(0, false).stages > 0) ? 5 : 4;
}

uint32_t CudaIndex::tc_chunks(bool fp8) const {
    return static_cast<uint32_t>((fp8 ? kf8 : kb16 * 2) / 128);
}

// Shared-memory plan of a tensor-core pass. kcap = 0 plans pass 2 (no heaps). Pass 1 wants
// k′ = max(32, 2k) heap entries per query (enough that most queries certify) beside a 4-deep ring
// with the query block resident; it gives up, in order: the ring depth for a k′ that still holds k
// (queries that do not certify take the threshold pass), then the resident query block (its slabs
// then travel with every ring stage), then the k′ margin (k′ = k).
CudaIndex::TcPlan CudaIndex::plan_tc(uint64_t kcap, bool fp8) const {
    const uint32_t nchunks = tc_chunks(fp8);
    TcPlan out;
    if (kcap == 0) {
        out.stages = tc_stages_for(nchunks, 0, fp8, false, smem_optin);
        // The query slabs stay in shared memory only beside a ring that is deep enough: a base slab a
        // stage comes from L2 at best, and with two stages its latency shows on every slab. 1M × 512 in
        // BF16, 512 queries: 829 us with two 32 KB stages beside the queries, 605 with four 48 KB stages
        // that carry the query slabs too; × 448 (three stages) 586 -> 555. FP8 slabs pass through twice
        // as fast, so the extra bytes weigh more: × 1,024 1,022 -> 876, × 768 (three stages) 696 -> 704.
        if (out.stages < (fp8 ? 3u : 4u)) {
            out.stream_a = true;
            out.stages = tc_stages_for(nchunks, 0, fp8, true, smem_optin);
        }
        return out;
    }
    auto largest = [&](bool stream_a, bool four) {
        uint32_t best = 0;
        for (uint32_t kp = 8; kp <= 2048; kp += 8) {
            const uint32_t stg = tc_stages_for(nchunks, kp, fp8, stream_a, smem_optin);
            if (four ? stg == 4 : stg != 0) best = kp;
        }
        return best;
    };
    const uint32_t kmax4 = largest(false, true), kmax = largest(false, false), kmax_s = largest(true, false);
    uint32_t want = rerank_width ? rerank_width : static_cast<uint32_t>(std::max<uint64_t>(32, 2 * kcap));
    if (want > rows) want = static_cast<uint32_t>(rows);
    uint32_t kp = want;
    if (kp > kmax4 && kcap <= kmax4 && !rerank_width) kp = kmax4;
    if (kp > kmax) kp = kmax;
    if (kp >= kcap && kp > 0) {
        out.kp = kp;
        out.stages = tc_stages_for(nchunks, kp, fp8, false, smem_optin);
        return out;
    }
    kp = std::min(want, kmax_s);  // streamed query slabs
    if (kp < kcap) return out;    // no tensor-core plan: the FP32 scan serves this k
    out.kp = kp;
    out.stream_a = true;
    out.stages = tc_stages_for(nchunks, kp, fp8, true, smem_optin);
    return out;
}

uint32_t CudaIndex::group_candidates(uint64_t kcap) const {
    uint64_t want = rerank_width ? std::max<uint64_t>(rerank_width, kcap) : std::max<uint64_t>(32, 2 * kcap);
    want = std::min<uint64_t>(want, rows);
    return want <= kMaxGroupCandidates && want >= kcap ? static_cast<uint32_t>(want) : 0u;
}

int CudaIndex::enqueue_prep_queries(const float* d_raw, uint64_t n, int mode, int path, cudaStream_t s) {
    int st;
    PrepArgs p;
    p.src = d_raw;
    p.rows = n;
    p.dims = static_cast<uint32_t>(dims);
    p.out = d_qn;
    p.out_stride = static_cast<uint32_t>(ds);
    p.mode = mode;
    p.err = w_err;
    p.sm_count = sm_count;
    // What the path's later kernels expect zeroed, and the two-pass TF32 scan's slack.
    if (path == 4 || path == 5) {
        if ((st = ivf_plan_words(*this, &p.zero[0], &p.zero_words[0]))) return st;
    } else if (path == 6) {
        if ((st = grow_device(d_floor, cap_floor, n, "tc workspace"))) return st;
        p.zero[0] = reinterpret_cast<uint32_t*>(d_floor);
        p.zero_words[0] = 2 * n;
        p.zero[1] = d_fbn;
        p.zero_words[1] = 1;
    } else if (path == 7) {
        p.tf_slack = d_q_resid;  // (settle_path has grown it, and d_cnt2)
        p.tf_row_max = d_tfnorm + rows;
        p.tf_c_norm = tf32_c_norm();
        p.tf_collected = d_cnt2;
        p.tf_over = kSecondPassCap + 1;
        p.zero[1] = d_fbn;
        p.zero_words[1] = 4;
    }
    if (path == 2 || path == 3 || path == 5) {
        const uint64_t nq_alloc = (n + 127) / 128 * 128;
        if ((st = grow_device(d_q_resid, cap_q_resid, n, "query buffer"))) return st;
        if (path == 2 || path == 5) {
            const bool grew = nq_alloc * kb16 > cap_q_bf16;
            if ((st = grow_device(d_q_bf16, cap_q_bf16, nq_alloc * kb16, "query buffer"))) return st;
            if (grew) cudaMemsetAsync(d_q_bf16, 0, cap_q_bf16 * sizeof(__nv_bfloat16), s);
            p.out_bf16 = d_q_bf16;
            p.bf16_stride = static_cast<uint32_t>(kb16);
            p.resid_bf16 = d_q_resid;
        } else {
            const bool grew = nq_alloc * kf8 > cap_q_fp8;
            if ((st = grow_device(d_q_fp8, cap_q_fp8, nq_alloc * kf8, "query buffer"))) return st;
            if (grew) cudaMemsetAsync(d_q_fp8, 0, cap_q_fp8, s);
            if ((st = grow_device(d_q_scale, cap_q_scale, n, "query buffer"))) return st;
            p.out_fp8 = d_q_fp8;
            p.fp8_stride = static_cast<uint32_t>(kf8);
            p.fp8_scale = d_q_scale;
            p.resid_fp8 = d_q_resid;
        }
    }
    launch_prep_rows(p, s);
    stats.kernel_launches += 1;
    return NNDEX_OK;
}

int CudaIndex::enqueue_tc(bool fp8, uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt,
                          cudaStream_t s) {
    int st;
    const TcPlan plan = plan_tc(kcap, fp8);
    if (!plan.stages || plan.kp < kcap)
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: k'=%u does not fit", plan.kp);
    const uint32_t nqb = (n + 127) / 128;
    // Autotuned: when the last batch rarely certified in pass 1, pass 1 only has to produce each
    // query's threshold T, and a sample of the rows (every 8th tile) gives a valid one.
    // The tuner's plan may fix it instead (only bases of ≥ 64 tiles are sampled).
    // At k ≥ 64 the rules start sampled: a full pass 1 then carries the largest heaps and almost
    // never certifies (the k′ the shared memory allows is little above k), and the rule's state is
    // shared with the index's small-k batches, which may keep it at 1.
    const uint32_t want = forced_stride ? forced_stride : (kcap >= 64 ? 8u : tc_sample_stride);
    const uint32_t stride = (want > 1 && rows >= 256ull * 64) ? want : 1;
    uint64_t nranges = 0, range_rows = 0;
    tc_ranges(rows, nqb, nranges, range_rows);
    // A sampled pass 1 writes group maxima instead of keeping heaps, where plan_groups finds enough.
    const uint32_t gkp = stride > 1 ? group_candidates(kcap) : 0u;
    uint32_t group = 0, gm_tiles = 0, span = 1;
    if (gkp) plan_groups(nqb, gkp, stride, group, span, gm_tiles, nranges, range_rows);
    tc_groups = group != 0;
    const uint32_t kp = tc_groups ? gkp : plan.kp;
    const uint64_t gm_words = nranges * gm_tiles * (tc_groups ? 256 / group : 0);  // per query, 4 bytes each
    const uint64_t per_query = tc_groups ? (gm_words + 1) / 2 : nranges * kp;
    if ((st = grow_device(d_thr, cap_thr, n, "tc workspace"))) return st;
    if ((st = grow_device(d_ws, cap_ws, per_query * n, "tc workspace"))) return st;
    if ((st = grow_device(d_ids, cap_ids, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_cand_idx, cap_cand_idx, static_cast<uint64_t>(n) * kp, "tc workspace"))) return st;
    if ((st = grow_device(d_cand_sim, cap_cand_sim, static_cast<uint64_t>(n) * kp, "tc workspace"))) return st;
    if ((st = grow_device(d_cand_cnt, cap_cand_cnt, n, "tc workspace"))) return st;
    if ((st = grow_device(d_cert, cap_cert, n, "tc workspace"))) return st;
    if ((st = grow_device(d_kth, cap_kth, n, "tc workspace"))) return st;
    CUtensorMap tmap_q;
    if ((st = encode_query_tmap(fp8, fp8 ? static_cast<void*>(d_q_fp8) : static_cast<void*>(d_q_bf16), n, &tmap_q)))
        return st;
    TcArgs a;
    a.tmap_q = &tmap_q;
    a.tmap_b = fp8 ? &tmap_fp8 : &tmap_bf16;
    a.nranges = static_cast<uint32_t>(nranges);
    fill_tc_params(fp8, n, range_rows, a.p);
    last_tc_stride = stride;
    stats.pass1_tile_stride = stride;
    stats.path = fp8 ? 3 : 2;
    stats.rerank_width = kp;
    stats.rows_scanned += rows * n;
    cudaEvent_t ev_a = nullptr;
    cudaError_t e;
    if (tc_groups) {
        const TcPlan plan2 = plan_tc(0, fp8);  // no heaps: pass 2's shared-memory plan
        a.stages = plan2.stages;
        a.stream_a = plan2.stream_a;
        a.p.tile_stride = stride;
        a.p.gm = reinterpret_cast<uint32_t*>(d_ws);
        a.p.gm_tiles = gm_tiles;
        a.p.gm_group = group;
        a.p.gm_span = span;
        scan_event_begin(s, ev_a);
        e = launch_scan_tc(a, fp8 ? kTcFp8 : kTcBf16, 2, s);
        scan_event_end(s, ev_a);
        if (e != cudaSuccess) return cuda_error(e, "tensor-core scan launch");
        TcThresholdArgs t;
        t.gm = a.p.gm;
        t.words = gm_words;
        t.group = group;
        t.tiles = gm_tiles;
        t.span = span;
        t.stride = stride;
        t.parts = nranges;
        t.range_rows = range_rows;
        t.rows = rows;
        t.base = d_base;
        t.ds = static_cast<uint32_t>(ds);
        t.queries = d_qn;
        t.nq = n;
        t.kp = kp;
        t.k = kcap;
        t.q_resid = d_q_resid;
        t.q_scale = fp8 ? d_q_scale : nullptr;
        t.eps_rows = a.p.eps_rows;
        t.eps_acc = a.p.eps_acc;
        t.cand_idx = d_cand_idx;
        t.cand_sim = d_cand_sim;
        t.cand_cnt = d_cand_cnt;
        t.cert = d_cert;
        t.kth = d_kth;
        t.ids = d_ids;
        t.live = d_fbn + 1;
        if ((e = launch_threshold(t, s)) != cudaSuccess) return cuda_error(e, "threshold launch");
        stats.kernel_launches += 2;
        return NNDEX_OK;
    }
    cudaMemsetAsync(d_thr, 0, n * sizeof(unsigned long long), s);
    a.stages = plan.stages;
    a.stream_a = plan.stream_a;
    a.p.q_resid = d_q_resid;
    a.p.q_scale = fp8 ? d_q_scale : nullptr;
    a.p.kprime = kp;
    a.p.heap_k = stride > 1 ? std::max(1u, std::min(kp, kcap)) : kp;  // a sampled pass 1 only yields T
    a.p.thr_global = d_thr;
    a.p.ws_keys = d_ws;
    a.p.tile_stride = stride;
    scan_event_begin(s, ev_a);
    e = launch_scan_tc(a, fp8 ? kTcFp8 : kTcBf16, 0, s);
    scan_event_end(s, ev_a);
    if (e != cudaSuccess) return cuda_error(e, "tensor-core scan launch");
    MergeArgs m;
    m.ws_keys = d_ws;
    m.nq = n;
    m.per_query = per_query;
    m.k = kp;
    m.out_stride = kp;
    m.idx_out = d_cand_idx;
    m.sim_out = d_cand_sim;
    m.count_out = d_cand_cnt;
    if ((st = merge_workspace(per_query, n, kp, m, s))) return st;
    if ((e = launch_merge_topk(m, s)) != cudaSuccess) return cuda_error(e, "merge launch");
    RerankArgs r;
    r.base = d_base;
    r.ds = static_cast<uint32_t>(ds);
    r.queries = d_qn;
    r.cand_idx = d_cand_idx;
    r.cand_sim = d_cand_sim;
    r.cand_cnt = d_cand_cnt;
    r.nq = n;
    r.kp = kp;
    r.k = kcap;
    r.idx_out = o_idx;
    r.sim_out = o_sim;
    r.cnt_out = o_cnt;
    r.cert_out = d_cert;
    r.kth_out = d_kth;
    r.certify = stride == 1;
    if ((e = launch_rerank(r, s)) != cudaSuccess) return cuda_error(e, "rerank launch");
    stats.kernel_launches += 3;
    return NNDEX_OK;
}

// The groups of a sampled pass 1 (every stride-th tile) for kp candidates per query, and its ranges,
// split over the sampled tiles. Groups of 32 columns where a query has at least 64 of them per
// candidate (two of its best rows then rarely share one, which would lower T), of as many tiles as
// still leave 64 (fewer words to write, read and hold: 512 bytes per candidate at most, what the
// heaps' slots are admitted at); groups of 8 columns on smaller samples, and none (group 0, the ranges
// as they were) where even those are fewer than four per candidate.
void CudaIndex::plan_groups(uint32_t nqb, uint32_t kp, uint32_t stride, uint32_t& group, uint32_t& span,
                            uint32_t& gm_tiles, uint64_t& nranges, uint64_t& range_rows) const {
    const uint64_t sampled = ((rows + 255) / 256 + stride - 1) / stride;
    group = sampled * 8 >= 64ull * kp ? 32u : (sampled * 32 >= 4ull * kp ? 8u : 0u);
    span = 1;
    if (!group) return;
    uint64_t nr = 0, rr = 0;
    tc_ranges(sampled * 256, nqb, nr, rr, 256);
    const uint64_t per_range = rr / 256;
    while (group == 32 && span < kMaxGroupSpan && span * 2 <= per_range && sampled * 8 >= 64ull * kp * span * 2) span *= 2;
    nranges = nr;
    range_rows = rr * stride;
    gm_tiles = static_cast<uint32_t>((per_range + span - 1) / span);
}

// Row ranges of the tensor-core grid over `scan_rows` rows: about four waves of CTAs, each range a
// multiple of the 256-row tile. Concurrent CTAs share ranges, so a base tile is read from HBM about
// once.
void CudaIndex::tc_ranges(uint64_t scan_rows, uint32_t nqb, uint64_t& nranges, uint64_t& range_rows,
                          uint64_t min_rows) const {
    tc_range_split(scan_rows, nqb, static_cast<uint64_t>(sm_count), nranges, range_rows, min_rows);
}

void CudaIndex::fill_tc_params(bool fp8, uint32_t n, uint64_t range_rows, TcParams& p) const {
    const uint64_t kb = fp8 ? kf8 : kb16;
    p.nq = n;
    p.nchunks = tc_chunks(fp8);
    p.rows = rows;
    p.range_rows = range_rows;
    p.row_scale = fp8 ? d_row_scale : nullptr;
    p.tile_scale = fp8 ? d_tile_scale : nullptr;
    p.row_resid = fp8 ? d_res8 : d_res16;
    p.eps_rows = fp8 ? eps_fp8 : eps_bf16;
    // FP32 accumulation of kb exact products (|Σ| ≤ 1 + ε): kb·2^-23, with a 4× margin.
    p.eps_acc = 4.0f * static_cast<float>(kb) * 1.1920929e-07f;
    p.status = w_status;
}

int CudaIndex::encode_query_tmap(bool fp8, void* buf, uint32_t n, CUtensorMap* map) const {
    const uint64_t nq_alloc = (n + 127) / 128 * 128;
    const bool ok = fp8 ? encode_tmap_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, buf, kf8, nq_alloc, kf8, 128, 128,
                                         CU_TENSOR_MAP_SWIZZLE_128B)
                        : encode_tmap_2d(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, buf, kb16, nq_alloc, kb16 * 2, 64,
                                         128, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!ok)
        return set_error(NNDEX_ERR_CUDA,
                         "cuda execution error: cuTensorMapEncodeTiled failed (queries: %s, %u rows, row length %llu, "
                         "buffer %p, driver result %d)",
                         fp8 ? "FP8" : "BF16", n, (unsigned long long)(fp8 ? kf8 : kb16), buf, last_encode_result());
    return NNDEX_OK;
}

// After pass 1: queries whose certificate held are final. The others run pass 2 (collect every row
// whose upper bound reaches their exact k-th score, rerank exactly) — all on the device, sized for
// the worst case (every query uncertified), the kernels reading the count that the compaction left.
int CudaIndex::enqueue_tc_pass2(bool fp8, uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim,
                                uint32_t* o_cnt, cudaStream_t s) {
    int st;
    const uint32_t cap2 = kSecondPassCap;
    const uint64_t row_bytes = fp8 ? kf8 : kb16 * 2;
    const uint64_t n_alloc = (n + 127) / 128 * 128;
    if ((st = grow_device(d_ids, cap_ids, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_q2_lp, cap_q2_lp, n_alloc * row_bytes, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_q2_resid, cap_q2_resid, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_q2_scale, cap_q2_scale, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_q2_thr, cap_q2_thr, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_rows2, cap_rows2, static_cast<uint64_t>(n) * cap2, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_cnt2, cap_cnt2, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_ok2, cap_ok2, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_tcfail, cap_tcfail, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_rslots, cap_rslots, static_cast<uint64_t>(n) * rerank_chunks(cap2) * kcap,
                          "pass-2 buffer")))
        return st;
    uint32_t* d_m = d_fbn + 1;      // uncertified queries
    uint32_t* d_fail = d_fbn + 2;   // of them, collections that overflowed
    cudaError_t e = cudaSuccess;
    if (!tc_groups) {
        launch_compact_zero_flags(d_cert, n, d_ids, d_m, s);
        e = launch_gather_queries(d_ids, n, fp8 ? static_cast<const void*>(d_q_fp8)
                                                : static_cast<const void*>(d_q_bf16),
                                  static_cast<uint32_t>(row_bytes), d_q2_lp, d_q_resid, d_q2_resid,
                                  fp8 ? d_q_scale : nullptr, d_q2_scale, d_kth, d_q2_thr, s, d_m);
        if (e != cudaSuccess) return cuda_error(e, "gather launch");
        stats.kernel_launches += 2;
    }
    cudaMemsetAsync(d_cnt2, 0, n * sizeof(uint32_t), s);
    // after group maxima every query is in pass 2, in the batch's order: its own buffers serve
    void* q_lp = !tc_groups ? static_cast<void*>(d_q2_lp) : fp8 ? static_cast<void*>(d_q_fp8) : static_cast<void*>(d_q_bf16);
    const float* q_thr = tc_groups ? d_kth : d_q2_thr;
    CUtensorMap tmap_q2;
    if ((st = encode_query_tmap(fp8, q_lp, n, &tmap_q2))) return st;
    TcArgs a;
    a.tmap_q = &tmap_q2;
    a.tmap_b = fp8 ? &tmap_fp8 : &tmap_bf16;
    const TcPlan plan2 = plan_tc(0, fp8);
    a.stages = plan2.stages;
    a.stream_a = plan2.stream_a;
    // Two query blocks per CTA (where both fit beside a ring: D ≤ 256 in BF16, 512 in FP8) read half
    // the base bytes per FLOP but run M = 128, N = 128 MMAs, which read as many query bytes from
    // shared memory as base bytes. On 10M × 256 at 4,096 queries that made BF16 7 % slower, and FP8
    // 7 % faster only while the row ranges left SMs idle in a last partial round (the autotuner has
    // taken one block for FP8 since): the rule takes one block, and the autotuner times both.
    // CTA pairs (qb = 3): two CTAs, one query block each, share every 256-row base tile through
    // M = 256 MMAs, so each SM reads half the base bytes per FLOP without narrowing the MMA.
    const uint32_t want_qb = forced_qb ? forced_qb : 1u;
    const uint32_t pair_stages = (want_qb == 2 && n > 128) ? tc_pair_stages_for(tc_chunks(fp8), fp8, smem_optin) : 0;
    const uint32_t cta_pair_stages =
        (want_qb == 3 && n > 128) ? tc_cta_pair_stages_for(tc_chunks(fp8), fp8, smem_optin) : 0;
    if (pair_stages || cta_pair_stages) {
        a.qb = pair_stages ? 2 : 3;
        a.stages = pair_stages ? pair_stages : cta_pair_stages;
        a.stream_a = false;
        a.tmap_b = fp8 ? &tmap_fp8_h : &tmap_bf16_h;
    }
    stats.pass2_query_blocks = a.qb;
    fill_tc_params(fp8, n, 0, a.p);
    a.p.q_resid = tc_groups ? d_q_resid : d_q2_resid;
    a.p.q_scale = !fp8 ? nullptr : tc_groups ? d_q_scale : d_q2_scale;
    a.p.q_thr = q_thr;
    a.p.cand_rows = d_rows2;
    a.p.cand_cnt = d_cnt2;
    a.p.cap2 = cap2;
    a.p.live_q = d_m;
    a.p.sm_count = static_cast<uint32_t>(sm_count);
    // (query block, row range) items for any count ≤ n: at most 8 per SM plus one per block
    // (tc_range_split: at most 8 rounds, or one range per block)
    a.live_items = 8u * static_cast<uint32_t>(sm_count) + static_cast<uint32_t>(n_alloc / 128) + 1u;
    cudaEvent_t ev_a = nullptr;
    scan_event_begin(s, ev_a);
    e = launch_scan_tc(a, fp8 ? kTcFp8 : kTcBf16, 1, s);
    scan_event_end(s, ev_a);
    if (e != cudaSuccess) return cuda_error(e, "tensor-core scan launch (pass 2)");
    e = launch_rerank_collected(d_base, static_cast<uint32_t>(ds), d_qn, d_ids, n, d_rows2, d_cnt2, cap2, kcap,
                                q_thr, d_rslots, o_idx, o_sim, o_cnt, d_ok2, s, false, d_m);
    if (e != cudaSuccess) return cuda_error(e, "rerank launch (pass 2)");
    launch_compact_zero_flags(d_ok2, n, d_tcfail, d_fail, s, d_m, batch_report());
    stats.kernel_launches += 4;
    last_tc_n = n;
    return NNDEX_OK;
}

// What the host reads after a tensor-core batch, written by its last kernel.
BatchReport CudaIndex::batch_report() const {
    BatchReport r;
    r.cnt = d_cnt2;
    r.cap = kSecondPassCap;
    r.host_counts = h_fbn;
    if (w_err == d_err) {
        r.flags = d_err;
        r.host_flags = reinterpret_cast<unsigned long long*>(h_flags);
    }
    return r;
}

int CudaIndex::finish_tc(uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt,
                         cudaStream_t s) {
    const uint32_t m = h_fbn[1], failed_n = h_fbn[2];
    stats.certified = m == 0 ? 1u : 0u;
    stats.second_pass_queries = m;
    // The rule for the next batch (when no tuned plan fixes the stride): a full pass 1 pays off only
    // when it certifies most queries.
    if (!forced_stride) {
        const uint32_t before = tc_sample_stride;
        if (last_tc_stride == 1) tc_sample_stride = (m * 2 > n) ? 8u : 1u;
        else if (m * 2 <= n) tc_sample_stride = 1;
        if (tc_sample_stride != before) drop_graphs();  // a captured batch keeps its stride
    }
    tc_patched = false;
    int st;
    stats.pass2_rows += h_fbn_rows();
    if (failed_n == 0) return NNDEX_OK;
    std::vector<uint32_t> failed;
    if (tc_retry_rest && failed_n <= tc_retry_rest_m) {
        --tc_retry_rest;
        if ((st = overflowed_queries(m, failed_n, s, &failed))) return st;
    } else {
        if ((st = retry_tc_pass2(stats.path == 3, failed_n, kcap, o_idx, o_sim, o_cnt, s, &failed))) return st;
        if (!retry_paid(failed_n, static_cast<uint32_t>(failed.size()))) {
            tc_retry_rest = kTcRetryRest;
            tc_retry_rest_m = failed_n;
        }
    }
    tc_patched = true;
    stats.fp32_fallback_queries += static_cast<uint32_t>(failed.size());
    if (failed.empty()) return NNDEX_OK;
    // ---- the FP32 scan for queries whose collected set overflowed again ----
    return rerun_exact_fp32(failed, kcap, o_idx, o_sim, o_cnt, s);
}

// Whether the second pass 2 of m queries, which left `failed` of them overflowed, cost less than the FP32 scan of
// the others (us): a re-run query takes about 16 of copies, its share of a scan per 16 queries that the scan
// no longer runs for; the pass about 20, then the exact scores of 8,192 rows a query. 64k × 1,024 in FP8,
// k = 100, with / without: 16 queries, 9 left, 853 / 704; 128, 82 left, 2,517 / 2,664; 512, 295 left, 7,324 /
// 9,221; 32k × 1,024, 2, none left, 584 / 441; 256k × 1,024 2, none left, 441 / 489; 128k × 256 16, 5 of them
// overflowed, none left, 312 / 354. And it reads the copy: 1.3M × 8 in FP8, 8 queries, one of them overflowed, none
// left, 458 / 351; 3.5M × 34, 141, 135 left, 7,343 / 6,603; 2M × 8, 26, 24 left, 1,555 / 1,258.
bool CudaIndex::retry_paid(uint32_t m, uint32_t failed) const {
    const double d = static_cast<double>(ds), scans = (m + 15) / 16 - (failed + 15) / 16, n = static_cast<double>(rows);
    const double copy = n * static_cast<double>(stats.path == 3 ? kf8 : 2 * kb16) * ((m + 127) / 128);
    return 16.0 * (m - failed) + scans * n * d * 5.3e-7 > 20.0 + 0.1 * d + m * d * 3.3e-3 + copy * 1.5e-7;
}

// The queries whose collection overflowed, without another pass.
int CudaIndex::overflowed_queries(uint32_t m, uint32_t failed_n, cudaStream_t s, std::vector<uint32_t>* failed) {
    int st;
    if ((st = grow_host(h_ids, cap_hids, m, "pinned buffer"))) return st;
    if ((st = grow_host(h_ok2, cap_hok2, failed_n, "pinned buffer"))) return st;
    cudaMemcpyAsync(h_ids, d_ids, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h_ok2, d_tcfail, failed_n * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(e, "search");
    failed->resize(failed_n);
    for (uint32_t i = 0; i < failed_n; ++i) (*failed)[i] = h_ids[h_ok2[i]];
    return NNDEX_OK;
}

// A collection overflows when T is far below the query's true k-th score (a sampled pass 1, or FP8's
// wide slack over a dense cluster). The 8,192 rows it did collect are an arbitrary part of the rows
// above T − slack, so their exact k-th score is a much higher T, and one more pass over the copy
// collects few rows. On 2M × 512 in FP8, 21 such queries of 1,000 (k = 100) took 2.5 ms on the FP32
// scan, copied row by row; their second pass takes 0.45 ms.
int CudaIndex::retry_tc_pass2(bool fp8, uint32_t m, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt,
                              cudaStream_t s, std::vector<uint32_t>* failed) {
    int st;
    const uint32_t cap2 = kSecondPassCap;
    const uint32_t row_bytes = static_cast<uint32_t>(fp8 ? kf8 : kb16 * 2);
    if ((st = grow_device(d_fbq, cap_fbq, m, "fallback buffer"))) return st;
    cudaError_t e = launch_rerank_collected(d_base, static_cast<uint32_t>(ds), d_qn, d_ids, m, d_rows2, d_cnt2, cap2,
                                            kcap, d_kth, d_rslots, nullptr, nullptr, nullptr, nullptr, s, false, nullptr,
                                            nullptr, d_tcfail, d_kth, d_fbq);
    if (e != cudaSuccess) return cuda_error(e, "rerank launch (overflow)");
    e = launch_gather_queries(d_fbq, m, fp8 ? static_cast<const void*>(d_q_fp8) : static_cast<const void*>(d_q_bf16),
                              row_bytes, d_q2_lp, d_q_resid, d_q2_resid, fp8 ? d_q_scale : nullptr, d_q2_scale, d_kth,
                              d_q2_thr, s);
    if (e != cudaSuccess) return cuda_error(e, "gather launch (overflow)");
    cudaMemsetAsync(d_cnt2, 0, m * sizeof(uint32_t), s);
    CUtensorMap tmap_q2;
    if ((st = encode_query_tmap(fp8, d_q2_lp, m, &tmap_q2))) return st;
    TcArgs a;
    a.tmap_q = &tmap_q2;
    a.tmap_b = fp8 ? &tmap_fp8 : &tmap_bf16;
    const TcPlan plan2 = plan_tc(0, fp8);
    a.stages = plan2.stages;
    a.stream_a = plan2.stream_a;
    uint64_t nranges = 0, range_rows = 0;
    tc_ranges(rows, (m + 127) / 128, nranges, range_rows, 256);
    a.nranges = static_cast<uint32_t>(nranges);
    fill_tc_params(fp8, m, range_rows, a.p);
    a.p.q_resid = d_q2_resid;
    a.p.q_scale = fp8 ? d_q2_scale : nullptr;
    a.p.q_thr = d_q2_thr;
    a.p.cand_rows = d_rows2;
    a.p.cand_cnt = d_cnt2;
    a.p.cap2 = cap2;
    cudaEvent_t ev_a = nullptr;
    scan_event_begin(s, ev_a);
    e = launch_scan_tc(a, fp8 ? kTcFp8 : kTcBf16, 1, s);
    scan_event_end(s, ev_a);
    if (e != cudaSuccess) return cuda_error(e, "tensor-core scan launch (overflow)");
    e = launch_rerank_collected(d_base, static_cast<uint32_t>(ds), d_qn, d_fbq, m, d_rows2, d_cnt2, cap2, kcap, d_q2_thr,
                                d_rslots, o_idx, o_sim, o_cnt, d_ok2, s);
    if (e != cudaSuccess) return cuda_error(e, "rerank launch (overflow)");
    stats.kernel_launches += 6;
    // few enough (the usual case): in the page of the host's words
    uint32_t* ids = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(h_flags) + kWordBytes);
    uint32_t* ok = ids + kFewIds;
    if (m > kFewIds) {
        if ((st = grow_host(h_ids, cap_hids, m, "pinned buffer"))) return st;
        if ((st = grow_host(h_ok2, cap_hok2, m, "pinned buffer"))) return st;
        ids = h_ids;
        ok = h_ok2;
    }
    cudaMemcpyAsync(ids, d_fbq, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(ok, d_ok2, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
    if (w_err == d_err) cudaMemcpyAsync(h_flags, d_err, 2 * sizeof(uint64_t), cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(e, "search");
    if ((st = check_device_words())) return st;
    failed->clear();
    for (uint32_t i = 0; i < m; ++i)
        if (!ok[i]) failed->push_back(ids[i]);
    return NNDEX_OK;
}

int CudaIndex::rerun_exact_fp32(const std::vector<uint32_t>& qs, uint32_t kcap, uint64_t* o_idx, float* o_sim,
                                uint32_t* o_cnt, cudaStream_t s) {
    int st;
    const uint32_t mf = static_cast<uint32_t>(qs.size());
    if ((st = grow_device(d_qsub, cap_qsub, static_cast<uint64_t>(mf) * ds, "fallback buffer"))) return st;
    for (uint32_t i = 0; i < mf; ++i)
        cudaMemcpyAsync(d_qsub + static_cast<uint64_t>(i) * ds, d_qn + static_cast<uint64_t>(qs[i]) * ds,
                        ds * sizeof(float), cudaMemcpyDeviceToDevice, s);
    if ((st = grow_device(d_fb_idx, cap_fb_idx, static_cast<uint64_t>(mf) * kcap, "fallback buffer"))) return st;
    if ((st = grow_device(d_fb_sim, cap_fb_sim, static_cast<uint64_t>(mf) * kcap, "fallback buffer"))) return st;
    if ((st = grow_device(d_fb_cnt, cap_fb_cnt, mf, "fallback buffer"))) return st;
    const uint32_t path = stats.path;
    if ((st = enqueue_exact_fp32(d_qsub, mf, kcap, kcap, d_fb_idx, d_fb_sim, d_fb_cnt, s))) return st;
    stats.path = path;
    // (a small host batch's outputs are in pinned host memory)
    for (uint32_t i = 0; i < mf; ++i) {
        const uint64_t q = qs[i];
        cudaMemcpyAsync(o_idx + q * kcap, d_fb_idx + static_cast<uint64_t>(i) * kcap, kcap * sizeof(uint64_t),
                        cudaMemcpyDefault, s);
        cudaMemcpyAsync(o_sim + q * kcap, d_fb_sim + static_cast<uint64_t>(i) * kcap, kcap * sizeof(float),
                        cudaMemcpyDefault, s);
        if (o_cnt) cudaMemcpyAsync(o_cnt + q, d_fb_cnt + i, sizeof(uint32_t), cudaMemcpyDefault, s);
    }
    return wait_rerun(s);
}

// Waits for a re-run that followed its batch, and reads the status words again: a device wait that ran out
// in it has left part of the queries' results unwritten.
int CudaIndex::wait_rerun(cudaStream_t s) {
    if (take_injected_rerun_timeout()) launch_unanswered_wait(kInjectedWaitCycles, w_status, s);
    if (w_err == d_err) cudaMemcpyAsync(h_flags, d_err, 2 * sizeof(uint64_t), cudaMemcpyDeviceToHost, s);
    const cudaError_t e = cudaStreamSynchronize(s);
    return e != cudaSuccess ? cuda_error(e, "search") : check_device_words();
}

// K12 (small batches, FP32 precision): the TF32 candidate scan, the merge of each query's per-CTA
// candidates, and the exact rerank with its certificate into the outputs.
int CudaIndex::enqueue_tf32(uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt,
                            cudaStream_t s) {
    int st;
    const Tf32Plan plan = plan_tf32(n, kcap);
    if (!plan.kp) return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: no TF32 scan plan for k=%u", kcap);
    const uint32_t kp = plan.kp;
    const uint32_t ctas = static_cast<uint32_t>(sm_count);
    const uint64_t per_query = static_cast<uint64_t>(ctas) * plan.kp_cta;
    // the FP32 scan that re-runs uncertified queries shares the candidate workspace
    ScanPlan fb_plan;
    if (!plan_fallback(6, n, kcap, fb_plan))
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: no FP32 scan plan for k=%u", kcap);
    const uint64_t fb_per_query = static_cast<uint64_t>(fb_plan.ctas_per_group) * kcap;
    if ((st = grow_device(d_ws, cap_ws, std::max(per_query, fb_per_query) * n, "scan workspace"))) return st;
    if ((st = grow_device(d_fbq, cap_fbq, n, "fallback buffer"))) return st;
    if ((st = grow_device(d_cand_idx, cap_cand_idx, static_cast<uint64_t>(n) * kp, "tc workspace"))) return st;
    if ((st = grow_device(d_cand_sim, cap_cand_sim, static_cast<uint64_t>(n) * kp, "tc workspace"))) return st;
    if ((st = grow_device(d_cand_cnt, cap_cand_cnt, n, "tc workspace"))) return st;
    if ((st = grow_device(d_cert, cap_cert, n, "tc workspace"))) return st;
    if ((st = grow_device(d_kth, cap_kth, n, "tc workspace"))) return st;
    // The queries straight from the prepared buffer: rows past n read as zeros.
    CUtensorMap tmap_q;
    if (!encode_tmap_2d(&tmap_q, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d_qn, ds, n, ds * sizeof(float), 32, 16,
                        CU_TENSOR_MAP_SWIZZLE_128B))
        return set_error(NNDEX_ERR_CUDA, "cuda execution error: cuTensorMapEncodeTiled failed (queries, driver "
                                         "result %d)", last_encode_result());
    Tf32ScanArgs a;
    a.nq = n;
    a.nbox = static_cast<uint32_t>(ds / 32);
    a.ds = static_cast<uint32_t>(ds);
    a.rows = rows;
    a.kp = plan.kp_cta;
    a.cap = plan.cap;
    a.queries = d_qn;
    a.row_norms = d_tfnorm;
    a.c_norm = tf32_c_norm();
    a.evict_first = n <= 16;
    a.ws_keys = d_ws;
    a.floor_keys = d_floor;
    a.status = w_status;
    cudaEvent_t ev_a = nullptr;
    scan_event_begin(s, ev_a);
    cudaError_t e = launch_scan_tf32(tmap_f32, tmap_q, a, plan.stages, ctas, s);
    scan_event_end(s, ev_a);
    if (e != cudaSuccess) return cuda_error(e, "TF32 scan launch");
    MergeArgs m;
    m.ws_keys = d_ws;
    m.nq = n;
    m.per_query = per_query;
    m.k = kp;
    m.out_stride = kp;
    m.idx_out = d_cand_idx;
    m.sim_out = d_cand_sim;
    m.count_out = d_cand_cnt;
    if ((st = merge_workspace(per_query, n, kp, m, s))) return st;
    if ((e = launch_merge_topk(m, s)) != cudaSuccess) return cuda_error(e, "merge launch");
    RerankArgs r;
    r.base = d_base;
    r.ds = static_cast<uint32_t>(ds);
    r.queries = d_qn;
    r.cand_idx = d_cand_idx;
    r.cand_sim = d_cand_sim;
    r.cand_cnt = d_cand_cnt;
    r.nq = n;
    r.kp = kp;
    r.k = kcap;
    r.idx_out = o_idx;
    r.sim_out = o_sim;
    r.cnt_out = o_cnt;
    r.cert_out = d_cert;
    r.kth_out = d_kth;
    r.certify = true;
    r.floor_keys = d_floor;  // rows the CTAs' lists left out score below it
    r.fb_ids = d_fbq;
    r.fb_count = host_fallback ? h_fbn : d_fbn;
    if ((e = launch_rerank(r, s)) != cudaSuccess) return cuda_error(e, "rerank launch");
    // Uncertified queries re-run on the FP32 scan, on the device: the rerank listed them.
    if (!host_fallback) {
        if ((st = enqueue_fp32_fallback(fb_plan, n, kcap, o_idx, o_sim, o_cnt, s))) return st;
        fbn_stream = s;
        fbn_pending = true;
        stats.kernel_launches += 2;
    }
    last_tc_n = n;
    stats.kernel_launches += 3;
    stats.path = 6;
    stats.rerank_width = kp;
    stats.rows_scanned += rows * n;
    return NNDEX_OK;
}

// The FP32 scan that re-runs a TF32 batch's listed queries (path 6 or 7).
bool CudaIndex::plan_fallback(int path, uint32_t n, uint32_t kcap, ScanPlan& plan) const {
    if (!plan_scan_fp32(n, static_cast<uint32_t>(ds), kcap, rows, sm_count, smem_optin, plan)) return false;
    if (path == 7) {  // usually few queries: up to a CTA per SM for each group of 16, within 256 MB of keys
        const uint64_t per = std::min<uint64_t>(static_cast<uint64_t>(sm_count), (32ull << 20) / (static_cast<uint64_t>(n) * kcap));
        plan.ctas_per_group = static_cast<uint32_t>(std::max<uint64_t>(plan.ctas_per_group, per));
    }
    return true;
}

// A host-buffer batch's listed queries, their number read where the batch was waited for: the two
// launches, 8 us of a batch of 64 queries over 50k rows when none is listed, wait for one that is.
int CudaIndex::finish_tf32(int path, uint32_t n, uint32_t kcap) {
    const uint32_t listed = h_fbn[0] & 0xFFFFu;
    if (path == 7 && 2 * listed > n) tf32_rest = kTf32Rest;  // (settle_path)
    stats.fp32_fallback_queries += listed;
    stats.certified = stats.fp32_fallback_queries == 0 ? 1u : 0u;
    if (listed == 0) return NNDEX_OK;
    ScanPlan plan;
    if (!plan_fallback(path, n, kcap, plan))
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: no FP32 scan plan for k=%u", kcap);
    int st;
    if (path == 6) {  // counted in host memory
        const cudaError_t e = cudaMemcpyAsync(d_fbn, h_fbn, sizeof(uint32_t), cudaMemcpyHostToDevice, stream);
        if (e != cudaSuccess) return cuda_error(e, "fallback count");
    }
    if ((st = enqueue_fp32_fallback(plan, n, kcap, d_idx, d_sim, d_cnt, stream))) return st;
    stats.kernel_launches += 2;
    if (!mapped_io) cudaMemcpyAsync(h_res, d_res, res_bytes, cudaMemcpyDeviceToHost, stream);
    cudaEventRecord(ev1, stream);
    return wait_rerun(stream);
}

// The scan reads the listed queries' rows, the merge writes each result into the query's own output
// row; both return at once when none is listed.
int CudaIndex::enqueue_fp32_fallback(const ScanPlan& plan, uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim,
                                     uint32_t* o_cnt, cudaStream_t s) {
    const uint64_t per_query = static_cast<uint64_t>(plan.ctas_per_group) * kcap;
    ScanArgs fa;
    fa.tmap = &tmap_f32;
    fa.tmap_tile = &tmap_f32_176;
    fa.tmap_112 = &tmap_f32_112;
    fa.queries = d_qn;
    fa.nq = n;
    fa.dq = static_cast<uint32_t>(ds);
    fa.rows = rows;
    fa.k = kcap;
    fa.ws_keys = d_ws;
    fa.status = w_status;
    fa.live = d_fbn;
    fa.ids = d_fbq;
    cudaError_t e;
    if ((e = launch_scan_fp32(fa, plan, s)) != cudaSuccess) return cuda_error(e, "fallback scan launch");
    MergeArgs fm;
    fm.ws_keys = d_ws;
    fm.nq = n;
    fm.per_query = per_query;
    fm.k = kcap;
    fm.out_stride = kcap;
    fm.idx_out = o_idx;
    fm.sim_out = o_sim;
    fm.count_out = o_cnt;
    fm.live = d_fbn;
    fm.out_rows = d_fbq;
    int st;
    if ((st = merge_workspace(per_query, n, kcap, fm, s))) return st;
    if ((e = launch_merge_topk(fm, s)) != cudaSuccess) return cuda_error(e, "fallback merge launch");
    return NNDEX_OK;
}

int CudaIndex::grow_tf32_batch(const Tf32BatchPlan& plan, uint32_t n, uint32_t kcap, uint64_t fb_keys) {
    int st;
    const uint64_t words = plan.nranges * plan.gm_tiles * (256 / plan.group);
    if ((st = grow_device(d_q_resid, cap_q_resid, n, "query buffer"))) return st;
    if ((st = grow_device(d_cnt2, cap_cnt2, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_ids, cap_ids, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_cand_idx, cap_cand_idx, static_cast<uint64_t>(n) * plan.kp, "tc workspace"))) return st;
    if ((st = grow_device(d_cand_sim, cap_cand_sim, static_cast<uint64_t>(n) * plan.kp, "tc workspace"))) return st;
    if ((st = grow_device(d_cand_cnt, cap_cand_cnt, n, "tc workspace"))) return st;
    if ((st = grow_device(d_cert, cap_cert, n, "tc workspace"))) return st;
    if ((st = grow_device(d_kth, cap_kth, n, "tc workspace"))) return st;
    if ((st = grow_device(d_rows2, cap_rows2, static_cast<uint64_t>(n) * kSecondPassCap, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_ok2, cap_ok2, n, "pass-2 buffer"))) return st;
    if ((st = grow_device(d_rslots, cap_rslots, static_cast<uint64_t>(n) * rerank_chunks(kSecondPassCap) * kcap,
                          "pass-2 buffer")))
        return st;
    if ((st = grow_device(d_fbq, cap_fbq, n, "fallback buffer"))) return st;
    // last: the FP32 scan has its keys there too, and keeps what it has where one of the others fails
    return grow_device(d_ws, cap_ws, std::max((words + 1) / 2, fb_keys) * n, "scan workspace");
}

// The path a batch planned on the two-pass TF32 scan takes, decided before anything of it is enqueued. Without
// memory for the collections: the FP32 scan, whose workspace is far smaller. What the attempt had grown
// is given back, and the next batches do not try again (each try would free, allocate and drop
// every captured graph). Where most of a batch's collections overflowed (many rows within the bound of the k-th
// score: copies of a few rows, tight clusters), the FP32 scan had nearly all of the work to do again, and
// the next batches go to it likewise: 200k × 128, 8 distinct rows, 64 queries 306 us on the FP32 scan, 508
// through both; 256 queries 746 and 1,557.
int CudaIndex::settle_path(int* path, uint32_t n, uint32_t kcap) {
    if (*path != 7) return NNDEX_OK;
    // what the last device-buffer batch to finish said of itself (one may still be running)
    const uint32_t last = __atomic_exchange_n(h_fbn + 3, 0u, __ATOMIC_RELAXED);
    if (2 * (last & 0xFFFFu) > last >> 16) tf32_rest = kTf32Rest;
    if (tf32_rest) {
        --tf32_rest;
        *path = 1;
        return NNDEX_OK;
    }
    if (settled_n == n && settled_k == kcap && settled_host == host_fallback && settled_epoch == alloc_epoch())
        return NNDEX_OK;
    settled_n = 0;
    const Tf32BatchPlan plan = plan_tf32_batch(n, kcap);
    ScanPlan fb_plan;
    if (!plan.kp || !plan_fallback(7, n, kcap, fb_plan)) {
        *path = 1;
        return NNDEX_OK;
    }
    struct Grown {
        void** p;
        size_t* cap;
        size_t before;
    };
    auto at = [](auto& p, size_t& cap) { return Grown{reinterpret_cast<void**>(&p), &cap, cap}; };
    const Grown grown[] = {at(d_q_resid, cap_q_resid),   at(d_cnt2, cap_cnt2),         at(d_ids, cap_ids),
                           at(d_cand_idx, cap_cand_idx), at(d_cand_sim, cap_cand_sim), at(d_cand_cnt, cap_cand_cnt),
                           at(d_cert, cap_cert),         at(d_kth, cap_kth),           at(d_rows2, cap_rows2),
                           at(d_ok2, cap_ok2),           at(d_rslots, cap_rslots),     at(d_fbq, cap_fbq)};
    const int st = grow_tf32_batch(plan, n, kcap, static_cast<uint64_t>(fb_plan.ctas_per_group) * kcap);
    if (st == NNDEX_OK) {
        settled_n = n;
        settled_k = kcap;
        settled_host = host_fallback;
        settled_epoch = alloc_epoch();
    }
    if (st != NNDEX_ERR_OUT_OF_MEMORY) return st;
    cudaGetLastError();
    clear_error();
    for (const Grown& g : grown) {
        if (*g.cap == g.before) continue;
        release_raw(g.p);
        *g.cap = 0;
    }
    tf32_rest = kTf32Rest;
    *path = 1;
    return NNDEX_OK;
}

// Two-pass TF32 scan (FP32 indexes, 17 queries and more): K3's sampled pass 1 and collecting pass 2 on
// the FP32 base itself, read as TF32 by the tensor cores, with K12's bound at the rows' largest norms
// as every query's slack. The exact rerank sums in the FP32 scan's order, so rows and scores are the
// FP32 scan's bit for bit; a query whose collection overflows is re-run on it, on the device.
int CudaIndex::enqueue_tf32_batch(uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt,
                                  cudaStream_t s) {
    int st;
    const Tf32BatchPlan plan = plan_tf32_batch(n, kcap);
    ScanPlan fb_plan;
    if (!plan.kp || !plan_fallback(7, n, kcap, fb_plan))
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: no two-pass TF32 plan for k=%u", kcap);
    CUtensorMap tmap_q;  // the queries straight from the prepared buffer: rows past n read as zeros
    if (!encode_tmap_2d(&tmap_q, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d_qn, ds, n, ds * sizeof(float), 32, 128,
                        CU_TENSOR_MAP_SWIZZLE_128B))
        return set_error(NNDEX_ERR_CUDA, "cuda execution error: cuTensorMapEncodeTiled failed (queries, driver "
                                         "result %d)", last_encode_result());
    cudaError_t e = cudaSuccess;
    TcArgs a;
    a.tmap_q = &tmap_q;
    a.tmap_b = &tmap_f32_256;
    a.stages = plan.stages;
    a.stream_a = plan.stream_a;
    a.nranges = static_cast<uint32_t>(plan.nranges);
    a.p.nq = n;
    a.p.nchunks = static_cast<uint32_t>(ds / 32);
    a.p.rows = rows;
    a.p.range_rows = plan.range_rows;
    a.p.status = w_status;
    a.p.q_resid = d_q_resid;
    a.p.tile_stride = plan.stride;
    a.p.gm = reinterpret_cast<uint32_t*>(d_ws);
    a.p.gm_tiles = plan.gm_tiles;
    a.p.gm_group = plan.group;
    a.p.gm_span = plan.span;
    cudaEvent_t ev_a = nullptr;
    scan_event_begin(s, ev_a);
    e = launch_scan_tc(a, kTcTf32, 2, s);
    scan_event_end(s, ev_a);
    if (e != cudaSuccess) return cuda_error(e, "TF32 scan launch");
    TcThresholdArgs t;
    t.gm = a.p.gm;
    t.words = plan.nranges * plan.gm_tiles * (256 / plan.group);
    t.group = plan.group;
    t.tiles = plan.gm_tiles;
    t.span = plan.span;
    t.stride = plan.stride;
    t.parts = plan.nranges;
    t.range_rows = plan.range_rows;
    t.rows = rows;
    t.base = d_base;
    t.ds = static_cast<uint32_t>(ds);
    t.queries = d_qn;
    t.nq = n;
    t.kp = plan.kp;
    t.k = kcap;
    t.q_resid = d_q_resid;
    t.whole_slack = true;
    t.cand_idx = d_cand_idx;
    t.cand_sim = d_cand_sim;
    t.cand_cnt = d_cand_cnt;
    t.cert = d_cert;
    t.kth = d_kth;
    t.ids = d_ids;
    t.live = d_fbn + 1;
    if ((e = launch_threshold(t, s)) != cudaSuccess) return cuda_error(e, "threshold launch");
    uint64_t nranges = 0, range_rows = 0;
    tc_ranges(rows, (n + 127) / 128, nranges, range_rows, 256);
    a.nranges = static_cast<uint32_t>(nranges);
    a.p.range_rows = range_rows;
    a.p.tile_stride = 1;
    a.p.q_thr = d_kth;
    a.p.cand_rows = d_rows2;
    a.p.cand_cnt = d_cnt2;
    a.p.cap2 = kSecondPassCap;
    scan_event_begin(s, ev_a);
    e = launch_scan_tc(a, kTcTf32, 1, s);
    scan_event_end(s, ev_a);
    if (e != cudaSuccess) return cuda_error(e, "TF32 scan launch (pass 2)");
    e = launch_rerank_collected(d_base, static_cast<uint32_t>(ds), d_qn, d_ids, n, d_rows2, d_cnt2, kSecondPassCap, kcap,
                                d_kth, d_rslots, o_idx, o_sim, o_cnt, d_ok2, s, false, nullptr, nullptr, nullptr, nullptr,
                                nullptr, OverflowList{d_fbq, d_fbn, d_fbn + 3, host_fallback ? h_fbn : h_fbn + 3});
    if (e != cudaSuccess) return cuda_error(e, "rerank launch (pass 2)");
    if (!host_fallback) {
        if ((st = enqueue_fp32_fallback(fb_plan, n, kcap, o_idx, o_sim, o_cnt, s))) return st;
        fbn_stream = s;
        fbn_pending = true;
        stats.kernel_launches += 2;
    }
    last_tc_n = n;
    stats.kernel_launches += 5;
    stats.path = 7;
    stats.rerank_width = plan.kp;
    stats.pass1_tile_stride = plan.stride;
    stats.second_pass_queries += n;
    stats.rows_scanned += rows * n;
    return NNDEX_OK;
}

// The device-side fallback's count into the statistics (waits for its stream once).
int CudaIndex::fetch_fallback_stats() {
    if (!fbn_pending) return NNDEX_OK;
    cudaMemcpyAsync(h_fbn, fbn_pieces ? d_fbn_sum : d_fbn, sizeof(uint32_t), cudaMemcpyDeviceToHost, fbn_stream);
    const cudaError_t e = cudaStreamSynchronize(fbn_stream);
    if (e != cudaSuccess) return cuda_error(e, "fallback count");
    fbn_pending = false;
    stats.fp32_fallback_queries += h_fbn[0];
    stats.certified = stats.fp32_fallback_queries == 0 ? 1u : 0u;
    return NNDEX_OK;
}


int CudaIndex::tune_host(uint64_t n, uint64_t kcap, int mode, TunePlan* plan) {
    std::vector<TunePlan> cands = tune_candidates(n, kcap);
    const nndex_cuda_search_stats before = stats;
    const bool report = error_report;
    error_report = false;  // the timed runs record no score errors
    double best_ms = 0.0;
    int best = -1, last_err = NNDEX_OK;
    for (size_t c = 0; c < cands.size(); ++c) {
        double ms = 0.0;
        int cst = NNDEX_OK;
        for (int rep = 0; rep < 2 && cst == NNDEX_OK; ++rep) {
            forced_stride = cands[c].stride;
            forced_qb = cands[c].qb;
            const auto t0 = std::chrono::steady_clock::now();
            int path = cands[c].path;
            cst = settle_path(&path, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap));
            if (cst == NNDEX_OK) cst = enqueue_host_batch(n, kcap, mode, path);
            const cudaError_t e = cudaStreamSynchronize(stream);
            if (cst == NNDEX_OK && e != cudaSuccess) cst = cuda_error(e, "search");
            if (cst == NNDEX_OK) cst = check_device_words();
            if (cst == NNDEX_OK && (cands[c].path == 2 || cands[c].path == 3))
                cst = finish_tc(static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt, stream);
            if (cst == NNDEX_OK && cands[c].path == 5)
                cst = ivf_finish_tc(*this, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt,
                                    stream);
            if (cst == NNDEX_OK && host_fallback && (stats.path == 6 || stats.path == 7))
                cst = finish_tf32(path, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap));  // part of its time
            ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        }
        forced_stride = 0;
        forced_qb = 0;
        if (cst != NNDEX_OK) {
            last_err = cst;
            continue;
        }
        if (best < 0 || ms < best_ms) {
            best = static_cast<int>(c);
            best_ms = ms;
        }
    }
    error_report = report;
    if (best < 0) return last_err;
    clear_error();
    TuneEntry ent;
    ent.plan = cands[best];
    ent.ms = best_ms;
    ent.candidates = static_cast<uint32_t>(cands.size());
    tune_cache[tune_key(n, kcap)] = ent;
    stats = before;
    stats.tuned = 1;
    stats.tune_candidates = ent.candidates;
    *plan = ent.plan;
    return NNDEX_OK;
}

// Enqueues one batch of the host-buffer search on `stream` (the queries already in h_q): status
// resets, upload, prep, the path's scan and merge, and the downloads into the pinned buffers.
int CudaIndex::enqueue_host_batch(uint64_t n, uint64_t kcap, int mode, int path) {
    int st;
    h_flags[0] = h_flags[1] = 0;  // (a replay's are reset by run_host_batch)
    h_fbn[0] = 0;
    if (!mapped_io) cudaMemcpyAsync(d_qraw, h_q, n * dims * sizeof(float), cudaMemcpyHostToDevice, stream);
    if ((st = enqueue_prep_queries(mapped_io ? h_q : d_qraw, n, mode, path, stream))) return st;
    if (path == 4) {
        if ((st = ivf_search(*this, d_qn, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt,
                             stream)))
            return st;
    } else if (path == 5) {
        if ((st = ivf_search_tc(*this, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt,
                                stream)))
            return st;
    } else if (path == 1) {
        if ((st = enqueue_exact_fp32(d_qn, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap),
                                     static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt, stream)))
            return st;
    } else if (path == 6) {
        if ((st = enqueue_tf32(static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt, stream)))
            return st;
    } else if (path == 7) {
        if ((st = enqueue_tf32_batch(static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt, stream)))
            return st;
    } else {
        if ((st = enqueue_tc(path == 3, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt,
                             stream)))
            return st;
        if ((st = enqueue_tc_pass2(path == 3, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim,
                                   d_cnt, stream)))
            return st;
    }
    if (error_report)
        serr_record(static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt, stream);
    if (!mapped_io) cudaMemcpyAsync(h_res, d_res, res_bytes, cudaMemcpyDeviceToHost, stream);  // idx, sim, cnt
    return NNDEX_OK;
}

// The batch through a CUDA graph when one is cached for this shape, capturing it when the same
// shape came in the previous call (its buffers are then allocated, so nothing allocates during
// the capture); otherwise directly. No path needs a host decision in the middle of its batch: the
// FP32 scan (1), the tensor-core scans (2, 3, 5: pass 2 and its compaction run on the device; the
// rare FP32 re-run of an overflowed collection follows the batch), the IVF list scan (4) and the
// TF32 scans (6 and 7, the re-run of their listed queries likewise).
int CudaIndex::run_host_batch(uint64_t n, uint64_t kcap, int mode, int path) {
    const bool graphable = use_graphs && !scan_timing && !error_report && !sync_check_enabled() &&
                           path >= 1 && path <= 7 &&
                           !(graph_failed_paths & (1u << path));
    if (!graphable) return enqueue_host_batch(n, kcap, mode, path);
    const uint64_t epoch = alloc_epoch();
    const uint32_t np = static_cast<uint32_t>(ivf_scratch.nprobe);
    auto same = [&](const GraphEntry& g) {
        return g.path == path && g.mode == mode && g.n == n && g.kcap == kcap && g.nprobe == np;
    };
    for (size_t i = 0; i < graphs.size(); ++i) {
        if (!same(graphs[i])) continue;
        if (graphs[i].epoch != epoch) {
            cudaGraphExecDestroy(graphs[i].exec);
            graphs.erase(graphs.begin() + static_cast<long>(i));
            break;
        }
        h_flags[0] = h_flags[1] = 0;
        h_fbn[0] = 0;
        const cudaError_t e = cudaGraphLaunch(graphs[i].exec, stream);
        if (e != cudaSuccess) return cuda_error(e, "graph launch");
        // the capture's statistics: counters added to this call's, the rest as captured
        const nndex_cuda_search_stats acc = stats;
        stats = graphs[i].stats;
        stats.kernel_launches += acc.kernel_launches;
        stats.rows_scanned += acc.rows_scanned;
        stats.second_pass_queries += acc.second_pass_queries;
        stats.fp32_fallback_queries += acc.fp32_fallback_queries;
        stats.ivf_rows_streamed = acc.ivf_rows_streamed;
        stats.ivf_rows_union = acc.ivf_rows_union;
        count_launch(static_cast<uint32_t>(graphs[i].launches));
        stats.graph = 2;
        return NNDEX_OK;
    }
    if (!(same(graph_seen) && graph_seen.epoch == epoch)) {
        graph_seen = GraphEntry{path, mode, n, kcap, epoch, np};
        return enqueue_host_batch(n, kcap, mode, path);
    }
    // Second call of this shape with nothing reallocated in between: capture it.
    const nndex_cuda_search_stats before = stats;
    const uint64_t launches0 = kernel_launches_total();
    cudaError_t e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return enqueue_host_batch(n, kcap, mode, path);
    int st = enqueue_host_batch(n, kcap, mode, path);
    cudaGraph_t graph = nullptr;
    e = cudaStreamEndCapture(stream, &graph);
    cudaGraphExec_t exec = nullptr;
    if (st == NNDEX_OK && e == cudaSuccess && alloc_epoch() == epoch)
        e = cudaGraphInstantiate(&exec, graph, 0);
    else if (e == cudaSuccess)
        e = cudaErrorStreamCaptureInvalidated;
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();  // a failed capture leaves no sticky error
    if (e != cudaSuccess || !exec) {
        // run it the ordinary way; a path that cannot be captured is not tried again
        if (st == NNDEX_OK) graph_failed_paths |= 1u << path;
        stats = before;
        graph_seen = GraphEntry{};
        return enqueue_host_batch(n, kcap, mode, path);
    }
    GraphEntry g{path, mode, n, kcap, epoch, np};
    g.exec = exec;
    g.launches = kernel_launches_total() - launches0;
    g.stats = stats;  // counters as this batch's increments
    g.stats.kernel_launches -= before.kernel_launches;
    g.stats.rows_scanned -= before.rows_scanned;
    g.stats.second_pass_queries -= before.second_pass_queries;
    g.stats.fp32_fallback_queries -= before.fp32_fallback_queries;
    if (graphs.size() >= 8) {
        cudaGraphExecDestroy(graphs.front().exec);
        graphs.erase(graphs.begin());
    }
    graphs.push_back(g);
    if ((e = cudaGraphLaunch(exec, stream)) != cudaSuccess) return cuda_error(e, "graph launch");
    stats.graph = 1;
    return NNDEX_OK;
}

int CudaIndex::search_host(const float* queries, uint64_t nq, uint64_t k, int mode, uint64_t* idx_out,
                           float* sim_out, uint64_t* counts_out) {
    std::lock_guard<std::mutex> lock(mu);
    cudaSetDevice(device);
    begin_call();
    order_after_previous(stream);
    use_host_words();
    host_fallback = !error_report;  // a report records what the device-side re-run has written
    const uint64_t kcap = std::min<uint64_t>(k, rows);
    if (kcap > kMaxFusedK)
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: k=%llu above the fused top-k limit %u",
                         (unsigned long long)kcap, kMaxFusedK);
    int st0;
    if (error_report && (st0 = serr_begin(nq, kcap, stream))) return st0;
    cudaEventRecord(ev0, stream);
    const uint64_t chunk = kMaxBatchChunk;
    for (uint64_t q0 = 0; q0 < nq; q0 += chunk) {
        const uint64_t n = std::min<uint64_t>(chunk, nq - q0);
        int st;
        if ((st = ensure_query_capacity(n))) return st;
        if ((st = ensure_result_capacity(n, kcap))) return st;
        // Each copy of a small batch costs the GPU more (4 to 12 us with the gaps around it) than the
        // kernels' own reads and writes of pinned memory over PCIe: up to 64 KB each way, rows that
        // query prep reads once (prep.cu). One query against 50k × 128: 82 -> 57 us a call.
        mapped_io = !error_report && dims <= 1024 && n * dims * sizeof(float) <= kMappedIoBytes && res_bytes <= kMappedIoBytes;
        if (mapped_io) {
            d_idx = h_idx;
            d_sim = h_sim;
            d_cnt = h_cnt;
        }
        std::memcpy(h_q, queries + q0 * dims, n * dims * sizeof(float));
        bool measure = false;
        const TuneEntry* cached = nullptr;
        TunePlan plan = plan_for(n, kcap, &measure, &cached);
        if (measure) {
            if ((st = tune_host(n, kcap, mode, &plan))) return st;
        } else if (cached) {
            stats.tuned = 2;
            stats.tune_candidates = cached->candidates;
        }
        int path = plan.path;
        if ((st = settle_path(&path, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap)))) return st;
        serr_off = q0;
        forced_stride = plan.stride;
        forced_qb = plan.qb;
        st = run_host_batch(n, kcap, mode, path);
        forced_stride = 0;
        forced_qb = 0;
        if (st) return st;
        cudaEventRecord(ev1, stream);  // before the wait: the device time ends with the last batch
        cudaError_t e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) return cuda_error(e, "search");
        if ((st = check_device_words())) return st;
        if (path == 2 || path == 3 || path == 5) {
            // pass 2 ran on the device; a query whose collection overflowed is re-run now
            st = path == 5 ? ivf_finish_tc(*this, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim,
                                           d_cnt, stream)
                           : finish_tc(static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), d_idx, d_sim, d_cnt,
                                       stream);
            if (st) return st;
            if (tc_patched && !mapped_io) {
                cudaMemcpyAsync(h_res, d_res, res_bytes, cudaMemcpyDeviceToHost, stream);
                if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return cuda_error(e, "search");
            }
        }
        if (host_fallback && (stats.path == 6 || stats.path == 7) &&
            (st = finish_tf32(path, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap))))
            return st;
        if (path == 4) {
            stats.rows_scanned += ivf_scratch.h_probed[0];
            stats.ivf_rows_streamed += ivf_scratch.h_probed[1];
            stats.ivf_rows_union += ivf_scratch.h_probed[2];
        }
        std::memcpy(idx_out + q0 * kcap, h_idx, n * kcap * sizeof(uint64_t));
        std::memcpy(sim_out + q0 * kcap, h_sim, n * kcap * sizeof(float));
        if (counts_out)
            for (uint64_t i = 0; i < n; ++i) counts_out[q0 + i] = h_cnt[i];
    }
    done_stream = nullptr;  // every batch was waited for: nothing for a later call to be ordered after
    ms_pending = nq != 0;   // the device time between ev0 and ev1, read with the statistics
    return NNDEX_OK;
}

// One piece of a device-buffer search (≤ kMaxBatchChunk queries) on `path`: query prep, the path's
// scan and merge into the outputs. *synced is set when the path waited for the stream.
int CudaIndex::run_device_chunk(const float* dq, uint64_t n, uint64_t kcap, int path, uint64_t* oi, float* os,
                                uint32_t* oc, cudaStream_t s, bool* synced) {
    int st;
    if ((st = settle_path(&path, static_cast<uint32_t>(n), static_cast<uint32_t>(kcap)))) return st;
    if ((st = enqueue_prep_queries(dq, n, normalized ? 2 : 0, path, s))) return st;
    const uint32_t n32 = static_cast<uint32_t>(n), k32 = static_cast<uint32_t>(kcap);
    if (path == 4) return ivf_search(*this, d_qn, n32, k32, oi, os, oc, s);
    if (path == 5) {
        *synced = true;
        if ((st = ivf_search_tc(*this, n32, k32, oi, os, oc, s))) return st;
        const cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_error(e, "IVF search");
        if ((st = check_device_words())) return st;
        return ivf_finish_tc(*this, n32, k32, oi, os, oc, s);
    }
    if (path == 1) return enqueue_exact_fp32(d_qn, n32, k32, k32, oi, os, oc, s);
    if (path == 6) return enqueue_tf32(n32, k32, oi, os, oc, s);  // its fallback runs on the device
    if (path == 7) return enqueue_tf32_batch(n32, k32, oi, os, oc, s);
    // the overflowed collections' re-runs need the host: these paths synchronise
    *synced = true;
    if ((st = enqueue_tc(path == 3, n32, k32, oi, os, oc, s))) return st;
    if ((st = enqueue_tc_pass2(path == 3, n32, k32, oi, os, oc, s))) return st;
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(e, "search");
    if ((st = check_device_words())) return st;
    return finish_tc(n32, k32, oi, os, oc, s);
}

int CudaIndex::search_device(const float* d_queries, uint64_t nq, uint64_t k, uint64_t* d_idx_out,
                             float* d_sim_out, uint32_t* d_cnt_out, cudaStream_t s, int synchronize) {
    std::lock_guard<std::mutex> lock(mu);
    cudaSetDevice(device);
    begin_call();
    if (!s) s = cudaStreamLegacy;
    order_after_previous(s);
    const uint64_t kcap = std::min<uint64_t>(k, rows);
    int st;
    if ((st = ensure_query_capacity(std::min<uint64_t>(nq, kMaxBatchChunk)))) return st;
    if (error_report && (st = serr_begin(nq, kcap, s))) return st;
    use_device_words();
    host_fallback = false;
    cudaMemsetAsync(d_err, 0, 2 * sizeof(unsigned long long), s);
    // the pieces of a larger call share the word of the listed queries' number: it is added up after each
    fbn_pieces = nq > kMaxBatchChunk;
    if (fbn_pieces) cudaMemsetAsync(d_fbn_sum, 0, sizeof(uint32_t), s);
    bool synced = false, done = false;  // done: the last piece waited and its status words were clean
    for (uint64_t q0 = 0; q0 < nq; q0 += kMaxBatchChunk) {
        const uint64_t n = std::min<uint64_t>(kMaxBatchChunk, nq - q0);
        uint64_t* oi = d_idx_out + q0 * kcap;
        float* os = d_sim_out + q0 * kcap;
        uint32_t* oc = d_cnt_out ? d_cnt_out + q0 : nullptr;
        const float* dq = d_queries + q0 * dims;
        bool measure = false;
        const TuneEntry* cached = nullptr;
        TunePlan plan = plan_for(n, kcap, &measure, &cached);
        if (measure) {
            // the first batch of this shape: time every candidate plan on it, keep the fastest
            std::vector<TunePlan> cands = tune_candidates(n, kcap);
            const nndex_cuda_search_stats before = stats;
            double best_ms = 0.0;
            int best = -1, last_err = NNDEX_OK;
            for (size_t c = 0; c < cands.size(); ++c) {
                double ms = 0.0;
                int cst = NNDEX_OK;
                for (int rep = 0; rep < 2 && cst == NNDEX_OK; ++rep) {
                    forced_stride = cands[c].stride;
                    forced_qb = cands[c].qb;
                    bool sy = false;
                    const auto t0 = std::chrono::steady_clock::now();
                    cst = run_device_chunk(dq, n, kcap, cands[c].path, oi, os, oc, s, &sy);
                    const cudaError_t e = cudaStreamSynchronize(s);
                    if (cst == NNDEX_OK && e != cudaSuccess) cst = cuda_error(e, "search");
                    ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
                }
                forced_stride = 0;
                forced_qb = 0;
                if (cst != NNDEX_OK) {
                    last_err = cst;
                    continue;
                }
                if (best < 0 || ms < best_ms) {
                    best = static_cast<int>(c);
                    best_ms = ms;
                }
            }
            if (best < 0) return last_err;
            clear_error();
            TuneEntry ent;
            ent.plan = cands[best];
            ent.ms = best_ms;
            ent.candidates = static_cast<uint32_t>(cands.size());
            tune_cache[tune_key(n, kcap)] = ent;
            stats = before;
            stats.tuned = 1;
            stats.tune_candidates = ent.candidates;
            plan = ent.plan;
            synced = true;
        } else if (cached) {
            stats.tuned = 2;
            stats.tune_candidates = cached->candidates;
        }
        forced_stride = plan.stride;
        forced_qb = plan.qb;
        done = false;
        st = run_device_chunk(dq, n, kcap, plan.path, oi, os, oc, s, &done);
        forced_stride = 0;
        forced_qb = 0;
        if (st) return st;
        if (fbn_pieces && (stats.path == 6 || stats.path == 7)) launch_add_word(d_fbn_sum, d_fbn, s);
        synced |= done;
        if (error_report) {
            done = false;
            serr_off = q0;
            serr_record(static_cast<uint32_t>(n), static_cast<uint32_t>(kcap), oi, os, oc, s);
        }
    }
    if (done) {  // nothing was enqueued since
        mark_done(s);
        return NNDEX_OK;
    }
    if (synchronize || synced) {
        cudaMemcpyAsync(h_flags, d_err, 2 * sizeof(uint64_t), cudaMemcpyDeviceToHost, s);  // err, status
        mark_done(s);
        cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return cuda_error(e, "search");
        if (stats.path == 4) {
            stats.rows_scanned = ivf_scratch.h_probed[0];
            stats.ivf_rows_streamed = ivf_scratch.h_probed[1];
            stats.ivf_rows_union = ivf_scratch.h_probed[2];
        }
        return check_device_words();
    }
    mark_done(s);
    return NNDEX_OK;
}

// Score-error report: buffers for the call's nq × kcap results and a cleared accumulator.
int CudaIndex::serr_begin(uint64_t nq, uint64_t kcap, cudaStream_t s) {
    int st;
    if ((st = grow_device(d_serr, cap_serr, nq * kcap, "score-error buffer"))) return st;
    if (!d_serr_acc) {
        cudaError_t e;
        if ((e = cudaMalloc(&d_serr_acc, 3 * sizeof(unsigned long long))) != cudaSuccess ||
            (e = cudaMallocHost(&h_serr_acc, 3 * sizeof(unsigned long long))) != cudaSuccess)
            return cuda_error(e, "score-error buffer");
    }
    cudaMemsetAsync(d_serr_acc, 0, 3 * sizeof(unsigned long long), s);
    serr_nq = nq;
    serr_k = kcap;
    serr_off = 0;
    serr_stream = s;
    serr_pending = true;
    stats.score_errors = 1;
    return NNDEX_OK;
}

// The errors of one piece of the call (its first query at serr_off; queries normalised in d_qn).
void CudaIndex::serr_record(uint32_t n, uint32_t kcap, const uint64_t* idx, const float* sim, const uint32_t* cnt,
                            cudaStream_t s) {
    launch_score_errors(d_base, ds, d_qn, n, kcap, idx, sim, cnt, d_serr + serr_off * kcap, d_serr_acc, s);
    stats.kernel_launches += 1;
}

// Max and mean error into the statistics, once per call (waits for the call's stream).
int CudaIndex::serr_fetch_stats() {
    if (!serr_pending) return NNDEX_OK;
    cudaMemcpyAsync(h_serr_acc, d_serr_acc, 3 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, serr_stream);
    const cudaError_t e = cudaStreamSynchronize(serr_stream);
    if (e != cudaSuccess) return cuda_error(e, "score errors");
    serr_pending = false;
    double mx, sum;
    std::memcpy(&mx, &h_serr_acc[0], sizeof(double));
    std::memcpy(&sum, &h_serr_acc[1], sizeof(double));
    stats.max_score_error = mx;
    stats.mean_score_error = h_serr_acc[2] ? sum / static_cast<double>(h_serr_acc[2]) : 0.0;
    return NNDEX_OK;
}

// A new call's statistics: what was still to be read into the last one's is dropped with them (its stream may
// be gone by now).
void CudaIndex::begin_call() {
    stats = nndex_cuda_search_stats{};
    ms_pending = fbn_pending = serr_pending = false;
}

// The index's scratch buffers are shared by every call: work enqueued on one stream must not
// overlap work of an earlier call on another stream.
void CudaIndex::order_after_previous(cudaStream_t s) {
    if (done_ev && done_stream && done_stream != s) cudaStreamWaitEvent(s, done_ev, 0);
}
void CudaIndex::mark_done(cudaStream_t s) {
    if (!done_ev) cudaEventCreateWithFlags(&done_ev, cudaEventDisableTiming);
    cudaEventRecord(done_ev, s);
    done_stream = s;
}

int CudaIndex::stream_status() {
    std::lock_guard<std::mutex> lock(mu);
    cudaSetDevice(device);
    cudaStreamSynchronize(stream);
    cudaMemcpy(h_flags, d_err, 2 * sizeof(uint64_t), cudaMemcpyDeviceToHost);
    return check_device_words();
}

// ---- construction ----------------------------------------------------------------------------

static int select_device(int32_t requested, int& device) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDeviceCount");
    int d = requested < 0 ? 0 : requested;
    if (d >= n)
        return set_error(NNDEX_ERR_DEVICE_INDEX, "gpu device index %d is out of range (found %d adapter(s))", d, n);
    device = d;
    return NNDEX_OK;
}

// Construction in three steps (create_index below, and the streaming builder in builder.cu):
// index_begin allocates the device copies for rows × dims; index_prep_rows runs K1 (validate,
// normalise, pad, low-precision copies) over raw rows already on the device; index_finish checks
// the error word and completes the index (residual bounds, tensor maps, the IVF).
int index_begin(uint64_t rows, uint64_t dims, uint32_t flags, const nndex_cuda_opts* opts, CudaIndex** out) {
    *out = nullptr;
    if (rows >= (1ull << 31))
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: rows=%llu above the 2^31-1 row limit",
                         (unsigned long long)rows);
    const uint64_t dp = (dims + 7) / 8 * 8;
    if (dp > NNDEX_MAX_DIMS)
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: dims=%llu above the %u limit",
                         (unsigned long long)dims, NNDEX_MAX_DIMS);
    nndex_cuda_opts o{};
    o.device = -1;
    if (opts) o = *opts;
    int device = 0;
    int st = select_device(o.device, device);
    if (st) return st;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_error(e, "cudaSetDevice");
    // The no-allocation entry point's array is bound here, on the index's device: with lazy module
    // loading its memory is taken when its address is first looked up.
    if ((st = noalloc_bind(device))) return st;

    CudaIndex* ix = new (std::nothrow) CudaIndex();
    if (!ix) return set_error(NNDEX_ERR_OUT_OF_MEMORY, "cuda execution error: host allocation failed");
    ix->device = device;
    ix->rows = rows;
    ix->dims = dims;
    ix->dp = dp;
    ix->ds = (dims + 31) / 32 * 32;
    ix->rows_alloc = (rows + 255) / 256 * 256;  // whole 256-row tensor-core tiles
    ix->flags = flags;
    ix->precision = o.precision;
    ix->rerank_width = o.rerank_width;
    ix->normalized = (flags & NNDEX_FLAG_NORMALIZED) != 0;
    ix->approx = (flags & NNDEX_FLAG_APPROX) != 0;
    ix->opts = o;
    int value = 0;
    if ((e = cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device)) == cudaSuccess) ix->sm_count = value;
    if (e == cudaSuccess &&
        (e = cudaDeviceGetAttribute(&value, cudaDevAttrMaxSharedMemoryPerBlockOptin, device)) == cudaSuccess)
        ix->smem_optin = static_cast<size_t>(value);
    auto fail = [&](int code) {
        delete ix;
        return code;
    };
    if ((e = cudaStreamCreateWithFlags(&ix->stream, cudaStreamNonBlocking)) != cudaSuccess)
        return fail(cuda_error(e, "cudaStreamCreate"));
    cudaEventCreate(&ix->ev0);
    cudaEventCreate(&ix->ev1);
    if ((e = ix->alloc_words()) != cudaSuccess) return fail(cuda_error(e, "alloc"));
    // Everything on the device that lasts as long as the index, in one allocation: the driver takes 0.3
    // to 1 ms for each, and as much to free it. Low-precision scoring copies: K1 writes them in the same
    // pass as the rows.
    const bool bf16 = (flags & NNDEX_FLAG_BF16) != 0, fp8 = (flags & NNDEX_FLAG_FP8) != 0;
    if (bf16) ix->kb16 = (dims + 63) / 64 * 64;
    if (fp8) ix->kf8 = (dims + 127) / 128 * 128;
    auto carve = [&](Carver c, bool tf_norms) {
        c.take(ix->d_base, ix->rows_alloc * ix->ds);
        if (bf16) {
            c.take(ix->d_base_bf16, ix->rows_alloc * ix->kb16);
            c.take(ix->d_res16, rows);
        }
        if (fp8) {
            c.take(ix->d_base_fp8, ix->rows_alloc * ix->kf8);
            c.take(ix->d_row_scale, ix->rows_alloc);
            c.take(ix->d_tile_scale, ix->rows_alloc / 256);
            c.take(ix->d_res8, rows);
        }
        uint8_t* words = nullptr;
        c.take(words, CudaIndex::kWordBytes);
        ix->set_device_words(words);
        // Row norms of the TF32 scans' bounds (8 bytes per row, written by K1; the last entry their maxima).
        ix->d_tfnorm = nullptr;
        if (tf_norms) c.take(ix->d_tfnorm, rows + 1);
        return c.used;
    };
    bool tf_norms = true;
    e = cudaMalloc(&ix->d_mem, carve(Carver{}, true));
    if (e != cudaSuccess) {  // without the norms (no memory) FP32 batches take the FP32 scan
        cudaGetLastError();
        tf_norms = false;
        e = cudaMalloc(&ix->d_mem, carve(Carver{}, false));
    }
    if (e != cudaSuccess) {
        ix->d_mem = nullptr;
        return fail(cuda_error(e, bf16 || fp8 ? "base and low-precision copies allocation" : "base allocation"));
    }
    carve(Carver{static_cast<uint8_t*>(ix->d_mem)}, tf_norms);
    // What K1 does not write: the rows that fill the last tile, and the words.
    const uint64_t pad = ix->rows_alloc - rows;
    cudaMemsetAsync(ix->d_err, 0, CudaIndex::kWordBytes, ix->stream);
    if (tf_norms) cudaMemsetAsync(ix->d_tfnorm + rows, 0, sizeof(float2), ix->stream);
    if (pad) {
        cudaMemsetAsync(ix->d_base + rows * ix->ds, 0, pad * ix->ds * sizeof(float), ix->stream);
        if (bf16) cudaMemsetAsync(ix->d_base_bf16 + rows * ix->kb16, 0, pad * ix->kb16 * 2, ix->stream);
        if (fp8) {
            cudaMemsetAsync(ix->d_base_fp8 + rows * ix->kf8, 0, pad * ix->kf8, ix->stream);
            cudaMemsetAsync(ix->d_row_scale + rows, 0, pad * sizeof(float), ix->stream);
        }
    }
    ix->use_device_words();
    *out = ix;
    return NNDEX_OK;
}

void index_prep_rows(CudaIndex* ix, const float* d_src, uint64_t row0, uint64_t n) {
    PrepArgs p;
    p.src = d_src;
    p.rows = n;
    p.dims = static_cast<uint32_t>(ix->dims);
    p.row_base = row0;
    p.out = ix->d_base + row0 * ix->ds;
    p.out_stride = static_cast<uint32_t>(ix->ds);
    p.mode = ix->normalized ? 2 : 0;
    p.err = ix->d_err;
    p.sm_count = ix->sm_count;
    if (ix->d_tfnorm) {
        p.tf_norms = ix->d_tfnorm + row0;
        p.tf_max = ix->d_tfnorm + ix->rows;
    }
    if (ix->d_base_bf16) {
        p.out_bf16 = ix->d_base_bf16 + row0 * ix->kb16;
        p.bf16_stride = static_cast<uint32_t>(ix->kb16);
        p.resid_bf16 = ix->d_res16 + row0;
    }
    if (ix->d_base_fp8) {
        p.out_fp8 = ix->d_base_fp8 + row0 * ix->kf8;
        p.fp8_stride = static_cast<uint32_t>(ix->kf8);
        p.fp8_scale = ix->d_row_scale + row0;
        p.resid_fp8 = ix->d_res8 + row0;
    }
    launch_prep_rows(p, ix->stream);
}

int index_finish(CudaIndex* ix) {
    auto fail = [&](int code) {
        delete ix;
        return code;
    };
    cudaError_t e;
    cudaMemcpyAsync(&ix->h_flags[0], ix->d_err, sizeof(uint64_t), cudaMemcpyDeviceToHost, ix->stream);
    if ((e = cudaStreamSynchronize(ix->stream)) != cudaSuccess) return fail(cuda_error(e, "upload"));
    if (ix->h_flags[0] != 0) return fail(err_code(static_cast<int>(~ix->h_flags[0] & 0xFF)));
    if (ix->d_res16 || ix->d_res8) {
        // ε of the certificate: the largest residual norm ‖x − x̂‖ over the rows.
        unsigned int* d_max = ix->d_max;  // zero since index_begin
        if (ix->d_res16) launch_max_reduce(ix->d_res16, ix->rows, d_max, ix->stream);
        if (ix->d_res8) launch_max_reduce(ix->d_res8, ix->rows, d_max + 1, ix->stream);
        unsigned int hm[2] = {0, 0};
        cudaMemcpyAsync(hm, d_max, sizeof(hm), cudaMemcpyDeviceToHost, ix->stream);
        e = cudaStreamSynchronize(ix->stream);
        if (e != cudaSuccess) return fail(cuda_error(e, "residual reduction"));
        std::memcpy(&ix->eps_bf16, &hm[0], 4);
        std::memcpy(&ix->eps_fp8, &hm[1], 4);
    }
    if (!encode_tmap_2d(&ix->tmap_f32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ix->d_base, ix->ds, ix->rows_alloc,
                        ix->ds * sizeof(float), 32, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_tmap_2d(&ix->tmap_f32_176, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ix->d_base, ix->ds, ix->rows_alloc,
                        ix->ds * sizeof(float), 32, 176, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_tmap_2d(&ix->tmap_f32_112, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ix->d_base, ix->ds, ix->rows_alloc,
                        ix->ds * sizeof(float), 32, 112, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_tmap_2d(&ix->tmap_f32_256, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ix->d_base, ix->ds, ix->rows_alloc,
                        ix->ds * sizeof(float), 32, 256, CU_TENSOR_MAP_SWIZZLE_128B))
        return fail(set_error(NNDEX_ERR_CUDA, "cuda execution error: cuTensorMapEncodeTiled failed"));
    if (ix->d_base_bf16 &&
        (!encode_tmap_2d(&ix->tmap_bf16, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ix->d_base_bf16, ix->kb16,
                         ix->rows_alloc, ix->kb16 * 2, 64, 256, CU_TENSOR_MAP_SWIZZLE_128B) ||
         !encode_tmap_2d(&ix->tmap_bf16_h, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ix->d_base_bf16, ix->kb16,
                         ix->rows_alloc, ix->kb16 * 2, 64, 128, CU_TENSOR_MAP_SWIZZLE_128B)))
        return fail(set_error(NNDEX_ERR_CUDA, "cuda execution error: cuTensorMapEncodeTiled failed (BF16)"));
    if (ix->d_base_fp8 &&
        (!encode_tmap_2d(&ix->tmap_fp8, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, ix->d_base_fp8, ix->kf8, ix->rows_alloc,
                         ix->kf8, 128, 256, CU_TENSOR_MAP_SWIZZLE_128B) ||
         !encode_tmap_2d(&ix->tmap_fp8_h, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, ix->d_base_fp8, ix->kf8, ix->rows_alloc,
                         ix->kf8, 128, 128, CU_TENSOR_MAP_SWIZZLE_128B)))
        return fail(set_error(NNDEX_ERR_CUDA, "cuda execution error: cuTensorMapEncodeTiled failed (FP8)"));
    if (ix->d_row_scale) {
        // FP8 scan: the scale extremes of each 256-row tile (its epilogue's per-tile cut)
        launch_tile_scale(ix->d_row_scale, ix->rows, ix->rows_alloc / 256, ix->d_tile_scale, ix->stream);
    }
    if (ix->approx) {
        // src/approx.rs:46-100, built once at construction instead of on the first approx search.
        const int st = ivf_build(*ix);
        if (st != NNDEX_OK) return fail(st);
    }
    return NNDEX_OK;
}

int create_index(const float* matrix, bool on_device, uint64_t n_values, uint64_t rows, uint64_t dims,
                 uint32_t flags, const nndex_cuda_opts* opts, CudaIndex** out) {
    if (!out) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null output handle");
    *out = nullptr;
    if (!shape_ok(n_values, rows, dims)) return err_shape(rows, dims, n_values);
    if (!matrix) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null matrix");
    CudaIndex* ix = nullptr;
    int st = index_begin(rows, dims, flags, opts, &ix);
    if (st) return st;
    cudaError_t e = cudaSuccess;
    // K1: upload in chunks (≈32 MB of raw rows each: a pageable copy is as fast as with 256, and there is less to map and free), validate + normalise + pad on the device.
    if (on_device) {
        // The caller may still be writing the matrix on any stream: wait for the device first.
        if ((e = cudaDeviceSynchronize()) != cudaSuccess) {
            delete ix;
            return cuda_error(e, "cudaDeviceSynchronize");
        }
        index_prep_rows(ix, matrix, 0, rows);
    } else {
        uint64_t chunk_rows = std::max<uint64_t>(1, (32ull << 20) / (dims * sizeof(float)));
        chunk_rows = std::min(chunk_rows, rows);
        const int nbuf = chunk_rows < rows ? 2 : 1;
        float* d_raw[2] = {nullptr, nullptr};
        cudaEvent_t done[2];
        if ((e = cudaMalloc(&d_raw[0], nbuf * chunk_rows * dims * sizeof(float))) != cudaSuccess) {
            delete ix;
            return cuda_error(e, "upload staging");
        }
        d_raw[1] = d_raw[0] + (nbuf - 1) * chunk_rows * dims;
        for (int b = 0; b < 2; ++b) cudaEventCreateWithFlags(&done[b], cudaEventDisableTiming);
        int b = 0;
        for (uint64_t r0 = 0; r0 < rows; r0 += chunk_rows, b ^= 1) {
            const uint64_t n = std::min(chunk_rows, rows - r0);
            cudaEventSynchronize(done[b]);
            e = cudaMemcpyAsync(d_raw[b], matrix + r0 * dims, n * dims * sizeof(float), cudaMemcpyHostToDevice,
                                ix->stream);
            if (e != cudaSuccess) break;
            index_prep_rows(ix, d_raw[b], r0, n);
            cudaEventRecord(done[b], ix->stream);
        }
        cudaStreamSynchronize(ix->stream);
        cudaFree(d_raw[0]);
        for (int i = 0; i < 2; ++i) cudaEventDestroy(done[i]);
        if (e != cudaSuccess) {
            delete ix;
            return cuda_error(e, "upload");
        }
    }
    if ((st = index_finish(ix))) return st;
    *out = ix;
    return NNDEX_OK;
}

// A second handle on the same device-resident index: it shares the read-only data (base copies,
// tensor maps, the IVF) and owns its stream, status words and per-search scratch, so several can
// search concurrently (server slots).
int make_view(const CudaIndex& src, CudaIndex** out) {
    *out = nullptr;
    cudaSetDevice(src.device);
    CudaIndex* v = new (std::nothrow) CudaIndex();
    if (!v) return set_error(NNDEX_ERR_OUT_OF_MEMORY, "cuda execution error: host allocation failed");
    v->owns_base = false;
    v->device = src.device;
    v->sm_count = src.sm_count;
    v->smem_optin = src.smem_optin;
    v->rows = src.rows;
    v->rows_alloc = src.rows_alloc;
    v->dims = src.dims;
    v->dp = src.dp;
    v->ds = src.ds;
    v->flags = src.flags;
    v->normalized = src.normalized;
    v->approx = src.approx;
    v->opts = src.opts;
    v->d_base = src.d_base;
    v->tmap_f32 = src.tmap_f32;
    v->tmap_f32_176 = src.tmap_f32_176;
    v->tmap_f32_112 = src.tmap_f32_112;
    v->tmap_f32_256 = src.tmap_f32_256;
    v->precision = src.precision;
    v->kb16 = src.kb16;
    v->kf8 = src.kf8;
    v->d_base_bf16 = src.d_base_bf16;
    v->d_base_fp8 = src.d_base_fp8;
    v->d_row_scale = src.d_row_scale;
    v->d_tile_scale = src.d_tile_scale;
    v->eps_bf16 = src.eps_bf16;
    v->eps_fp8 = src.eps_fp8;
    v->d_res16 = src.d_res16;
    v->d_res8 = src.d_res8;
    v->d_tfnorm = src.d_tfnorm;
    v->tmap_bf16 = src.tmap_bf16;
    v->tmap_fp8 = src.tmap_fp8;
    v->tmap_bf16_h = src.tmap_bf16_h;
    v->tmap_fp8_h = src.tmap_fp8_h;
    v->rerank_width = src.rerank_width;
    v->tc_sample_stride = src.tc_sample_stride;
    // a view (a serving slot) never stops a batch to time plans: the source's measured plans, else
    // the rules
    v->tune_cache = src.tune_cache;
    v->autotune = src.autotune ? 2 : 0;
    v->ivf = src.ivf;
    v->ivf_scratch.nprobe = src.ivf_scratch.nprobe;
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&v->stream, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaEventCreate(&v->ev0)) != cudaSuccess || (e = cudaEventCreate(&v->ev1)) != cudaSuccess ||
        (e = cudaMalloc(&v->d_mem, CudaIndex::kWordBytes)) != cudaSuccess || (e = v->alloc_words()) != cudaSuccess) {
        delete v;
        return cuda_error(e, "index view");
    }
    v->set_device_words(static_cast<uint8_t*>(v->d_mem));
    cudaMemsetAsync(v->d_err, 0, CudaIndex::kWordBytes, v->stream);
    v->use_device_words();
    cudaStreamSynchronize(v->stream);
    *out = v;
    return NNDEX_OK;
}

int fill_devinfo(int device, nndex_cuda_devinfo* out) {
    cudaDeviceProp prop;
    cudaError_t e = cudaGetDeviceProperties(&prop, device);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetDeviceProperties");
    std::memset(out, 0, sizeof(*out));
    out->index = static_cast<uint64_t>(device);
    std::snprintf(out->name, sizeof(out->name), "%s", prop.name);
    std::snprintf(out->driver, sizeof(out->driver), "NVIDIA");
    int drv = 0, rt = 0;
    cudaDriverGetVersion(&drv);
    cudaRuntimeGetVersion(&rt);
    std::snprintf(out->driver_info, sizeof(out->driver_info), "CUDA driver %d.%d, runtime %d.%d", drv / 1000,
                  (drv % 1000) / 10, rt / 1000, (rt % 1000) / 10);
    std::snprintf(out->backend, sizeof(out->backend), "Cuda");
    std::snprintf(out->device_type, sizeof(out->device_type), prop.integrated ? "IntegratedGpu" : "DiscreteGpu");
    out->sm_count = prop.multiProcessorCount;
    out->cc_major = prop.major;
    out->cc_minor = prop.minor;
    out->hbm_bytes = prop.totalGlobalMem;
    out->l2_bytes = prop.l2CacheSize;
    return NNDEX_OK;
}

uint64_t launches() { return g_launches.load(); }

}  // namespace nndex

// =============================================================================================
// C ABI
// =============================================================================================
using namespace nndex;

extern "C" {

const char* nndex_cuda_last_error(void) { return last_error(); }

uint64_t nndex_cuda_kernel_launch_count(void) { return launches(); }

int nndex_cuda_set_scan_timing(nndex_cuda_index* index, int enable) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    std::lock_guard<std::mutex> lock(index->impl->mu);
    index->impl->scan_timing = enable != 0;
    return NNDEX_OK;
}

int nndex_cuda_scan_timing(nndex_cuda_index* index, double* total_ms, uint64_t* launches_out) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    cudaSetDevice(ix->device);
    double sum = 0.0;
    for (size_t i = 0; i < ix->scan_events_used; ++i) {
        cudaError_t e = cudaEventSynchronize(ix->scan_events[i].second);
        if (e != cudaSuccess) return cuda_error(e, "scan timing");
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, ix->scan_events[i].first, ix->scan_events[i].second);
        sum += ms;
    }
    if (total_ms) *total_ms = sum;
    if (launches_out) *launches_out = ix->scan_events_used;
    ix->scan_events_used = 0;
    return NNDEX_OK;
}

int nndex_cuda_list_devices(nndex_cuda_devinfo* out, uint32_t capacity, uint32_t* count) {
    clear_error();
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) n = 0;
    else if (e != cudaSuccess) return cuda_error(e, "cudaGetDeviceCount");
    if (count) *count = static_cast<uint32_t>(n);
    for (int d = 0; d < n && static_cast<uint32_t>(d) < capacity && out; ++d) {
        int st = fill_devinfo(d, &out[d]);
        if (st) return st;
    }
    return NNDEX_OK;
}

int nndex_cuda_info(const nndex_cuda_index* index, nndex_cuda_devinfo* out) {
    clear_error();
    if (!index || !out) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null argument");
    return fill_devinfo(index->impl->device, out);
}

int nndex_cuda_create(const float* host_matrix, uint64_t n_values, uint64_t rows, uint64_t dims, uint32_t flags,
                      const nndex_cuda_opts* opts, nndex_cuda_index** out) {
    clear_error();
    if (!out) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null output handle");
    CudaIndex* impl = nullptr;
    int st = create_index(host_matrix, false, n_values, rows, dims, flags, opts, &impl);
    if (st) return st;
    *out = new nndex_cuda_index{impl};
    return NNDEX_OK;
}

int nndex_cuda_create_from_device(const float* device_matrix, uint64_t n_values, uint64_t rows, uint64_t dims,
                                  uint32_t flags, const nndex_cuda_opts* opts, nndex_cuda_index** out) {
    clear_error();
    if (!out) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null output handle");
    CudaIndex* impl = nullptr;
    int st = create_index(device_matrix, true, n_values, rows, dims, flags, opts, &impl);
    if (st) return st;
    *out = new nndex_cuda_index{impl};
    return NNDEX_OK;
}

void nndex_cuda_destroy(nndex_cuda_index* index) {
    if (!index) return;
    delete index->impl;
    delete index;
}

int nndex_cuda_rows(const nndex_cuda_index* index, uint64_t* rows, uint64_t* dims, uint64_t* padded_dims) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    if (rows) *rows = index->impl->rows;
    if (dims) *dims = index->impl->dims;
    if (padded_dims) *padded_dims = index->impl->dp;
    return NNDEX_OK;
}

int nndex_cuda_search(nndex_cuda_index* index, const float* host_query, uint64_t query_len, uint64_t k,
                      uint64_t* idx_out, float* sim_out, uint64_t* count_out) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    // src/lib.rs:336-344: k == 0 first, then the dimensionality.
    if (k == 0) return err_topk();
    if (query_len != ix->dims) return err_query_dims(ix->dims, query_len);
    if (!host_query || !idx_out || !sim_out)
        return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null buffer");
    uint64_t cnt = 0;
    int st = ix->search_host(host_query, 1, k, ix->normalized ? 2 : 1, idx_out, sim_out, &cnt);
    if (st) return st;
    if (count_out) *count_out = cnt;
    return NNDEX_OK;
}

int nndex_cuda_search_batch(nndex_cuda_index* index, const float* host_queries, uint64_t n_values,
                            uint64_t query_rows, uint64_t k, uint64_t* idx_out, float* sim_out,
                            uint64_t* counts_out) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    // src/lib.rs:378-381: the shape first, then k == 0.
    if (!shape_ok(n_values, query_rows, ix->dims)) return err_shape(query_rows, ix->dims, n_values);
    if (k == 0) return err_topk();
    if (!host_queries || !idx_out || !sim_out)
        return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null buffer");
    return ix->search_host(host_queries, query_rows, k, ix->normalized ? 2 : 0, idx_out, sim_out, counts_out);
}

int nndex_cuda_search_batch_device(nndex_cuda_index* index, const float* dev_queries, uint64_t query_rows,
                                   uint64_t query_dims, uint64_t k, uint64_t* dev_idx_out, float* dev_sim_out,
                                   uint32_t* dev_counts_out, void* stream, int synchronize) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    if (query_rows == 0 || query_dims != ix->dims) return err_shape(query_rows, ix->dims, query_rows * query_dims);
    if (k == 0) return err_topk();
    if (!dev_queries || !dev_idx_out || !dev_sim_out)
        return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null buffer");
    if (std::min<uint64_t>(k, ix->rows) > kMaxFusedK)
        return set_error(NNDEX_ERR_UNSUPPORTED, "cuda execution error: k above the fused top-k limit %u",
                         kMaxFusedK);
    return ix->search_device(dev_queries, query_rows, k, dev_idx_out, dev_sim_out, dev_counts_out,
                             static_cast<cudaStream_t>(stream), synchronize);
}

int nndex_cuda_set_precision(nndex_cuda_index* index, uint32_t precision, uint32_t rerank_width) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    if (precision > NNDEX_PRECISION_FP8)
        return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: unknown precision %u", precision);
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    if ((precision == NNDEX_PRECISION_BF16 && !ix->d_base_bf16) || (precision == NNDEX_PRECISION_FP8 && !ix->d_base_fp8))
        return set_error(NNDEX_ERR_INVALID_ARGUMENT,
                         "cuda execution error: the index keeps no %s copy (create it with NNDEX_FLAG_%s)",
                         precision == NNDEX_PRECISION_BF16 ? "BF16" : "FP8",
                         precision == NNDEX_PRECISION_BF16 ? "BF16" : "FP8");
    ix->precision = precision;
    ix->drop_graphs();
    ix->rerank_width = rerank_width;
    return NNDEX_OK;
}

int nndex_cuda_last_candidates(nndex_cuda_index* index, uint64_t query_rows, uint64_t* idx_out, float* approx_out,
                               uint64_t capacity, uint32_t* kprime, float* eps_rows, uint32_t* certified_out) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    cudaSetDevice(ix->device);
    const uint32_t kp = ix->stats.rerank_width;
    if (kprime) *kprime = kp;
    if (eps_rows)
        *eps_rows = ix->stats.path == 3 ? ix->eps_fp8 : ix->stats.path >= 6 ? ix->tf32_eps() : ix->eps_bf16;
    if (kp == 0 || !ix->d_cand_idx) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: no low-precision search yet");
    if (ix->stats.path == 5)
        return set_error(NNDEX_ERR_UNSUPPORTED,
                         "cuda execution error: the IVF list scan's candidates are list positions, not exported");
    const uint64_t n = query_rows * kp;
    if (n > capacity || n > ix->cap_cand_idx)
        return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: candidate buffer too small");
    cudaError_t e = cudaDeviceSynchronize();  // the search may have run on any stream
    if (e == cudaSuccess && idx_out) e = cudaMemcpy(idx_out, ix->d_cand_idx, n * sizeof(uint64_t), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && approx_out) e = cudaMemcpy(approx_out, ix->d_cand_sim, n * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && certified_out) {
        if (query_rows > ix->last_tc_n)
            return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: more rows than the last batch");
        e = cudaMemcpy(certified_out, ix->d_cert, query_rows * sizeof(uint32_t), cudaMemcpyDeviceToHost);
    }
    if (e != cudaSuccess) return cuda_error(e, "candidates");
    return NNDEX_OK;
}

int nndex_cuda_stream_status(nndex_cuda_index* index) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    return index->impl->stream_status();
}

int nndex_cuda_last_search_stats(const nndex_cuda_index* index, nndex_cuda_search_stats* out) {
    clear_error();
    if (!index || !out) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null argument");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    if (ix->ms_pending) {
        cudaSetDevice(ix->device);
        float ms = 0.0f;
        if (cudaEventElapsedTime(&ms, ix->ev0, ix->ev1) != cudaSuccess) cudaGetLastError();
        ix->stats.device_ms = ms;
        ix->ms_pending = false;
    }
    if (ix->serr_pending || ix->fbn_pending) {
        cudaSetDevice(ix->device);
        int st = ix->serr_fetch_stats();
        if (!st) st = ix->fetch_fallback_stats();
        if (st) return st;
    }
    *out = ix->stats;
    return NNDEX_OK;
}

int nndex_cuda_set_error_report(nndex_cuda_index* index, int enable) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    cudaSetDevice(ix->device);
    cudaStreamSynchronize(ix->stream);
    ix->error_report = enable != 0;
    ix->drop_graphs();
    return NNDEX_OK;
}

int nndex_cuda_last_score_errors(nndex_cuda_index* index, uint64_t query_rows, uint64_t k, double* errors_out) {
    clear_error();
    if (!index || !errors_out) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null argument");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    const uint64_t kcap = std::min<uint64_t>(k, ix->rows);
    if (!ix->stats.score_errors || !ix->d_serr)
        return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: the last search recorded no score errors "
                                                     "(nndex_cuda_set_error_report)");
    if (query_rows != ix->serr_nq || kcap != ix->serr_k)
        return set_error(NNDEX_ERR_INVALID_ARGUMENT,
                         "cuda execution error: the last search had %llu queries at k=%llu, not %llu at k=%llu",
                         (unsigned long long)ix->serr_nq, (unsigned long long)ix->serr_k,
                         (unsigned long long)query_rows, (unsigned long long)kcap);
    cudaSetDevice(ix->device);
    cudaError_t e = cudaStreamSynchronize(ix->serr_stream);
    if (e == cudaSuccess)
        e = cudaMemcpy(errors_out, ix->d_serr, query_rows * kcap * sizeof(double), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_error(e, "score errors");
    return NNDEX_OK;
}

int nndex_cuda_ivf_layout(nndex_cuda_index* index, uint64_t* nlist_out, float* centroids, uint64_t* offsets,
                          uint64_t* original_indices, uint64_t* init_rows) {
    clear_error();
    if (!index || !nlist_out) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null argument");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    *nlist_out = 0;
    if (!ix->ivf) return NNDEX_OK;
    const IvfIndex& v = *ix->ivf;
    *nlist_out = v.nlist;
    cudaSetDevice(ix->device);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess && centroids)
        e = cudaMemcpy2D(centroids, ix->dp * sizeof(float), v.d_centroids, ix->ds * sizeof(float), ix->dp * sizeof(float),
                         v.nlist, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && original_indices) {
        std::vector<uint32_t> m(ix->rows);
        e = cudaMemcpy(m.data(), v.d_row_map, ix->rows * sizeof(uint32_t), cudaMemcpyDeviceToHost);
        for (uint64_t i = 0; i < ix->rows; ++i) original_indices[i] = m[i];
    }
    if (e != cudaSuccess) return cuda_error(e, "IVF layout copy");
    if (offsets) std::copy(v.h_offsets.begin(), v.h_offsets.end(), offsets);
    if (init_rows) std::copy(v.h_init_rows.begin(), v.h_init_rows.end(), init_rows);
    return NNDEX_OK;
}

int nndex_cuda_ivf_restore(nndex_cuda_index* index, uint64_t nlist, const float* centroids, const uint64_t* offsets,
                           const uint64_t* original_indices, const uint64_t* init_rows) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    if (!ix->owns_base)
        return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: cannot restore an IVF into a view");
    cudaSetDevice(ix->device);
    cudaError_t e = cudaDeviceSynchronize();  // searches in flight on any stream read the old IVF
    if (e != cudaSuccess) return cuda_error(e, "IVF restore");
    ix->drop_graphs();
    const int st = ivf_restore(*ix, nlist, centroids, offsets, original_indices, init_rows);
    if (st == NNDEX_OK) ix->approx = true;
    return st;
}

int nndex_cuda_base_checksum(nndex_cuda_index* index, uint64_t* checksum) {
    clear_error();
    if (!index || !checksum) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null argument");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    cudaSetDevice(ix->device);
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return cuda_error(e, "checksum");
    return base_checksum(*ix, checksum);
}

int nndex_cuda_set_graphs(nndex_cuda_index* index, int enable) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    cudaSetDevice(ix->device);
    cudaStreamSynchronize(ix->stream);
    ix->use_graphs = enable != 0;
    ix->drop_graphs();
    return NNDEX_OK;
}

int nndex_cuda_set_nprobe(nndex_cuda_index* index, uint32_t nprobe) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    std::lock_guard<std::mutex> lock(ix->mu);
    ix->opts.nprobe = nprobe;
    ix->ivf_scratch.nprobe = nprobe;
    ix->drop_graphs();
    return NNDEX_OK;
}

int nndex_cuda_ivf_stats_get(const nndex_cuda_index* index, nndex_cuda_ivf_stats* out) {
    clear_error();
    if (!index || !out) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null argument");
    const CudaIndex* ix = index->impl;
    *out = ix->ivf ? ix->ivf->stats : nndex_cuda_ivf_stats{};
    return NNDEX_OK;
}

int nndex_cuda_fp64_scores(nndex_cuda_index* index, const float* dev_queries_normalized, uint64_t query_rows,
                           const uint64_t* dev_pairs_query, const uint64_t* dev_pairs_row, uint64_t n,
                           double* dev_out) {
    clear_error();
    if (!index) return set_error(NNDEX_ERR_INVALID_ARGUMENT, "cuda execution error: null index");
    CudaIndex* ix = index->impl;
    (void)query_rows;
    std::lock_guard<std::mutex> lock(ix->mu);
    cudaSetDevice(ix->device);
    launch_fp64_pairs(ix->d_base, ix->ds, dev_queries_normalized, ix->dims, dev_pairs_query, dev_pairs_row, n, dev_out,
                      ix->stream);
    cudaError_t e = cudaStreamSynchronize(ix->stream);
    if (e != cudaSuccess) return cuda_error(e, "fp64 scores");
    return NNDEX_OK;
}

}  // extern "C"
