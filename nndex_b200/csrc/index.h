// index.h — the CUDA backend object behind the C ABI (one per NNdex built with the Cuda backend).
#pragma once

#include <memory>
#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>
#include <vector>

#include "internal.h"
#include "ivf.h"

namespace nndex {

// Queries handled per scan launch sequence; larger batches are processed in chunks.
constexpr uint64_t kMaxBatchChunk = 16384;
// Rows a pass-2 query may collect before it is re-run on the FP32 scan.
constexpr uint32_t kSecondPassCap = 8192;

// Host-buffer batches up to this size, queries and results each, run without copies.
constexpr size_t kMappedIoBytes = 64 << 10;

// FP32 batches take the two-pass TF32 scan where the FP32 scan's work, rows × queries × (stored dims + 64), is at
// least what the other's parts cost in the same measure (about 8 us per 1e8): its launches, beyond the FP32
// scan's; the rows that a query's threshold and rerank gather, k × dims; a query's blocks; and, of a base beyond
// L2, the rows that pass 1 reads besides. A host-buffer batch has two launches fewer (its listed queries wait
// until there is one) and waits in any case. Fitted to 1,600 batches of 1,000 to 1M rows × 32 to 1,536 dims, 17
// to 9,000 queries, k of 1 to 256 on normal rows: by this line 10 of them (host: 10) take more than 5 % longer
// than on the FP32 scan, 45 (26) could have been 5 % faster on the other side; by 2.5e8 multiply-adds alone 158
// took longer, up to 2.4 times as long. FP32 / two-pass scan, device buffers: 50k × 128, k = 10, 32 queries
// 52 / 57 us, 40 62 / 56, 256 189 / 66; 1,200 × 128, 1,628 queries 85 / 144; 20k × 512, 25 queries, k = 10 72 / 76,
// k = 256 83 / 132; 100k × 512, 32 queries, k = 10 154 / 116, k = 256 187 / 244; 1M × 768, 256 queries 11,285 / 857.
inline uint64_t tf32_batch_costs(uint64_t rows, uint64_t ds, uint64_t nq, uint64_t k, uint64_t stride, bool host) {
    const uint64_t again = rows * ds * sizeof(float) > (126ull << 20) ? rows * ds / stride * 8 : 0;
    return (host ? 80000000ull : 290000000ull) + k * ds * 10000 + nq * (host ? 300000 : 600000) + again;
}

// After a batch that the two-pass TF32 scan could not serve, this many go to the FP32 scan before it is tried
// again: a batch that tries in vain costs at most about twice the FP32 scan, so 3 % over 32.
constexpr uint32_t kTf32Rest = 31;

// Likewise the second pass 2 of overflowed collections (paths 2 and 3), where it cost more than the FP32 scan of
// what it served (CudaIndex::retry_paid). In vain for all of them: 458k × 11 in BF16, 32 tight clusters, 123 queries 2,023
// us without it, 2,353 with it; 9 queries over 316k × 175 in FP8 457 and 516.
constexpr uint32_t kTcRetryRest = 31;

// Incremented whenever a scratch or staging buffer of any index is (re)allocated: a captured
// CUDA graph is valid only while the epoch it was captured in lasts.
uint64_t alloc_epoch();
void bump_alloc_epoch();
// Host-side fault injection (tests): after `skip` scratch allocations that go ahead, the next n fail as out
// of memory.
void inject_alloc_failures(uint32_t skip, uint32_t n);
bool take_injected_alloc_failure();
// The next n re-runs of listed queries are followed by a device wait that runs out (tests).
void inject_rerun_timeouts(uint32_t n);
bool take_injected_rerun_timeout();
constexpr long long kInjectedWaitCycles = 2000000;  // about 1 ms
void launch_unanswered_wait(long long budget_cycles, uint32_t* status, cudaStream_t s);
// Scratch growth. By default a buffer that must grow is freed with cudaFree (which waits for the
// whole device) and reallocated with cudaMalloc. A serving slot instead grows its buffers in
// stream order on its own stream (cudaFreeAsync / cudaMallocAsync), so a slot meeting a larger
// batch does not wait for the batches the other slots are running; every buffer it grows is then
// stream-ordered memory from the start (a slot is a fresh view). The stream is per thread.
void set_scratch_stream(cudaStream_t s);
cudaStream_t scratch_stream();
// Frees `p` and allocates `bytes` (0 → 1) into it under the current thread's growth mode.
cudaError_t regrow_raw(void** p, size_t bytes);

int set_error(int code, const char* fmt, ...);
int last_encode_result();  // CUresult of this thread's last tensor-map encode
void clear_error();
const char* last_error();
int cuda_error(cudaError_t e, const char* what);
// NNdexError::ShapeMismatch (src/lib.rs:109-112).
int err_shape(uint64_t rows, uint64_t dims, uint64_t values);

struct CudaIndex {
    bool owns_base = true;    // false for a view (make_view): the device data belongs to another handle
    int device = 0;
    int sm_count = 148;
    size_t smem_optin = 232448;
    uint64_t rows = 0;        // stored rows
    uint64_t rows_alloc = 0;  // rows rounded up to 128 (zero rows beyond `rows`)
    uint64_t dims = 0;        // caller dimensionality
    uint64_t dp = 0;          // nndex padded_dims (multiple of 8, src/lib.rs:192)
    uint64_t ds = 0;          // device row stride: dims rounded up to 32 floats (one 128 B TMA slab)
    uint32_t flags = 0;
    bool normalized = false;
    bool approx = false;
    nndex_cuda_opts opts{};

    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t done_ev = nullptr;        // completion of the last call's device work
    cudaStream_t done_stream = nullptr;   // the stream it ran on
    bool ms_pending = false;              // stats.device_ms is still to be read from ev0 and ev1
    std::mutex mu;

    float* d_base = nullptr;  // rows_alloc × ds FP32, normalised, zero padded
    CUtensorMap tmap_f32{};
    CUtensorMap tmap_f32_176{};  // box {32 floats, 176 rows}: the 11-warp wide FP32 scan's tiles
    CUtensorMap tmap_f32_112{};  // box {32 floats, 112 rows}: the 7-warp wide FP32 scan's tiles
    CUtensorMap tmap_f32_256{};  // box {32 floats, 256 rows}: the two-pass TF32 scan's tiles

    // Low-precision scoring copies (NNDEX_FLAG_BF16 / NNDEX_FLAG_FP8), K3.
    uint32_t precision = NNDEX_PRECISION_AUTO;
    uint64_t kb16 = 0;                         // BF16 row length: dims rounded up to 64
    uint64_t kf8 = 0;                          // FP8 row length: dims rounded up to 128
    __nv_bfloat16* d_base_bf16 = nullptr;      // rows_alloc × kb16
    uint8_t* d_base_fp8 = nullptr;             // rows_alloc × kf8 (E4M3)
    float* d_row_scale = nullptr;              // rows_alloc: FP8 dequantisation scale per row
    float2* d_tile_scale = nullptr;            // rows_alloc / 256: FP8 {min, max} scale per 256-row tile
    float eps_bf16 = 0.0f, eps_fp8 = 0.0f;     // max row residual norm ‖x − x̂‖
    float* d_res16 = nullptr;                  // rows: ‖x − x̂‖ of the BF16 copy
    float* d_res8 = nullptr;                   // rows: ‖x − x̂‖ of the FP8 copy
    CUtensorMap tmap_bf16{}, tmap_fp8{};
    CUtensorMap tmap_bf16_h{}, tmap_fp8_h{};   // the same with 128-row boxes (two-block pass 2)
    // per-search buffers of the tensor-core path
    __nv_bfloat16* d_q_bf16 = nullptr;
    size_t cap_q_bf16 = 0;
    uint8_t* d_q_fp8 = nullptr;
    size_t cap_q_fp8 = 0;
    float* d_q_scale = nullptr;
    size_t cap_q_scale = 0;
    float2* d_tfnorm = nullptr;  // TF32 scans: per row {‖x‖, ‖x − tf32_head(x)‖}, rounded up; the last
                                 // entry (index rows) holds the largest of each (shared by views)
    float* d_q_resid = nullptr;
    size_t cap_q_resid = 0;
    unsigned long long* d_thr = nullptr;
    size_t cap_thr = 0;
    uint64_t* d_cand_idx = nullptr;
    size_t cap_cand_idx = 0;
    float* d_cand_sim = nullptr;
    size_t cap_cand_sim = 0;
    uint32_t* d_cand_cnt = nullptr;
    size_t cap_cand_cnt = 0;
    uint32_t* d_cert = nullptr;
    size_t cap_cert = 0;
    uint32_t* h_cert = nullptr;
    size_t cap_hcert = 0;
    float* d_qsub = nullptr;  // FP32 queries re-run after a failed certificate
    size_t cap_qsub = 0;
    uint64_t* d_fb_idx = nullptr;  // their FP32 results before they move to the query's slots
    size_t cap_fb_idx = 0;
    float* d_fb_sim = nullptr;
    size_t cap_fb_sim = 0;
    uint32_t* d_fb_cnt = nullptr;
    size_t cap_fb_cnt = 0;
    uint32_t last_tc_n = 0;  // queries of the last tensor-core batch (diagnostics)
    uint32_t tc_sample_stride = 1;  // pass-1 tile stride by the certification rule (1 = full pass 1)
    uint32_t forced_stride = 0;     // the tuned plan's pass-1 tile stride for the current batch (0 = rule)
    uint32_t forced_qb = 0;         // the tuned plan's pass-2 query blocks per CTA (0 = rule)
    uint32_t last_tc_stride = 1;
    bool tc_patched = false;  // after the batch, results of some queries were written again
    bool tc_groups = false;  // the batch's pass 1 wrote group maxima (every query goes to pass 2)
    float* d_kth = nullptr;  // pass 1: exact k-th score per query
    unsigned long long* d_floor = nullptr;  // TF32 scan: per query, a key its k'-th candidate reaches
    size_t cap_floor = 0;
    uint64_t* d_rslots = nullptr;  // pass 2: each rerank work item's best k keys
    size_t cap_rslots = 0;
    size_t cap_kth = 0;
    // pass 2 (threshold collection) buffers
    uint32_t* d_ids = nullptr;
    size_t cap_ids = 0;
    uint8_t* d_q2_lp = nullptr;
    size_t cap_q2_lp = 0;
    float* d_q2_resid = nullptr;
    size_t cap_q2_resid = 0;
    float* d_q2_scale = nullptr;
    size_t cap_q2_scale = 0;
    float* d_q2_thr = nullptr;
    size_t cap_q2_thr = 0;
    uint32_t* d_rows2 = nullptr;
    size_t cap_rows2 = 0;
    uint32_t* d_cnt2 = nullptr;
    size_t cap_cnt2 = 0;
    uint32_t* d_ok2 = nullptr;
    size_t cap_ok2 = 0;
    uint32_t* h_ids = nullptr;
    size_t cap_hids = 0;
    uint32_t* h_ok2 = nullptr;
    size_t cap_hok2 = 0;
    uint32_t rerank_width = 0;  // k′ override (0 = autotuned)


    // per-search buffers (grown on demand)
    float* d_qraw = nullptr;
    size_t cap_qraw = 0;
    float* d_qn = nullptr;
    size_t cap_qn = 0;
    uint64_t* d_ws = nullptr;
    size_t cap_ws = 0;
    // Results of the host-buffer search: idx (n·k u64), sim (n·k f32) and cnt (n u32) laid out
    // back to back in one device buffer and one pinned buffer, so a single copy downloads them
    // (ensure_result_capacity sets the three views for the batch's shape).
    uint8_t* d_res = nullptr;
    size_t cap_res = 0;
    uint8_t* h_res = nullptr;
    size_t cap_hres = 0;
    uint64_t* d_idx = nullptr;
    float* d_sim = nullptr;
    uint32_t* d_cnt = nullptr;
    uint64_t* h_idx = nullptr;
    float* h_sim = nullptr;
    uint32_t* h_cnt = nullptr;
    size_t res_bytes = 0;        // bytes of the current batch's results
    // The device's words and the host's, the first kWordBytes laid out alike. Status words (d_status = the word after
    // d_err), zero when clean: of construction and of device-buffer searches, read back with one copy
    // into h_flags. Then the counts of a two-pass batch (d_fbn, h_fbn), and construction's maxima (device)
    // or an IVF search's counts (host).
    static constexpr size_t kWordBytes = 256, kFbnAt = 64, kMaxAt = 128, kProbedAt = 192;
    // The host's go on with two lists of an overflowed batch's queries, kFewIds each.
    static constexpr size_t kHostWordBytes = 4096;
    static constexpr uint32_t kFewIds = (kHostWordBytes - kWordBytes) / 8;
    // Behind them: the queries and the results of batches up to kMappedIoBytes each.
    static constexpr size_t kHostBytes = kHostWordBytes + 2 * kMappedIoBytes;
    bool in_words(const void* p) const {
        const uint8_t *at = static_cast<const uint8_t*>(p), *words = reinterpret_cast<const uint8_t*>(h_flags);
        return words && at >= words && at < words + kHostBytes;
    }
    void* d_mem = nullptr;  // the allocation with the device's words, and an owner's rows and copies
    unsigned long long* d_err = nullptr;
    uint32_t* d_status = nullptr;
    unsigned int* d_max = nullptr;  // the largest residual norms of the BF16 and FP8 copies
    void set_device_words(uint8_t* at) {
        d_err = reinterpret_cast<unsigned long long*>(at);
        d_status = reinterpret_cast<uint32_t*>(d_err + 1);
        d_fbn = reinterpret_cast<uint32_t*>(at + kFbnAt);
        d_fbn_sum = d_fbn + kFbnBytes / sizeof(uint32_t);
        d_max = reinterpret_cast<unsigned int*>(at + kMaxAt);
    }
    void* words_page = nullptr;  // the registered memory with the host's words, if they are in such
    cudaError_t alloc_words();
    void free_words();
    // The current call's: d_err / d_status, or for a host-buffer search h_flags itself (the kernels
    // only ever write them on an error, and a host-buffer search waits before it reads them).
    unsigned long long* w_err = nullptr;
    uint32_t* w_status = nullptr;
    void use_device_words() {
        w_err = d_err;
        w_status = d_status;
    }
    void use_host_words() {
        w_err = reinterpret_cast<unsigned long long*>(h_flags);
        w_status = reinterpret_cast<uint32_t*>(h_flags + 1);
    }
    // Small host-buffer batches: the kernels read the queries from the pinned buffer and write the
    // results into the pinned buffer (d_idx, d_sim, d_cnt are its views), so that no copy runs.
    bool mapped_io = false;
    float* h_q = nullptr;
    size_t cap_hq = 0;
    uint64_t* h_flags = nullptr;

    // split cross-CTA merge (merge_topk_kernel with several blocks per query)
    uint64_t* d_part_keys = nullptr;
    size_t cap_part_keys = 0;
    uint32_t* d_part_done = nullptr;
    size_t cap_part_done = 0;
    int merge_workspace(uint64_t per_query, uint32_t nq, uint32_t k, MergeArgs& m, cudaStream_t s);

    nndex_cuda_search_stats stats{};
    std::shared_ptr<const IvfIndex> ivf;  // approximate mode (NNDEX_FLAG_APPROX), built at creation
    IvfScratch ivf_scratch;
    int approx_override = -1;   // -1: the index's mode; 0: exact; 1: approx (server batches)

    // CUDA graphs of the host-buffer search: the whole per-batch sequence (status resets, query
    // upload, query prep, scan, merge, result downloads) works on buffers this index owns, so a
    // shape seen twice in a row is captured once and replayed as one launch. A graph is dropped
    // when any scratch buffer has been reallocated since its capture (alloc_epoch()).
    struct GraphEntry {
        int path = 0, mode = 0;
        uint64_t n = 0, kcap = 0, epoch = 0;
        uint32_t nprobe = 0;  // the IVF scan's probe count at capture (0: chosen per batch)
        cudaGraphExec_t exec = nullptr;
        nndex_cuda_search_stats stats{};
        uint64_t launches = 0;
    };
    std::vector<GraphEntry> graphs;
    GraphEntry graph_seen;          // the last shape run without a graph (capture candidate)
    bool use_graphs = true;
    uint32_t graph_failed_paths = 0;  // paths whose capture failed (not tried again)
    void drop_graphs();

    // per-result score errors (nndex_cuda_set_error_report): |result − FP64 score| per result of the
    // last call, and {max as double bits, sum, count} for its statistics
    bool error_report = false;
    double* d_serr = nullptr;
    size_t cap_serr = 0;
    unsigned long long* d_serr_acc = nullptr;
    unsigned long long* h_serr_acc = nullptr;  // pinned copy of d_serr_acc
    uint64_t serr_nq = 0, serr_k = 0, serr_off = 0;  // the last call's shape; the current piece's first query
    cudaStream_t serr_stream = nullptr;
    bool serr_pending = false;  // statistics not yet read back
    int serr_begin(uint64_t nq, uint64_t kcap, cudaStream_t s);
    void serr_record(uint32_t n, uint32_t kcap, const uint64_t* idx, const float* sim, const uint32_t* cnt,
                     cudaStream_t s);
    int serr_fetch_stats();

    // Counters a device-side certificate fallback leaves on the device ({queries re-run on the FP32
    // scan, spare}), read back with the statistics.
    uint32_t* d_fbq = nullptr;  // the re-run queries' indices
    size_t cap_fbq = 0;
    // {TF32 re-runs, TC pass-2 queries, TC pass-2 overflows, a ticket (host: what the last device-buffer batch of
    // the two-pass TF32 scan listed, OverflowList), rows pass 2 collected (64 bits)}
    static constexpr size_t kFbnBytes = 6 * sizeof(uint32_t);
    uint32_t* d_fbn = nullptr;
    uint32_t* d_fbn_sum = nullptr;  // the word behind them: the first one summed over a device-buffer call's pieces
    bool fbn_pieces = false;        // the pending count is that sum
    uint32_t* h_fbn = nullptr;  // pinned copy
    uint32_t* d_tcfail = nullptr;  // TC pass 2: positions (in d_ids) of the queries whose collection overflowed
    size_t cap_tcfail = 0;
    uint64_t h_fbn_rows() const { return *reinterpret_cast<const unsigned long long*>(h_fbn + 4); }
    cudaStream_t fbn_stream = nullptr;
    bool fbn_pending = false;
    // A TF32 batch of a host-buffer search: its listed queries are counted in h_fbn, and re-run after the
    // batch where there are any (finish_tf32).
    bool host_fallback = false;
    bool plan_fallback(int path, uint32_t n, uint32_t kcap, ScanPlan& plan) const;
    int finish_tf32(int path, uint32_t n, uint32_t kcap);
    int fetch_fallback_stats();

    // scan-kernel timing (roofline reports)
    bool scan_timing = false;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> scan_events;
    size_t scan_events_used = 0;
    void scan_event_begin(cudaStream_t s, cudaEvent_t& a);
    void scan_event_end(cudaStream_t s, cudaEvent_t a);

    ~CudaIndex();
    int ensure_query_capacity(uint64_t nq);
    int ensure_result_capacity(uint64_t nq, uint64_t kcap);
    int enqueue_query_prep(uint64_t nq, int mode, cudaStream_t s);
    int enqueue_exact_fp32(const float* d_queries, uint32_t nq, uint32_t k, uint32_t out_stride, uint64_t* o_idx,
                           float* o_sim, uint32_t* o_cnt, cudaStream_t s);
    int check_device_words();
    int search_host(const float* queries, uint64_t nq, uint64_t k, int mode, uint64_t* idx_out, float* sim_out,
                    uint64_t* counts_out);
    int search_device(const float* d_queries, uint64_t nq, uint64_t k, uint64_t* d_idx_out, float* d_sim_out,
                      uint32_t* d_cnt_out, cudaStream_t s, int synchronize);
    int run_device_chunk(const float* dq, uint64_t n, uint64_t kcap, int path, uint64_t* oi, float* os,
                         uint32_t* oc, cudaStream_t s, bool* synced);
    // Path choice for a batch: 1 = FP32 scan, 2 = BF16 tensor-core scan, 3 = FP8 tensor-core scan,
    // 6 = TF32 tensor-core candidate scan + exact FP32 rerank (small batches of an FP32 index),
    // 7 = two-pass TF32 tensor-core scan + exact FP32 rerank (its larger batches).
    int choose_path(uint64_t nq, uint64_t kcap) const;
    // K12's plan for k results: candidates per query and CTA (0: no plan), buffer, ring depth.
    struct Tf32Plan {
        uint32_t kp = 0;      // candidates per query after the merge (k′)
        uint32_t kp_cta = 0;  // candidates per query and CTA
        uint32_t cap = 0, stages = 0;
    };
    Tf32Plan plan_tf32(uint64_t nq, uint64_t kcap) const;
    // The two-pass TF32 scan's plan for larger FP32 batches (kp 0: none): sampled pass 1 with group
    // maxima, then a collecting pass.
    struct Tf32BatchPlan {
        uint32_t kp = 0;  // candidates per query whose exact scores give T
        uint32_t stride = 1, group = 0, span = 1, gm_tiles = 0;
        uint64_t nranges = 0, range_rows = 0;  // pass 1
        uint32_t stages = 0;
        bool stream_a = false;
    };
    Tf32BatchPlan plan_tf32_batch(uint64_t nq, uint64_t kcap) const;
    float tf32_c_norm() const;  // C of K12's bound: ε = ‖q‖(‖d_x‖ + C‖x‖) + ‖d_q‖(‖x‖ + ‖d_x‖)
    float tf32_eps() const;     // the largest ε for unit rows and queries
    int ivf_path(uint64_t nq, uint64_t kcap) const;

    // Autotuner (autotune.cu): for each batch shape (exact or IVF, queries and k rounded up to
    // powers of two, nprobe, precision) the plans that return the same results are timed once on
    // the first batch of that shape, and the fastest is kept. A plan is a path and, for the
    // tensor-core scan, its pass-1 tile stride.
    struct TunePlan {
        int path = 0;
        uint32_t stride = 0;  // 0 = the certification rule
        uint32_t qb = 0;      // tensor-core pass 2: query blocks per CTA (1 or 2; 0 = the rule)
    };
    struct TuneEntry {
        TunePlan plan;
        double ms = 0.0;      // its wall time per batch when measured
        uint32_t candidates = 0;
        mutable uint64_t fit_nq = 0, fit_k = 0;  // the batch (and rerank width) that `fits` was last asked for
        mutable uint32_t fit_width = 0;
        mutable bool fit_host = false, fits = false;
    };
    int autotune = 1;  // 0 = rules only, 1 = measure once per shape, 2 = cached plans, else rules
    std::map<uint64_t, TuneEntry> tune_cache;
    uint64_t tune_key(uint64_t nq, uint64_t kcap) const;
    std::vector<TunePlan> tune_candidates(uint64_t nq, uint64_t kcap) const;
    TunePlan rule_plan(uint64_t nq, uint64_t kcap) const;
    // The plan for a batch: cached (*cached), or by the rules; *measure when the tuner should time the
    // candidates on this batch first.
    TunePlan plan_for(uint64_t nq, uint64_t kcap, bool* measure, const TuneEntry** cached) const;
    const TuneEntry* cached_plan(uint64_t nq, uint64_t kcap) const;
    bool plan_fits(const TunePlan& plan, uint64_t nq, uint64_t kcap) const;
    bool tc_fits(uint64_t kcap, bool fp8) const;
    // The first host-buffer batch of a shape: every candidate plan timed on it (the queries in h_q).
    int tune_host(uint64_t n, uint64_t kcap, int mode, TunePlan* plan);
    struct TcPlan {
        uint32_t kp = 0;        // pass-1 heap entries per query (0: no plan)
        uint32_t stages = 0;    // ring depth
        bool stream_a = false;  // query slabs staged per ring stage instead of resident
    };
    TcPlan plan_tc(uint64_t kcap, bool fp8) const;
    // k′ of a sampled pass 1 with group maxima: 2k (at least 32) unless set, 0 where the threshold
    // kernel's lists do not hold it.
    uint32_t group_candidates(uint64_t kcap) const;
    uint32_t tc_chunks(bool fp8) const;
    void plan_groups(uint32_t nqb, uint32_t kp, uint32_t stride, uint32_t& group, uint32_t& span, uint32_t& gm_tiles,
                     uint64_t& nranges, uint64_t& range_rows) const;
    void tc_ranges(uint64_t scan_rows, uint32_t nqb, uint64_t& nranges, uint64_t& range_rows,
                   uint64_t min_rows = 2048) const;
    void fill_tc_params(bool fp8, uint32_t n, uint64_t range_rows, TcParams& p) const;
    int encode_query_tmap(bool fp8, void* buf, uint32_t n, CUtensorMap* map) const;
    int enqueue_prep_queries(const float* d_raw, uint64_t n, int mode, int path, cudaStream_t s);
    int enqueue_tc(bool fp8, uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt,
                   cudaStream_t s);
    // Pass 2 of a tensor-core batch on the device, after enqueue_tc: the uncertified queries are
    // compacted and gathered, their rows collected against T and reranked, and the queries whose
    // collection overflowed compacted for the host (d_fbn[1..2], d_tcfail). No host round trip.
    int enqueue_tc_pass2(bool fp8, uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt,
                         cudaStream_t s);
    // Once the stream has completed a tensor-core batch (h_fbn read back with it): statistics, the
    // pass-1 stride rule, and the FP32 re-run of any query whose collection overflowed (device
    // outputs patched in place; synchronises the stream again only then).
    BatchReport batch_report() const;
    int finish_tc(uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt, cudaStream_t s);
    // Pass 2 once more for the m queries whose collection overflowed (positions in d_ids: d_tcfail),
    // against the T of the rows they did collect; the ones that overflow again are left in *failed.
    // batches whose overflowed queries still go to the FP32 scan without it, where they are at most so many (more
    // of them share the pass, and may be worth it)
    uint32_t tc_retry_rest = 0, tc_retry_rest_m = 0;
    bool retry_paid(uint32_t m, uint32_t failed) const;
    int overflowed_queries(uint32_t m, uint32_t failed_n, cudaStream_t s, std::vector<uint32_t>* failed);
    int retry_tc_pass2(bool fp8, uint32_t m, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt,
                       cudaStream_t s, std::vector<uint32_t>* failed);
    int enqueue_tf32(uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt, cudaStream_t s);
    int enqueue_tf32_batch(uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim, uint32_t* o_cnt, cudaStream_t s);
    int settle_path(int* path, uint32_t n, uint32_t kcap);
    // the shape that settle_path last had the buffers for; they are still there while nothing was reallocated
    uint32_t settled_n = 0, settled_k = 0;
    uint64_t settled_epoch = 0;
    bool settled_host = false;
    uint32_t tf32_rest = 0;  // batches of the two-pass TF32 scan's shapes still to go to the FP32 scan
    int grow_tf32_batch(const Tf32BatchPlan& plan, uint32_t n, uint32_t kcap, uint64_t fb_keys);
    // The FP32 scan of the d_fbn[0] queries listed in d_fbq, into their own output rows (enqueued
    // for up to n of them; its launches return at once when there are none).
    int enqueue_fp32_fallback(const ScanPlan& plan, uint32_t n, uint32_t kcap, uint64_t* o_idx, float* o_sim,
                              uint32_t* o_cnt, cudaStream_t s);
    // The FP32 scan for the listed queries (rows of d_qn), written into their output slots.
    int wait_rerun(cudaStream_t s);
    int rerun_exact_fp32(const std::vector<uint32_t>& qs, uint32_t kcap, uint64_t* o_idx, float* o_sim,
                         uint32_t* o_cnt, cudaStream_t s);
    int stream_status();
    int enqueue_host_batch(uint64_t n, uint64_t kcap, int mode, int path);
    int run_host_batch(uint64_t n, uint64_t kcap, int mode, int path);
    // Approximate mode with an IVF that gives a speedup (src/approx.rs:35-37 provides_speedup).
    bool uses_ivf() const {
        const bool want = approx_override < 0 ? approx : approx_override == 1;
        return want && ivf && rows >= 256 && ivf->nlist >= 4;
    }
    void order_after_previous(cudaStream_t s);
    void mark_done(cudaStream_t s);
    void begin_call();
};

// Tensor map of a row-major matrix (inner × outer elements), 2-D boxes.
bool encode_tmap_2d(CUtensorMap* map, CUtensorMapDataType dtype, uint32_t elem_bytes, const void* base,
                    uint64_t inner, uint64_t outer, uint64_t row_stride_bytes, uint32_t box_inner,
                    uint32_t box_outer, CUtensorMapSwizzle swizzle);
int make_view(const CudaIndex& src, CudaIndex** out);
int index_begin(uint64_t rows, uint64_t dims, uint32_t flags, const nndex_cuda_opts* opts, CudaIndex** out);
void index_prep_rows(CudaIndex* ix, const float* d_src, uint64_t row0, uint64_t n);
int index_finish(CudaIndex* ix);  // deletes ix on failure
int search_device_noalloc(CudaIndex* ix, const float* d_queries, uint64_t nq, uint64_t k, uint64_t* d_idx_out,
                          float* d_sim_out, uint32_t* d_cnt_out, cudaStream_t s);
// Looks up the no-allocation array's address on `device` (current), which loads the module that
// holds it; index creation calls it so that the array's memory is taken then, not at a first search.
int noalloc_bind(int device);

}  // namespace nndex

// The opaque handle behind the C ABI.
struct nndex_cuda_index {
    nndex::CudaIndex* impl;
};
