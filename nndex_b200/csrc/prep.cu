// prep.cu — K1: validation, normalisation and padding on the device.
//
// Replaces nndex's host-side preparation (src/lib.rs:239-244, 404-411, 461-599): one warp per
// row reads the raw f32 row once (coalesced), checks finiteness, computes the squared norm,
// rejects zero-norm rows, scales by 1/sqrt(norm_sq) and writes the zero-padded row. The same
// pass emits the BF16 copy and the FP8-E4M3 copy (per-row scale) for the low-precision scans,
// the per-row quantisation residual norms the exactness certificate uses, and the norms of the TF32
// scans' bounds.
//
// Arithmetic follows the reference exactly:
//   * dims >= 16 (src/lib.rs:472-473, 525-532): norm_sq = (f32) Σ (f64)x² (simsimd's FP64
//     accumulation), non-finite norm_sq → NonFiniteInput;
//   * dims < 16 and single queries (src/lib.rs:536-545, 558-569): sequential FP32 sum of x*x with
//     a per-element finite check, no fused multiply-add;
//   * norm_sq <= f32::EPSILON → ZeroNorm; inv = sqrt(norm_sq).recip() (two IEEE roundings),
//     x * inv in FP32 (src/lib.rs:547-551).
// Errors: the lowest failing row wins (the reference's row order): the complement of (row << 8) | code
// in a 64-bit word that starts at zero, reduced with atomicMax.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "common.cuh"
#include "internal.h"

namespace nndex {

constexpr uint32_t kErrNonFinite = NNDEX_ERR_NON_FINITE;
constexpr uint32_t kErrZeroNorm = NNDEX_ERR_ZERO_NORM;

NNDEX_DEVICE_INLINE void report_row_error(unsigned long long* err, uint64_t row, uint32_t code) {
    atomicMax(err, ~static_cast<unsigned long long>((row << 8) | code));
}

// mode: 0 = normalize_rows semantics, 1 = normalize_vector semantics (sequential FP32),
//       2 = already normalised (finite check + pad only).
// One warp per row, lane L holding the values L, L + 32, … . kR > 0: the row (at most 32·kR values) is
// read once, into registers; kR = 0: any length, re-read (from L1 / L2) for each output. The sums of a
// row run in the same order either way. The sequential FP32 norm takes its squares from the lanes one
// by one (a chain of adds on one lane that loaded each value itself took 10.4 us for a 128-value
// query; 2.1 us now). The optional outputs (low-precision copies, TF32 norms and slack, words to
// zero for the kernels behind this one) are skipped when null. Bound by HBM on whole matrices.
template <int kR>
__global__ void __launch_bounds__(256) prep_rows_kernel(const PrepArgs a) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    const uint32_t dims = a.dims;
#pragma unroll
    for (int z = 0; z < 2; ++z)
        for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < a.zero_words[z];
             i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
            a.zero[z][i] = 0;
    uint32_t max_n = 0, max_d = 0;  // TF32: the largest ‖x‖ and ‖x − tf32_head(x)‖, as bits
    for (uint64_t r = warp; r < a.rows; r += nwarps) {
        const float* s = a.src + r * dims;
        const uint64_t grow = a.row_base + r;
        float v[kR > 0 ? kR : 1];
        if constexpr (kR > 0) {
#pragma unroll
            for (int u = 0; u < kR; ++u) {
                const uint32_t i = lane + 32u * u;
                v[u] = i < dims ? s[i] : 0.0f;
            }
        }
        // f(value, index) over this lane's values below n, in order
        auto each = [&](uint32_t n, auto&& f) {
            if constexpr (kR > 0) {
#pragma unroll
                for (int u = 0; u < kR; ++u)
                    if (lane + 32u * u < n) f(v[u], lane + 32u * u);
            } else {
                for (uint32_t i = lane; i < n; i += 32) f(s[i], i);
            }
        };
        float inv = 1.0f;
        int code = 0;
        bool fin = true;
        if (a.mode == 2) {
            each(dims, [&](float x, uint32_t) { fin &= isfinite(x) != 0; });
            if (!__all_sync(0xffffffffu, fin)) code = kErrNonFinite;
        } else {
            float norm_sq = 0.0f;
            if (a.mode == 1 || dims < 16) {
                each(dims, [&](float x, uint32_t) { fin &= isfinite(x) != 0; });
                if (!__all_sync(0xffffffffu, fin)) {
                    code = kErrNonFinite;
                } else {
                    // squares and sums rounded one by one, in index order (every lane adds the same)
                    auto chunk = [&](float x, uint32_t n) {
                        const float sq = __fmul_rn(x, x);
                        if (n == 32) {
#pragma unroll
                            for (uint32_t j = 0; j < 32; ++j) norm_sq = __fadd_rn(norm_sq, __shfl_sync(0xffffffffu, sq, j));
                        } else {
                            for (uint32_t j = 0; j < n; ++j) norm_sq = __fadd_rn(norm_sq, __shfl_sync(0xffffffffu, sq, j));
                        }
                    };
                    if constexpr (kR > 0) {
#pragma unroll
                        for (int u = 0; u < kR; ++u)
                            if (32u * u < dims) chunk(v[u], dims - 32u * u < 32 ? dims - 32u * u : 32u);
                    } else {
                        for (uint32_t i0 = 0; i0 < dims; i0 += 32)
                            chunk(i0 + lane < dims ? s[i0 + lane] : 0.0f, dims - i0 < 32 ? dims - i0 : 32u);
                    }
                }
            } else {
                double acc = 0.0;
                each(dims, [&](float x, uint32_t) {
                    const double d = static_cast<double>(x);
                    acc = fma(d, d, acc);  // exact product of two f32 values in f64
                });
#pragma unroll
                for (int o2 = 16; o2 > 0; o2 >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
                norm_sq = static_cast<float>(acc);
                if (!isfinite(norm_sq)) code = kErrNonFinite;
            }
            if (code == 0 && norm_sq <= 1.1920929e-07f) code = kErrZeroNorm;
            if (code == 0) inv = __frcp_rn(__fsqrt_rn(norm_sq));
        }
        if (code != 0 && lane == 0) report_row_error(a.err, grow, code);
        // The normalised (or copied) row, zero padded to its stride. A rejected row is written as zeros
        // (residuals 0, FP8 scale 1): its batch fails, but the scans that were already queued behind
        // this kernel then read defined values, not stale memory.
        const uint32_t live_dims = code == 0 ? dims : 0u;
        auto value = [&](float x, uint32_t i) {
            return i < live_dims ? (a.mode == 2 ? x : __fmul_rn(x, inv)) : 0.0f;
        };
        if constexpr (kR > 0) {
#pragma unroll
            for (int u = 0; u < kR; ++u) v[u] = value(v[u], lane + 32u * u);
        }
        // f(output value, index) over this lane's values below n ≥ dims
        auto each_out = [&](uint32_t n, auto&& f) {
            if constexpr (kR > 0) {
#pragma unroll
                for (int u = 0; u < kR; ++u)
                    if (lane + 32u * u < n) f(v[u], lane + 32u * u);
                for (uint32_t i = lane + 32u * kR; i < n; i += 32) f(0.0f, i);
            } else {
                for (uint32_t i = lane; i < n; i += 32) f(i < live_dims ? value(s[i], i) : 0.0f, i);
            }
        };
        float* o = a.out + r * a.out_stride;
        float amax = 0.0f;
        each_out(a.out_stride, [&](float x, uint32_t i) {
            o[i] = x;
            amax = fmaxf(amax, fabsf(x));
        });
        if (a.out_bf16 != nullptr) {
            float rb = 0.0f;
            __nv_bfloat16* ob = a.out_bf16 + r * a.bf16_stride;
            each_out(a.bf16_stride, [&](float x, uint32_t i) {
                const __nv_bfloat16 b = __float2bfloat16_rn(x);
                ob[i] = b;
                const float d = x - __bfloat162float(b);
                rb = fmaf(d, d, rb);
            });
#pragma unroll
            for (int o2 = 16; o2 > 0; o2 >>= 1) rb += __shfl_xor_sync(0xffffffffu, rb, o2);
            if (lane == 0 && a.resid_bf16 != nullptr) a.resid_bf16[r] = sqrtf(rb);
        }
        if (a.out_fp8 != nullptr) {
#pragma unroll
            for (int o2 = 16; o2 > 0; o2 >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o2));
            // Per-row scale maps the row's max magnitude to 448 (E4M3's largest finite value).
            const float scale = amax > 0.0f ? amax / 448.0f : 1.0f;
            const float inv_scale = 1.0f / scale;
            float rf = 0.0f;
            uint8_t* of = a.out_fp8 + r * a.fp8_stride;
            each_out(a.fp8_stride, [&](float x, uint32_t i) {
                const __nv_fp8_e4m3 q(x * inv_scale);
                of[i] = q.__x;
                const float d = x - static_cast<float>(q) * scale;
                rf = fmaf(d, d, rf);
            });
#pragma unroll
            for (int o2 = 16; o2 > 0; o2 >>= 1) rf += __shfl_xor_sync(0xffffffffu, rf, o2);
            if (lane == 0) {
                a.fp8_scale[r] = scale;
                if (a.resid_fp8 != nullptr) a.resid_fp8[r] = sqrtf(rf);
            }
        }
        if (a.tf_norms != nullptr || a.tf_slack != nullptr) {
            // ‖x‖ and ‖x − tf32_head(x)‖ of the stored row, FP64 sums rounded up
            double s1 = 0.0, s2 = 0.0;
            each_out(a.out_stride, [&](float x, uint32_t) {
                const float d = x - tf32_head(x);  // exact: x and its head share the exponent
                s1 += static_cast<double>(x) * x;
                s2 += static_cast<double>(d) * d;
            });
#pragma unroll
            for (int o2 = 16; o2 > 0; o2 >>= 1) {
                s1 += __shfl_xor_sync(0xffffffffu, s1, o2);
                s2 += __shfl_xor_sync(0xffffffffu, s2, o2);
            }
            const float2 n = make_float2(__double2float_ru(__dsqrt_ru(s1)), __double2float_ru(__dsqrt_ru(s2)));
            if (a.tf_norms != nullptr) {
                if (lane == 0) a.tf_norms[r] = n;
                max_n = max(max_n, __float_as_uint(n.x));  // a NaN compares above every finite norm
                max_d = max(max_d, __float_as_uint(n.y));
            } else if (lane == 0) {
                // A query of the two-pass TF32 scan: the bound of |s̃ − the FP32 scan's score| over all
                // rows. The last term: products and operands below FP32's normal range, which either
                // side may flush.
                const float2 x = *a.tf_row_max;
                const float e = (n.x * fmaf(a.tf_c_norm, x.x, x.y) + n.y * (x.x + x.y)) * 1.01f +
                                (n.x + x.x + 1.0f) * static_cast<float>(a.out_stride) * 7.5231638e-37f;
                // every partial sum of a score stays below ‖q‖‖x‖: far from overflow, or no bound is
                // trusted and the query's collection counts as overflowed from the start
                const bool trusted = n.x * x.x <= 1e37f && e <= 1e37f;
                a.tf_slack[r] = trusted ? e : INFINITY;
                a.tf_collected[r] = trusted ? 0u : a.tf_over;
            }
        }
    }
    if (a.tf_norms != nullptr && lane == 0 && warp < a.rows) {
        atomicMax(reinterpret_cast<unsigned int*>(&a.tf_max->x), max_n);
        atomicMax(reinterpret_cast<unsigned int*>(&a.tf_max->y), max_d);
    }
}

void launch_prep_rows(const PrepArgs& a, cudaStream_t stream) {
    if (a.rows == 0) return;
    // few rows (queries): a warp per block, over as many SMs as there are
    const unsigned threads = a.rows <= static_cast<uint64_t>(a.sm_count) * 2 ? 32u : 256u;
    uint64_t blocks = (a.rows * 32 + threads - 1) / threads;
    const uint64_t max_blocks = static_cast<uint64_t>(a.sm_count) * 16;
    if (blocks > max_blocks) blocks = max_blocks;
    const unsigned g = static_cast<unsigned>(blocks);
    if (a.dims <= 128) prep_rows_kernel<4><<<g, threads, 0, stream>>>(a);
    else if (a.dims <= 256) prep_rows_kernel<8><<<g, threads, 0, stream>>>(a);
    else if (a.dims <= 512) prep_rows_kernel<16><<<g, threads, 0, stream>>>(a);
    else if (a.dims <= 1024) prep_rows_kernel<32><<<g, threads, 0, stream>>>(a);
    else prep_rows_kernel<0><<<g, threads, 0, stream>>>(a);
    count_launch();
}

}  // namespace nndex
