// fp32 rows -> split form (see gemm_f16.cu): the weights of an engine when it is built, activations that no kernel of this library
// produces so, and the bounds of a weight and its bias.
//
// A file of its own: a program's first launch of a kernel loads what was compiled with it, and an engine whose products all run on
// the few-row kernel needs nothing else of gemm_f16.cu (first engine of a process, 16 layers of width 512: 24.5 ms with the conversion in that file, 15.9 here).
#include <algorithm>

#include "../runtime.hpp"
#include "sm100.cuh"

namespace fxf {
namespace {

using namespace sm100;

// One block per row (rows are hundreds to thousands of floats): maximum, then the two planes from the row's second read,
// which hits L1 / L2.  l1_out (weights): the row's L1 norm.  Bound: bytes (8 read and written per element).
// MODE 0: f16 planes; 1: bf16 plane only.
template <int MODE>
__global__ void __launch_bounds__(128) split_rows_kernel(const float* __restrict__ x, int64_t ld, uint16_t* __restrict__ planes, int64_t plane, float* __restrict__ inv_out,
                                                         float* __restrict__ amax_out, float* __restrict__ l1_out, int64_t M, int K) {
    __shared__ float red[8];
    grid_dep_launch();
    grid_dep_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t r = blockIdx.x; r < M; r += gridDim.x) {
        const float* xr = x + r * ld;
        uint16_t* hr = planes + r * K;
        const bool vec = (reinterpret_cast<uintptr_t>(xr) & 15) == 0;
        auto load = [&](int k) {
            return vec ? *reinterpret_cast<const float4*>(xr + k) : make_float4(xr[k], xr[k + 1], xr[k + 2], xr[k + 3]);
        };
        if (MODE == 1) {
            for (int k = threadIdx.x * 4; k < K; k += 512) {
                const float4 v = load(k);
                *reinterpret_cast<uint2*>(hr + k) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
            }
            continue;
        }
        float m = 0.f, l1 = 0.f;
        for (int k = threadIdx.x * 4; k < K; k += 512) {
            const float4 v = load(k);
            m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
            l1 += (fabsf(v.x) + fabsf(v.y)) + (fabsf(v.z) + fabsf(v.w));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            l1 += __shfl_xor_sync(0xffffffffu, l1, o);
        }
        __syncthreads();
        if (lane == 0) { red[warp] = m; red[4 + warp] = l1; }
        __syncthreads();
        m = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
        float scale, inv;
        split_scale(m, scale, inv);
        if (threadIdx.x == 0) {
            inv_out[r] = inv;
            if (amax_out) amax_out[r] = m;
            if (l1_out) l1_out[r] = (red[4] + red[5]) + (red[6] + red[7]);
        }
        for (int k = threadIdx.x * 4; k < K; k += 512) {
            uint2 hi, lo;
            split_f16x4(load(k), scale, hi, lo);
            *reinterpret_cast<uint2*>(hr + k) = hi;
            *reinterpret_cast<uint2*>(hr + plane + k) = lo;
        }
    }
}

// bound = {largest L1 norm of a row, largest |bias|}; the norms were summed in fp32 (1.0001 covers that for any length in use).
// A NaN norm or bias gives no bound: fmaxf drops it, and what it enters is NaN whatever the scale.
__global__ void __launch_bounds__(1024) weight_bound_kernel(const float* __restrict__ l1, int64_t rows, const float* __restrict__ bias, int64_t n, float* __restrict__ bound) {
    __shared__ float red[2][32];
    grid_dep();
    float a = 0.f, b = 0.f;
    for (int64_t i = threadIdx.x; i < rows; i += blockDim.x) a = fmaxf(a, l1[i]);
    if (bias != nullptr)
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) b = fmaxf(b, fabsf(bias[i]));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    if (lane == 0) { red[0][warp] = a; red[1][warp] = b; }
    __syncthreads();
    if (warp > 0) return;
    a = red[0][lane]; b = red[1][lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    if (lane == 0) { bound[0] = a * 1.0001f; bound[1] = b; }
}

// A warp per row of w.  A normalised row has a 2-norm of at most sqrt(K) before gamma and beta, so |w · x| <= sqrt(K) ||w gamma|| + |w · beta|, which
// no input can exceed and a usual one comes within a few bits of, whatever the sizes of w and gamma.  1 %: operands rounded to bf16.
__global__ void __launch_bounds__(128) column_bounds_kernel(const float* __restrict__ w, int64_t rows, int K, const float* __restrict__ gamma, const float* __restrict__ beta,
                                                            const float* __restrict__ bias, float* __restrict__ bound) {
    grid_dep();
    const int lane = threadIdx.x & 31;
    const int64_t n = int64_t(blockIdx.x) * 4 + (threadIdx.x >> 5);
    if (n >= rows) return;
    double sq = 0, shift = 0, size = 0;
    for (int k = lane; k < K; k += 32) {
        const double v = w[n * K + k], g = v * gamma[k], s = v * beta[k];
        sq += g * g;
        shift += s;
        size += fabs(s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        shift += __shfl_xor_sync(0xffffffffu, shift, o);
        size += __shfl_xor_sync(0xffffffffu, size, o);
    }
    if (lane == 0) bound[n] = float((1.01 * sqrt(double(K) * sq) + fabs(shift) + 0.01 * size + fabs(double(bias[n]))) * 1.001);
}

// A block per head, a thread per column of 64.  A column d of Q and of K enter a score as one product, so their scales may differ from column to
// column as long as each pair multiplies to the same 2^C: the pair with the largest bound fills [-2^15, 2^15] on both sides, the others
// share what is left between them.  A factor moved from Q's weights to K's moves the scales along and no bit of the result.
// Every column of V has a scale of its own.
__global__ void __launch_bounds__(64) attention_scales_kernel(AttnScales s) {
    __shared__ int red[2][2];
    constexpr int kLimit = 60;   // of a scale's exponent: what the projection's epilogue and the core multiply stays in the range of fp32
    grid_dep();
    const int d = threadIdx.x, n = s.H * 64, q = int(blockIdx.x) * 64 + d;
    auto exponent = [](float b) { return (int(__float_as_uint(b) >> 23) & 255) - 126; };   // b < 2^exponent
    auto pow2 = [](int e) { return __int_as_float((e + 127) << 23); };
    const float bq = s.bound[q], bk = s.bound[n + q], bv = s.bound[2 * n + q];
    bool ok = bq < INFINITY && bk < INFINITY && bv < INFINITY;   // (NaN is not)
    const int eq = exponent(bq), ek = exponent(bk);
    const bool zero = bq == 0.f || bk == 0.f;                    // adds exactly nothing to a score
    int top = zero ? -1000 : eq + ek, top_v = -1000;
    for (int i = d; i < n; i += 64) top_v = max(top_v, exponent(s.bound[2 * n + i]));
    top = __reduce_max_sync(0xffffffffu, top);
    top_v = __reduce_max_sync(0xffffffffu, top_v);
    if ((d & 31) == 0) { red[0][d >> 5] = top; red[1][d >> 5] = top_v; }
    __syncthreads();
    top = max(red[0][0], red[0][1]);
    top_v = max(red[1][0], red[1][1]);
    const int C = top > -1000 ? 30 - top : 0;
    int aq, ak;
    if (zero) {
        aq = bq == 0.f ? 0 : min(15 - eq, kLimit);
        ak = bk == 0.f ? 0 : min(15 - ek, kLimit);
    } else {
        const int less = top - eq - ek;   // >= 0
        aq = min(15 - eq - less / 2, kLimit);
        ak = C - aq;
        if (less > kLimit) ak = min(min(ak, 15 - ek), kLimit);   // (too little for fp32 to notice: it may count for less)
        ok = ok && ak <= 15 - ek && ak <= kLimit;
    }
    const int av = min(15 - exponent(bv), kLimit), a_ctx = min(15 - top_v, kLimit);
    ok = ok && C >= -2 * kLimit && C <= 2 * kLimit && aq >= -kLimit && ak >= -kLimit && av >= -kLimit && a_ctx >= -kLimit;
    if (!ok) {
        *s.unusable = 1;
        return;
    }
    s.col_inv[q] = (s.q_winv ? s.q_winv[q] : 1.f) * pow2(aq);
    s.col_inv[n + q] = (s.kv_winv ? s.kv_winv[q] : 1.f) * pow2(ak);
    s.col_inv[2 * n + q] = (s.kv_winv ? s.kv_winv[n + q] : 1.f) * pow2(av);
    s.col_bias[q] = s.q_bias[q] * pow2(aq);
    s.col_bias[n + q] = s.kv_bias[q] * pow2(ak);
    s.col_bias[2 * n + q] = s.kv_bias[n + q] * pow2(av);
    s.v_inv[q] = pow2(-av);
    s.v_ctx[q] = pow2(a_ctx - av);
    if (d == 0) s.score_inv[blockIdx.x] = pow2(-C);
    if (q == 0) *s.ctx_inv = pow2(-a_ctx);
}

}  // namespace

int launch_split_rows(const float* x, int64_t ld, int64_t M, int64_t K, bool bf16, const SplitOut& out, float* l1_out, ExecCtx& ctx) {
    if (M == 0) return 0;
    FXF_CHECK(K % 8 == 0 && out.planes != nullptr, "split rows: K must be a multiple of 8");
    const int grid = int(std::min<int64_t>(M, int64_t(ctx.sm_count) * 16));
    tag_launch(ctx, bf16 ? "split_rows_bf16" : "split_rows_f16", 0, (bf16 ? 6.0 : 8.0) * double(M) * double(K));
    dependent(bf16 ? split_rows_kernel<1> : split_rows_kernel<0>, grid, 128, 0, ctx)(x, ld, out.planes, out.plane, out.inv, out.amax, l1_out, M, int(K));
    FXF_LAUNCHED(ctx);
    return 0;
}

int launch_weight_bound(const float* l1, int64_t rows, const float* bias, int64_t n, float* bound, ExecCtx& ctx) {
    tag_launch(ctx, "weight_bound", 0, 4.0 * double(rows + n));
    dependent(weight_bound_kernel, 1, 1024, 0, ctx)(l1, rows, bias, n, bound);
    FXF_LAUNCHED(ctx);
    return 0;
}

int launch_column_bounds(const float* w, int64_t rows, int64_t K, const float* gamma, const float* beta, const float* bias, float* bound, ExecCtx& ctx) {
    tag_launch(ctx, "column_bounds", 0, 4.0 * double(rows) * double(K));
    dependent(column_bounds_kernel, unsigned((rows + 3) / 4), 128, 0, ctx)(w, rows, int(K), gamma, beta, bias, bound);
    FXF_LAUNCHED(ctx);
    return 0;
}

int launch_attention_scales(const AttnScales& s, ExecCtx& ctx) {
    tag_launch(ctx, "attention_scales", 0, 4.0 * 64 * double(s.H) * 14);
    dependent(attention_scales_kernel, unsigned(s.H), 64, 0, ctx)(s);
    FXF_LAUNCHED(ctx);
    return 0;
}

}  // namespace fxf
