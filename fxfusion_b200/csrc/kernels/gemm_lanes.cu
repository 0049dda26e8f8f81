// Few-row GEMM in fp32 FFMA for sm_100a:  out[M,N] = act(norm(x)[M,K] · w[N,K]^T + bias[N] (+ residual)),  M <= 64.
//
// For products whose time is the latency between two launches.  A CTA owns R rows by a few columns, its lanes (and groups of warps) share
// K, and little stands between the end of the kernel before it and the multiplication: the CTA's weight rows (fp32, as the file has
// them) are on their way into shared memory before griddepcontrol.wait; then the R rows of x are staged, optionally normalised
// on the way (a LayerNorm whose result only this product reads), each warp multiplies R rows by C columns over its share of K, the
// lanes' sums are added by a butterfly that leaves every lane with its own outputs, the groups' through shared memory, and bias,
// residual and ReLU follow.  No conversion, no tensor memory, no cluster.
#include <algorithm>

#include "../runtime.hpp"
#include "sm100.cuh"

namespace fxf {
namespace {

using namespace sm100;

constexpr int kMaxRows = 64, kWarps = 8, kThreads = kWarps * 32;
constexpr size_t kSmemLimit = 208 * 1024;
enum : int { kErrLanesWeights = 161 };

struct LanesParams {
    const float *x, *w, *bias, *residual;
    float* out;
    int64_t ldx, ldo;
    const float *gamma, *beta;   // NULL: x as it is
    float eps;
    int M, N, K, col_groups;     // kWarps / col_groups groups of warps share K
    int relu, early_w;
    int* status;
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
constexpr int pow2_from(int n) { return n <= 1 ? 1 : 2 * pow2_from((n + 1) / 2); }

template <int R, int C>
__global__ void __launch_bounds__(kThreads, 1) gemm_lanes_kernel(LanesParams p) {
    extern __shared__ __align__(128) float sm[];
    constexpr int S = pow2_from(R * C), PER = S > 32 ? S / 32 : 1, SHARE = S >= 32 ? 1 : 32 / S;   // sums of a warp, of a lane, lanes with the same sum
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    __shared__ float part[kWarps][PER][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, K = p.K;
    const int cols = p.col_groups * C, n0 = int(blockIdx.x) * cols, have = min(cols, p.N - n0), m0 = int(blockIdx.y) * R, rows = min(R, p.M - m0);
    const int cg = warp % p.col_groups, kg = warp / p.col_groups, kgs = kWarps / p.col_groups;
    float* ws = sm;                       // [cols][K]
    float* xs = sm + size_t(cols) * K;    // [R][K]
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    grid_dep_launch();
    auto load_w = [&]() {
        mbar_expect_tx(&bar, uint32_t(have) * uint32_t(K) * 4u);
        for (int c = 0; c < have; c++) bulk_load(ws + size_t(c) * K, p.w + int64_t(n0 + c) * K, uint32_t(K) * 4u, &bar);
    };
    if (threadIdx.x == 0 && p.early_w) load_w();
    // the outputs of this lane: sums r * C + c, spread over the lanes by the butterfly below
    float bi[PER] = {}, res[PER] = {};
    int row[PER], col[PER];
    auto fetch_bias = [&]() {
#pragma unroll
        for (int i = 0; i < PER; i++)
            if (row[i] >= 0 && p.bias) bi[i] = p.bias[col[i]];
    };
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int idx = S >= 32 ? lane * PER + i : lane / SHARE, r = idx / C, c = idx - r * C;
        row[i] = m0 + r;
        col[i] = n0 + cg * C + c;
        if (r >= rows || col[i] >= p.N || lane % SHARE != 0 || kg != 0) row[i] = -1;
    }
    if (p.early_w) fetch_bias();
    grid_dep_wait();
    if (!p.early_w) {   // a weight that the kernel before this one may still write
        if (threadIdx.x == 0) load_w();
        fetch_bias();
    }
    // ---- rows of x into shared memory; rows that do not exist are zeros ----
    const int k4 = K / 4;
    if (p.gamma == nullptr) {
        for (int i = threadIdx.x; i < R * k4; i += kThreads) {
            const int r = i / k4, c = i - r * k4;
            const bool ok = r < rows;
            const float* src = ok ? p.x + int64_t(m0 + r) * p.ldx + c * 4 : p.x;
            const int bytes = ok ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(xs + size_t(r) * K + c * 4)), "l"(src), "r"(bytes) : "memory");
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    } else {
        constexpr int NV = 8;   // a row of up to 1024 elements in registers
        for (int r = warp; r < R; r += kWarps) {
            float4 v[NV];
            float s = 0.f, q = 0.f;
#pragma unroll
            for (int i = 0; i < NV; i++) {
                const int c = lane + 32 * i;
                v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c < k4 && r < rows) v[i] = *reinterpret_cast<const float4*>(p.x + int64_t(m0 + r) * p.ldx + c * 4);
            }
#pragma unroll
            for (int i = 0; i < NV; i++) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
            const float mean = warp_sum(s) / float(K);
#pragma unroll
            for (int i = 0; i < NV; i++)
                if (lane + 32 * i < k4) {
                    const float dx = v[i].x - mean, dy = v[i].y - mean, dz = v[i].z - mean, dw = v[i].w - mean;
                    q += (dx * dx + dy * dy) + (dz * dz + dw * dw);
                }
            const float rstd = 1.0f / sqrtf(warp_sum(q) / float(K) + p.eps), shift = -rstd * mean;
#pragma unroll
            for (int i = 0; i < NV; i++) {
                const int c = lane + 32 * i;
                if (c < k4) {
                    const float4 g = *(reinterpret_cast<const float4*>(p.gamma) + c), b = *(reinterpret_cast<const float4*>(p.beta) + c);
                    *reinterpret_cast<float4*>(xs + size_t(r) * K + c * 4) =
                        make_float4((v[i].x * rstd + shift) * g.x + b.x, (v[i].y * rstd + shift) * g.y + b.y, (v[i].z * rstd + shift) * g.z + b.z, (v[i].w * rstd + shift) * g.w + b.w);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < PER; i++)
        if (row[i] >= 0 && p.residual) res[i] = p.residual[int64_t(row[i]) * p.ldo + col[i]];
    if (!mbar_wait(&bar, 0, &abort_flag)) give_up(&abort_flag, p.status, kErrLanesWeights);
    __syncthreads();
    if (abort_flag) {
        let_copies_land(&abort_flag);
        return;
    }
    // ---- R x C sums per lane ----
    float acc[S];
#pragma unroll
    for (int i = 0; i < S; i++) acc[i] = 0.f;
    const float* wr = ws + size_t(cg) * C * K;
#pragma unroll 2
    for (int k = kg * 128 + lane * 4; k < K; k += kgs * 128) {
        float4 xv[R];
#pragma unroll
        for (int r = 0; r < R; r++) xv[r] = *reinterpret_cast<const float4*>(xs + r * K + k);
#pragma unroll
        for (int c = 0; c < C; c++) {
            const float4 wv = *reinterpret_cast<const float4*>(wr + c * K + k);
#pragma unroll
            for (int r = 0; r < R; r++)
                acc[r * C + c] = fmaf(xv[r].w, wv.w, fmaf(xv[r].z, wv.z, fmaf(xv[r].y, wv.y, fmaf(xv[r].x, wv.x, acc[r * C + c]))));
        }
    }
    // ---- add over the lanes: at every step a lane keeps one half of its sums and sends the other ----
    int o = 16;
#pragma unroll
    for (int n = S; n > PER; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; i++) {
            const float send = up ? acc[i] : acc[i + n / 2], mine = up ? acc[i + n / 2] : acc[i];
            acc[i] = mine + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    if (S < 32) {
#pragma unroll
        for (; o > 0; o >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
    }
    if (kgs > 1) {   // and over the groups, in order
        if (kg > 0) {
#pragma unroll
            for (int i = 0; i < PER; i++) part[warp][i][lane] = acc[i];
        }
        __syncthreads();
        if (kg > 0) return;
        for (int g = 1; g < kgs; g++) {
#pragma unroll
            for (int i = 0; i < PER; i++) acc[i] += part[g * p.col_groups + cg][i][lane];
        }
    }
#pragma unroll
    for (int i = 0; i < PER; i++)
        if (row[i] >= 0) {
            const float v = acc[i] + bi[i] + res[i];
            p.out[int64_t(row[i]) * p.ldo + col[i]] = p.relu ? relu_keep_nan(v) : v;
        }
}

using LanesKernel = void (*)(LanesParams);
struct LanesPlan { LanesKernel kernel = nullptr; int rows = 0, cols = 0, col_groups = 0; size_t smem = 0; double us = 0; };
template <int R>
LanesKernel kernel_for(int c) {
    return c == 1 ? gemm_lanes_kernel<R, 1> : (c == 2 ? gemm_lanes_kernel<R, 2> : (c == 4 ? gemm_lanes_kernel<R, 4> : gemm_lanes_kernel<R, 8>));
}
LanesKernel kernel_for(int r, int c) {
    return r == 1 ? kernel_for<1>(c) : (r == 2 ? kernel_for<2>(c) : (r == 4 ? kernel_for<4>(c) : (r == 8 ? kernel_for<8>(c) : kernel_for<16>(c))));
}

// The tile with the least modelled time: multiplications or shared-memory reads (whichever is more), rows of x and weights through the L2
// port of an SM, the butterfly, and the fuller the device the less of the next kernel starts beside this one.  Fitted to 1090 launches
// in chains (M = 1 to 32, nine shapes of 256 x 256 to 3072 x 768): the pick is 4 % above the best measured tile on average, 24 % at worst.
LanesPlan plan(int64_t M, int64_t N, int64_t K, int sm_count) {
    LanesPlan best;
    if (M < 1 || M > kMaxRows || K % 4 != 0) return best;
    const int fewest = M == 1 ? 1 : (M == 2 ? 2 : (M <= 4 ? 4 : 8));
    const double cycles = 1850;   // per microsecond
    for (int r : {fewest, M > 8 ? 16 : fewest})
        for (int cg : {1, 2, 4, 8})
            for (int c : {1, 2, 4, 8}) {
                const int64_t cb = int64_t(cg) * c, ctas = (N + cb - 1) / cb * ((M + r - 1) / r);
                const size_t smem = size_t(cb + r) * size_t(K) * 4;
                if (smem > kSmemLimit || ctas > 2 * sm_count) continue;
                const double per_sm = double((ctas + sm_count - 1) / sm_count), fill = std::min(1.0, double(ctas) / sm_count), k = double(K) / cycles;
                const double us = 1.7 + per_sm * (std::max(1.6 * r * double(cb) * k / 128, 0.8 * cg * (r + c) * k * 4 / 128) + (2.1 * r + 0.4 * double(cb)) * k * 4 / 50) + 0.4 * r * c / 64 + 0.25 * fill + (cg < kWarps ? 0.08 : 0.0);
                if (best.kernel == nullptr || us < best.us) {
                    best.kernel = kernel_for(r, c);
                    best.rows = r; best.cols = c; best.col_groups = cg; best.smem = smem;
                    best.us = us;
                }
            }
    return best;
}

}  // namespace

// Against gemm_rows.cu, whose time in the same chains is 2.45 us + 1.15 per 1000 of K + 0.3 per 1000 of N + 0.062 per row from 9 on (within
// 15 %; the modelled minimum above is 5 to 15 % below what its tile measures).  us per launch, that kernel and this one:  1 row: 512 x 512 3.3, 2.0; 3072 x 768 4.9, 2.9; 768 x 3072 6.1, 3.5;  8 rows: 512 x 512 3.3, 2.9;
// 768 x 3072 6.2, 5.7;  32 rows: 256 x 256 4.9, 2.8; 512 x 512 4.6, 3.7; 768 x 768 5.1, 4.6; but 2304 x 768 6.7, 6.7 and 768 x 3072 7.1, 16.0.
// Neither formula knows what a CTA pays for its outputs, nor that a narrow product's clusters grow with K, so they count only inside what has been
// measured (42 shapes of 16 to 18000 columns, K 16 to 4096, 12 numbers of rows from 1 to 64).  Beyond it this kernel took, against the other, per launch:  1 row
// 16000 x 64 +0.3 us; 8 rows 16000 x 64 +3.3, 128 x 2048 +0.8, 1024 x 4096 +3.4; 9 rows 5000 x 32 +2.6; 16 rows 256 x 2048 +1.0; 32 rows 3000 x 32 +0.9; 33 rows 2048 x 128
// +0.9; 64 rows 704 x 704 and 1500 x 16 +1.2 and, with a CTA per output column as the model would have it, 16000 x 64 +26.
bool gemm_lanes_better(int64_t M, int64_t N, int64_t K, int sm_count) {
    if (M <= 8 ? N > 64 * int64_t(sm_count) || (M > 4 && K > 1408) : N > 3072 || M * N > 67000 || K > 1024 || M * N * K > 30000000) return false;
    const LanesPlan pl = plan(M, N, K, sm_count);
    return pl.kernel != nullptr && 1.13 * pl.us < 2.45 + 0.00115 * double(K) + 0.0003 * double(N) + 0.062 * double(std::max<int64_t>(M - 8, 0));
}

int launch_gemm_lanes(const F16GemmArgs& a, const float* w, const float* x, int64_t ldx, ExecCtx& ctx) {
    if (a.M == 0 || a.N == 0) return 0;
    const LanesPlan pl = plan(a.M, a.N, a.K, ctx.sm_count);
    FXF_CHECK(pl.kernel != nullptr && x != nullptr && w != nullptr && aligned16(x) && aligned16(w) && ldx % 4 == 0 && a.out != nullptr, "few-row GEMM (FFMA): unsupported operands");
    FXF_CHECK(a.norm.gamma == nullptr || (a.norm.beta != nullptr && aligned16(a.norm.gamma) && aligned16(a.norm.beta) && a.K <= kNormRowMax), "few-row GEMM (FFMA): unsupported LayerNorm");
    LanesParams p{};
    p.x = x; p.w = w; p.bias = a.bias; p.residual = a.residual; p.out = a.out;
    p.ldx = ldx; p.ldo = a.ldo;
    p.M = int(a.M); p.N = int(a.N); p.K = int(a.K);
    p.col_groups = pl.col_groups;
    p.gamma = a.norm.gamma; p.beta = a.norm.beta; p.eps = a.norm.eps;
    p.relu = a.relu ? 1 : 0;
    p.early_w = ctx.weights_settled ? 1 : 0;
    p.status = ctx.status;
    FXF_CUDA(cudaFuncSetAttribute(pl.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemLimit)));
    tag_launch(ctx, "gemm_lanes_ffma", 2.0 * double(a.M) * double(a.N) * double(a.K), 4.0 * (double(a.M) * a.K + double(a.N) * a.K + double(a.N) + double(a.M) * a.N));
    const int cb = pl.col_groups * pl.cols;
    FXF_CUDA(launch_dependent(pl.kernel, dim3(unsigned((a.N + cb - 1) / cb), unsigned((a.M + pl.rows - 1) / pl.rows)), dim3(kThreads), pl.smem, ctx.stream, 1, p));
    FXF_LAUNCHED(ctx);
    return 0;
}

}  // namespace fxf
