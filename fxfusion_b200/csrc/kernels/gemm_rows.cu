// Few-row GEMM for sm_100a:  out[M,N] = act(x[M,K] · w[N,K]^T + bias[N] (+ residual)),  M <= 64, on the tensor cores with the
// f16x3 arithmetic of gemm_f16.cu (weights in the same split form; see there).
//
// These products are weight reads: single-position decode steps, batch-sized MLP layers, the last-row vocabulary projection.
// The operands are swapped — a tile is 128 WEIGHT rows by all rows of x — so no tensor time goes into padding rows, and one
// tile's K range is cut over a cluster of up to 16 CTAs (pick_cluster), so that a 512-row weight already occupies 32 SMs.  Per CTA:
//   * weight slabs (128 rows x 64, both planes, 32 KB) by TMA.  They do not depend on the kernel before this one, so the first
//     STAGES slabs are requested before griddepcontrol.wait: the weight stream runs under the previous kernel;
//   * x comes as fp32 (or in split form): all warps fetch this CTA's K range of the rows, take the maximum of each row over
//     it, and write the two fp16 planes into swizzled shared memory.  The scale may differ between the CTAs of a cluster:
//     their results are only added after it has been divided out;
//   * MMAs of 128 x NB x 16; chains of one to three slabs in separate TMEM accumulators, added in fp32 registers;
//   * every CTA owns a share of the tile: the others push their partial sums of it into its shared memory (one bulk copy each,
//     counted on the owner's mbarrier), it adds them in rank order, applies scale, bias, residual and ReLU and stores rows of
//     consecutive columns.  Pulling the partial tiles after a cluster barrier instead, with another barrier before the exit,
//     cost 4000 to 7000 cycles of 9000 to 12000.
// Bound: HBM (4 bytes per weight element) for the large weights, launch-to-launch latency for the small ones.
#include <cuda.h>

#include <algorithm>
#include <atomic>

#include "../runtime.hpp"
#include "sm100.cuh"

namespace fxf {
namespace {

using namespace sm100;

constexpr int BN = 128, BK = 64, kThreads = 256, kWarps = kThreads / 32;
constexpr int kSlabsPerRound = 8;   // of the instances that have most
constexpr int kTmaWarp = 7, kMmaWarp = 6, kAccCols = 128, kMaxCluster = 16;   // TMEM columns per CTA
enum : int { kErrRowsFull = 141, kErrRowsEmpty = 142, kErrRowsDone = 143, kErrRowsReduce = 144, kErrRowsStats = 145 };

template <int NB, int STAGES, int XS>
struct alignas(1024) RowsSmem {
    uint16_t w[STAGES][2][BN * BK];   // [0] is reused for the partial tile [NB][128] once the products are done
    uint16_t x[XS][2][NB * BK];
    float recv[NB * BN + 64];         // [rank][share of the tile]: the cluster's partial sums of the elements this CTA owns
    float x_inv[NB];
    float2 stats[kMaxCluster][NB];    // (mean, centred sum of squares) of each row over each CTA's K range
    uint64_t full[STAGES], empty[STAGES], done, received, stats_in;
    uint32_t tmem_base;
    int abort_flag;
};

struct RowsParams {
    const float* x;               // [M] rows of K floats, ldx apart, or NULL:
    const uint16_t* x_planes;     // the rows in split form, ld_planes elements apart, 1 / scale x_inv_stride entries apart
    int64_t x_plane, ld_planes, x_inv_stride;
    const float* x_inv;
    int64_t ldx;
    const float *w_inv, *bias, *residual;
    float* out;
    int M, N, K, slabs;
    int64_t ldo;
    const float *gamma, *beta;    // NULL: x as it is
    float eps;
    int relu, early_w;
    int* status;
};

__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// `bytes` (a multiple of 16) of this CTA's shared memory to the same-named location of CTA `rank`, counted on its barrier
__device__ __forceinline__ void push_bulk(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar, uint32_t rank) {
    uint32_t d, b;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(dst), "r"(rank));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(bar), "r"(rank));
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(d), "r"(src), "r"(bytes), "r"(b) : "memory");
}

// eight bytes to the same-named location of CTA `rank`, counted on its barrier
__device__ __forceinline__ void push_pair(uint32_t dst, float2 v, uint32_t bar, uint32_t rank) {
    uint32_t d, b;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(dst), "r"(rank));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(bar), "r"(rank));
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(d), "f"(v.x), "f"(v.y), "r"(b) : "memory");
}
// N sums (1, 2 or 4) over the warp at once: lane l gets the total of sum l / (32 / N)
template <int N>
__device__ __forceinline__ float warp_sums(const float (&t)[N], int lane) {
    float v[N];
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = t[i];
    int o = 16;
#pragma unroll
    for (int n = N; n > 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; i++) {
            const float send = up ? v[i] : v[i + n / 2], mine = up ? v[i + n / 2] : v[i];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

template <int NB, int STAGES, int XS>
__global__ void __launch_bounds__(kThreads, STAGES <= 2 ? 2 : 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap map_w, RowsParams p) {
    extern __shared__ unsigned char smem_raw[];
    using Smem = RowsSmem<NB, STAGES, XS>;
    Smem& s = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr uint32_t kWBytes = 2 * BN * BK * 2;
    constexpr uint32_t kIdesc = umma_idesc_f16(BN, NB);
    // One accumulator for all corrections (hi·lo, lo·hi), the others for chains of hi·hi.  The tensor core truncates at every addition,
    // and the large sums take one per 16 K-elements so instead of three: 32 x 768 x 3072 lies 1.6e-7 from fp64 instead of 2.7e-7
    // (fp32 FFMA: 3.6e-7), at the same time.
    constexpr int NACC = kAccCols / NB - 1, COLS = NB >= 32 ? NB / 2 : NB, EPI_WARPS = NB >= 32 ? 8 : 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cs = int(cluster_nctarank()), rank = int(cluster_ctarank());
    const int tile = blockIdx.x / cs, n0 = tile * BN;
    const int m0 = blockIdx.y * NB, rows = min(NB, p.M - m0);   // this CTA's rows of x
    const int s0 = int(int64_t(p.slabs) * rank / cs), s1 = int(int64_t(p.slabs) * (rank + 1) / cs), count = s1 - s0;
    volatile int* abort_flag = &s.abort_flag;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&s.full[i], 1);
            mbar_init(&s.empty[i], 1);
        }
        mbar_init(&s.done, 1);
        mbar_init(&s.received, 1);
        mbar_init(&s.stats_in, 1);
        s.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)), "r"(kAccCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // shares of the tile's M * 128 elements, a multiple of 16 bytes each
    const int total = rows * BN, share = ((total + cs - 1) / cs + 3) & ~3, own0 = min(rank * share, total), own_n = min(share, total - own0);
    if (threadIdx.x == 0 && cs > 1) {
        mbar_expect_tx(&s.received, uint32_t(cs) * uint32_t(own_n) * 4u);
        if (p.gamma != nullptr) mbar_expect_tx(&s.stats_in, uint32_t(cs) * NB * 8u);
    }
    tc_fence_before();
    __syncthreads();
    if (cs > 1) cluster_sync_all();   // the peers' barriers exist (this runs under the previous kernel)
    tc_fence_after();
    const uint32_t tmem = s.tmem_base;
    grid_dep_launch();

    auto load_w = [&](int i) {   // slab i of this CTA
        const int st = i % STAGES;
        mbar_expect_tx(&s.full[st], kWBytes);
        tma_load_3d(s.w[st], &map_w, (s0 + i) * BK, n0, 0, &s.full[st]);
    };
    const bool producer = warp == kTmaWarp && lane == 0;
    int loaded = 0;   // producer: slabs requested so far
    if (producer && p.early_w)
        for (; loaded < min(STAGES, count); loaded++) load_w(loaded);
    // constants of this thread's output column (shares start at multiples of 4 elements, not of 128)
    const int nt = (own0 + threadIdx.x) & (BN - 1);
    const bool n_ok = n0 + nt < p.N;
    float wi = 0.f, bi = 0.f;
    auto column_constants = [&]() {
        if (n_ok) wi = p.w_inv[n0 + nt];
        if (n_ok && p.bias) bi = p.bias[n0 + nt];
    };
    if (p.early_w) column_constants();
    grid_dep_wait();
    if (!p.early_w) {   // the weight's conversion may be the kernel before this one
        column_constants();
        if (producer)
            for (; loaded < min(STAGES, count); loaded++) load_w(loaded);
    }

    float sum[COLS];
#pragma unroll
    for (int j = 0; j < COLS; j++) sum[j] = 0.f;
    const int quarter = warp & 3, mbase = NB >= 32 ? (warp >> 2) * COLS : 0;
    bool alive = true;
    int round = 0;
    for (int r0 = 0; r0 < count && alive; r0 += XS, round++) {
        const int ns = min(XS, count - r0), kb = (s0 + r0) * BK;
        // ---- this round's K range of the rows: fp32 -> two fp16 planes under one scale per row ----
        constexpr int V = (XS + 1) / 2, ROWS = NB / kWarps;   // float4 per lane and row (128 floats = two slabs each), rows per warp
        float4 v[ROWS][V];                                    // every row's loads are in flight before the first maximum
#pragma unroll
        for (int q = 0; q < ROWS; q++)
#pragma unroll
            for (int i = 0; i < V; i++) {
                const int r = q * kWarps + warp, at = i * 128 + lane * 4, k = kb + at;
                v[q][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < rows && at < ns * BK && k < p.K) {
                    if (p.x != nullptr) {
                        v[q][i] = *reinterpret_cast<const float4*>(p.x + (m0 + r) * p.ldx + k);
                    } else {
                        const uint2 h = *reinterpret_cast<const uint2*>(p.x_planes + (m0 + r) * p.ld_planes + k), l = *reinterpret_cast<const uint2*>(p.x_planes + p.x_plane + (m0 + r) * p.ld_planes + k);
                        const float inv = p.x_inv[(m0 + r) * p.x_inv_stride];
                        const float2 h0 = __half22float2(*reinterpret_cast<const __half2*>(&h.x)), h1 = __half22float2(*reinterpret_cast<const __half2*>(&h.y));
                        const float2 l0 = __half22float2(*reinterpret_cast<const __half2*>(&l.x)), l1 = __half22float2(*reinterpret_cast<const __half2*>(&l.y));
                        v[q][i] = make_float4((h0.x + l0.x) * inv, (h0.y + l0.y) * inv, (h1.x + l1.x) * inv, (h1.y + l1.y) * inv);
                    }
                }
            }
        if (p.gamma != nullptr) {   // (there is one round then) the statistics of a row are those of its parts, put together by every CTA of the cluster
            float4 g[V], bt[V];
            constexpr int G = 32 / ROWS;   // lanes that work on one row's statistics
            const int mine = lane / G, sub = lane % G;
            auto width = [&](int rk) { return float(min(p.slabs * (rk + 1) / cs * BK, p.K) - p.slabs * rk / cs * BK); };
            const float n_mine = width(rank), inv_all = 1.0f / float(p.K);
            bool in[V];
#pragma unroll
            for (int i = 0; i < V; i++) {
                const int at = i * 128 + lane * 4, k = kb + at;
                in[i] = at < ns * BK && k < p.K;
                g[i] = in[i] ? *reinterpret_cast<const float4*>(p.gamma + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                bt[i] = in[i] ? *reinterpret_cast<const float4*>(p.beta + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            float t[ROWS], mean[ROWS], rstd[ROWS];
#pragma unroll
            for (int q = 0; q < ROWS; q++) {
                t[q] = 0.f;
#pragma unroll
                for (int i = 0; i < V; i++) t[q] += (v[q][i].x + v[q][i].y) + (v[q][i].z + v[q][i].w);
            }
            float2 st;   // of row `mine`
            st.x = warp_sums(t, lane) / n_mine;
#pragma unroll
            for (int q = 0; q < ROWS; q++) {
                mean[q] = __shfl_sync(0xffffffffu, st.x, q * G);
                t[q] = 0.f;
#pragma unroll
                for (int i = 0; i < V; i++)
                    if (in[i]) {
                        const float dx = v[q][i].x - mean[q], dy = v[q][i].y - mean[q], dz = v[q][i].z - mean[q], dw = v[q][i].w - mean[q];
                        t[q] += (dx * dx + dy * dy) + (dz * dz + dw * dw);
                    }
            }
            st.y = warp_sums(t, lane);
            if (cs > 1) {
                for (int to = sub; to < cs; to += G) push_pair(smem_u32(&s.stats[rank][mine * kWarps + warp]), st, smem_u32(&s.stats_in), uint32_t(to));
                float n[2] = {0.f, 0.f};   // this lane's parts: sub and sub + G (a cluster has at most 16)
                if (sub < cs) n[0] = width(sub);
                if (sub + G < cs) n[1] = width(sub + G);
                __syncwarp();
                if (!__all_sync(0xffffffffu, mbar_wait(&s.stats_in, 0, abort_flag))) give_up(abort_flag, p.status, kErrRowsStats);
                float2 part[2];
#pragma unroll
                for (int j = 0; j < 2; j++) part[j] = n[j] > 0.f ? s.stats[sub + j * G][mine * kWarps + warp] : make_float2(0.f, 0.f);
                auto group_sum = [&](float x) {
#pragma unroll
                    for (int o = G / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    return x;
                };
                st.x = group_sum(n[0] * part[0].x + n[1] * part[1].x) * inv_all;
                const float d0 = part[0].x - st.x, d1 = part[1].x - st.x;
                st.y = group_sum(fmaf(n[0] * d0, d0, part[0].y) + fmaf(n[1] * d1, d1, part[1].y));
            }
            const float rs = 1.0f / sqrtf(st.y * inv_all + p.eps);
#pragma unroll
            for (int q = 0; q < ROWS; q++) {
                mean[q] = __shfl_sync(0xffffffffu, st.x, q * G);
                rstd[q] = __shfl_sync(0xffffffffu, rs, q * G);
            }
#pragma unroll
            for (int q = 0; q < ROWS; q++) {
                const float shift = -rstd[q] * mean[q];
                const bool real = q * kWarps + warp < rows;
#pragma unroll
                for (int i = 0; i < V; i++)
                    v[q][i] = real && in[i] ? make_float4((v[q][i].x * rstd[q] + shift) * g[i].x + bt[i].x, (v[q][i].y * rstd[q] + shift) * g[i].y + bt[i].y,
                                                          (v[q][i].z * rstd[q] + shift) * g[i].z + bt[i].z, (v[q][i].w * rstd[q] + shift) * g[i].w + bt[i].w)
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
#pragma unroll
        for (int q = 0; q < ROWS; q++) {
            const int r = q * kWarps + warp;
            float m = 0.f;
#pragma unroll
            for (int i = 0; i < V; i++) m = fmaxf(m, fmaxf(fmaxf(fabsf(v[q][i].x), fabsf(v[q][i].y)), fmaxf(fabsf(v[q][i].z), fabsf(v[q][i].w))));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            float scale, inv;
            split_scale(m, scale, inv);
            if (lane == 0) s.x_inv[r] = inv;
#pragma unroll
            for (int i = 0; i < V; i++) {
                const int sl = i * 2 + (lane >> 4);
                uint2 hi, lo;
                split_f16x4(v[q][i], scale, hi, lo);
                char* dst = reinterpret_cast<char*>(s.x[sl][0]) + r * 128 + ((((lane & 15) >> 1) ^ (r & 7)) << 4) + ((lane & 1) << 3);
                *reinterpret_cast<uint2*>(dst) = hi;
                *reinterpret_cast<uint2*>(dst + NB * BK * 2) = lo;
            }
        }
        fence_async_smem();
        __syncthreads();
        if (warp == kMmaWarp) {
            const uint32_t leader = elect_one();
            for (int i = 0; i < ns; i++) {
                const int g = r0 + i, st = g % STAGES;
                if (!(__all_sync(0xffffffffu, mbar_wait(&s.full[st], (g / STAGES) & 1, abort_flag)))) {
                    give_up(abort_flag, p.status, kErrRowsFull);
                    break;
                }
                tc_fence_after();
                if (leader) {
                    const uint64_t a = umma_desc_k_major_bytes<128>(smem_u32(s.w[st][0])), b = umma_desc_k_major_bytes<128>(smem_u32(s.x[i][0]));
                    constexpr uint64_t kALo = BN * BK * 2 / 16, kBLo = NB * BK * 2 / 16;
                    const uint32_t corr = tmem, acc = tmem + uint32_t(1 + i % NACC) * NB;
#pragma unroll
                    for (int kk = 0; kk < BK / 16; kk++) {
                        const uint64_t adv = uint64_t((kk * 32) >> 4);
                        umma_f16_ss<false>(corr, a + kALo + adv, b + adv, kIdesc, (i > 0 || kk > 0) ? 1u : 0u);
                        umma_f16_ss<false>(corr, a + adv, b + kBLo + adv, kIdesc, 1u);
                        umma_f16_ss<false>(acc, a + adv, b + adv, kIdesc, (i >= NACC || kk > 0) ? 1u : 0u);
                    }
                    umma_commit(&s.empty[st]);
                    if (i + 1 == ns) umma_commit(&s.done);
                }
            }
        }
        if (producer) {   // the ring is refilled while the products run (the next round's slabs included)
            for (; loaded < min(count, r0 + ns + STAGES); loaded++) {
                if (!mbar_wait(&s.empty[loaded % STAGES], ((loaded / STAGES) - 1) & 1, abort_flag)) {
                    give_up(abort_flag, p.status, kErrRowsEmpty);
                    break;
                }
                load_w(loaded);
            }
        }
        __syncwarp();
        alive = __all_sync(0xffffffffu, mbar_wait(&s.done, round & 1, abort_flag));
        if (!alive) give_up(abort_flag, p.status, kErrRowsDone);
        tc_fence_after();
        if (alive && warp < EPI_WARPS) {
            const int nacc = 1 + min(ns, NACC);   // the corrections first
            for (int a = 0; a < nacc; a++) {
                const uint32_t t = tmem + (uint32_t(quarter * 32) << 16) + uint32_t(a * NB + mbase);
                uint32_t d[COLS];
                tmem_ld(t, d);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < COLS; j++) sum[j] = fmaf(__uint_as_float(d[j]), s.x_inv[mbase + j], sum[j]);
            }
        }
        tc_fence_before();
        alive = __syncthreads_and(alive ? 1 : 0) != 0;   // the x planes, scales and accumulators may be reused
    }

    // ---- partial tile to shared memory, then the sum over the cluster ----
    float* part = reinterpret_cast<float*>(s.w[0]);
    if (warp < EPI_WARPS) {
#pragma unroll
        for (int j = 0; j < COLS; j++) part[(mbase + j) * BN + quarter * 32 + lane] = sum[j];
    }
    if (cs > 1) fence_async_smem();
    __syncthreads();
    const float* mine = part + own0;
    if (cs > 1) {
        if (warp == 0) {
            if (lane < cs) {
                const int q0 = min(lane * share, total), qn = min(share, total - q0);
                if (qn > 0) push_bulk(smem_u32(s.recv) + uint32_t(rank * qn) * 4u, smem_u32(part + q0), uint32_t(qn) * 4u, smem_u32(&s.received), uint32_t(lane));
            }
            __syncwarp();
        }
        if (!mbar_wait(&s.received, 0, abort_flag)) {
            give_up(abort_flag, p.status, kErrRowsReduce);
            alive = false;
        }
        mine = s.recv;
        // All this CTA was sent has arrived.  Once that holds for the whole cluster everyone may leave: nothing that was pushed
        // is still being read.  Arriving here (relaxed: no memory has to be ordered) takes the wait below off the path.
        __syncwarp();
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    }
    for (int i = threadIdx.x; alive && i < own_n; i += kThreads) {
        float t[kMaxCluster], v = 0.f;
#pragma unroll
        for (int q = 0; q < kMaxCluster; q++) t[q] = q < cs ? mine[q * own_n + i] : 0.f;
#pragma unroll
        for (int q = 0; q < kMaxCluster; q++) v += t[q];
        if (n_ok) {
            const int64_t off = int64_t(m0 + ((own0 + i) >> 7)) * p.ldo + n0 + nt;
            v = fmaf(v, wi, bi);
            if (p.residual != nullptr) v += p.residual[off];
            p.out[off] = p.relu ? relu_keep_nan(v) : v;
        }
    }
    tc_fence_before();
    if (cs > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    __syncthreads();
    let_copies_land(abort_flag);
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAccCols) : "memory");
    }
}

// The instances: rows of x per CTA, K-slabs per CTA that fit without refilling the rings, CTAs per SM (two slabs take 70-100 KB of
// shared memory: two CTAs share an SM, or one stands beside one of the kernel before it).
using RowsKernel = void (*)(const CUtensorMap, RowsParams);
struct RowsInstance { int index, rows, slabs, per_sm; RowsKernel kernel; size_t smem; };
template <int NB, int STAGES, int XS>
RowsInstance instance(int index) {
    static_assert(sizeof(RowsSmem<NB, STAGES, XS>) + 1024 <= 227 * 1024, "shared memory of a CTA");
    return {index, NB, XS, STAGES <= 2 ? 2 : 1, gemm_rows_kernel<NB, STAGES, XS>, sizeof(RowsSmem<NB, STAGES, XS>) + 1024};
}
const RowsInstance& instance_for(int64_t M, int per) {
    static const RowsInstance all[] = {instance<16, 2, 2>(0), instance<16, 4, 8>(1), instance<32, 2, 2>(2), instance<32, 4, 4>(3), instance<32, 4, 8>(4)};
    return all[M <= 16 ? (per <= 2 ? 0 : 1) : (per <= 2 ? 2 : (per <= 4 ? 3 : 4))];
}
int configure(const RowsInstance& r) {
    static std::atomic<unsigned> done[64];   // a bit per instance
    int dev = 0;
    FXF_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && (done[dev].load(std::memory_order_relaxed) >> r.index & 1u)) return 0;
    FXF_CUDA(cudaFuncSetAttribute(r.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(r.smem)));
    FXF_CUDA(cudaFuncSetAttribute(r.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (dev >= 0 && dev < 64) done[dev].fetch_or(1u << r.index, std::memory_order_relaxed);
    return 0;
}

// Clusters of `cs` CTAs, one CTA per SM, that the device holds at once.  A cluster lives inside one GPC, so this is not the number of
// SMs over cs, and differs between devices of the same kind.  Asked once per device: the answer does not change.  (148 SMs here:
// 33 clusters of 4, 22 of 6, 15 of 8, 7 of 11 to 16.)
int clusters_resident(int cs, int* out) {
    static std::atomic<int> known[64][kMaxCluster + 1];   // answer + 1
    int dev = 0;
    FXF_CUDA(cudaGetDevice(&dev));
    std::atomic<int>* slot = dev >= 0 && dev < 64 ? &known[dev][cs] : nullptr;
    *out = slot != nullptr ? slot->load(std::memory_order_relaxed) - 1 : -1;
    if (*out >= 0) return 0;
    const RowsInstance& r = instance_for(1, kMaxCluster);   // one CTA per SM
    if (configure(r)) return 1;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(cs);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(cs));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = r.smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(out, r.kernel, &cfg) != cudaSuccess) {   // a size this device does not launch at all
        (void)cudaGetLastError();
        *out = 0;
    }
    if (slot != nullptr) slot->store(*out + 1, std::memory_order_relaxed);
    return 0;
}

// CTAs per tile: the least modelled time over all cluster sizes.  In a chain of launches with weights from HBM a K-slab of a CTA takes
// 0.27 us for one row and 0.9 us for 32; clusters that do not fit the device at once form another wave of 4 us and its slabs; and
// the fuller the device, the less of the next kernel can start beside this one, up to 1.6 us.  Fitted to 511 shapes on 148 SMs (1 to
// 64 rows, 1 to 140 tiles, K = 200 to 6144, chains of 16): 0.5 % above the best measured size on average, and 16 % below the rule
// before it (up to 8 CTAs; 16 for at most 6 tiles), whose choice was the better one by at most 12 %.  Some of them, us per launch
// of 32 rows:
//   N =  768, K = 1536:  8 CTAs 6.2, 12 5.8      N = 2048, K = 1536:  8 12.7 (16 clusters; the device holds 15), 6 7.8, 12 7.4
//   N = 1024, K = 2048:  8 CTAs 7.1, 16 6.4      N = 2304, K =  768:  6  6.7, 4 7.4, 12 10.9
int pick_cluster(int64_t M, int tiles, int slabs, int max_slabs, int* cs_out) {
    double best = 0;
    *cs_out = 0;
    for (int cs = 1; cs <= std::min(kMaxCluster, slabs); cs++) {
        const int per = (slabs + cs - 1) / cs;
        if ((slabs + per - 1) / per != cs || per > max_slabs) continue;   // no more CTAs than give the fewest slabs
        const RowsInstance& inst = instance_for(M, per);
        int resident = 0;
        if (clusters_resident(cs, &resident)) return 1;
        resident *= inst.per_sm;
        if (resident < 1) continue;
        const int64_t clusters = int64_t(tiles) * ((M + inst.rows - 1) / inst.rows);
        const double fill = std::min(1.0, double(clusters) / resident), slab = 0.25 + 0.02 * double(std::min<int64_t>(M, 32));
        const double us = double((clusters + resident - 1) / resident) * (slab * per + 4.0) + 1.6 * fill;
        if (*cs_out == 0 || us < best) {
            *cs_out = cs;
            best = us;
        }
    }
    FXF_CHECK(*cs_out > 0, "few-row GEMM: no cluster size fits the device");
    return 0;
}

}  // namespace

bool gemm_rows_ok(int64_t M, int64_t N, int64_t K) { return M >= 1 && M <= 64 && gemm_f16_shape_ok(M, N, K); }
// From a tile per SM on, a persistent kernel that streams its weights without a break between tiles is the better one
// (launch_gemm_f16_swapped; 32 x 50257 x 768: 46 us here).
bool gemm_rows_streams(int64_t M, int64_t N, int sm_count) { return M <= 64 && (N + BN - 1) / BN >= sm_count; }

// x: fp32 rows `ldx` floats apart (16-byte aligned), or NULL with a.x in split form.
int launch_gemm_rows(const F16GemmArgs& a, const float* x, int64_t ldx, ExecCtx& ctx) {
    if (a.M == 0 || a.N == 0) return 0;
    FXF_CHECK(gemm_rows_ok(a.M, a.N, a.K) && !a.bf16 && a.w.planes && a.out && (x != nullptr || a.x.planes != nullptr), "few-row GEMM: unsupported operands");
    FXF_CHECK(x == nullptr || (aligned16(x) && ldx % 4 == 0), "few-row GEMM: unaligned rows");
    FXF_CHECK(a.norm.gamma == nullptr || (x != nullptr && a.norm.beta != nullptr && aligned16(a.norm.gamma) && aligned16(a.norm.beta) && a.K <= kNormRowMax), "few-row GEMM: unsupported LayerNorm");
    CUtensorMap map;
    const CUresult r = encode_planes(&map, a.w.planes, a.N, a.K, a.K, a.w.plane, 2, BK, BN);
    FXF_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled (rows) failed with code %d", int(r));
    RowsParams p{};
    p.x = x; p.ldx = ldx;
    if (x == nullptr) {
        p.x_planes = a.x.planes; p.x_plane = a.x.plane; p.ld_planes = a.x.ld ? a.x.ld : a.K; p.x_inv = a.x.inv; p.x_inv_stride = a.x.inv_stride;
    }
    p.w_inv = a.w.inv; p.bias = a.bias; p.residual = a.residual; p.out = a.out;
    p.M = int(a.M); p.N = int(a.N); p.K = int(a.K); p.ldo = a.ldo;
    p.slabs = int((a.K + BK - 1) / BK);
    p.gamma = a.norm.gamma; p.beta = a.norm.beta; p.eps = a.norm.eps;
    p.relu = a.relu ? 1 : 0;
    p.early_w = ctx.weights_settled ? 1 : 0;
    p.status = ctx.status;
    const int tiles = int((a.N + BN - 1) / BN);
    int cs = 0;
    // rows that are normalised on the way stay in registers meanwhile: no more than one round of slabs
    if (pick_cluster(a.M, tiles, p.slabs, a.norm.gamma ? kSlabsPerRound : p.slabs, &cs)) return 1;
    const RowsInstance& inst = instance_for(a.M, (p.slabs + cs - 1) / cs);
    if (configure(inst)) return 1;
    tag_launch(ctx, "gemm_f16x3_rows_tcgen05", 2.0 * double(a.M) * double(a.N) * double(a.K),
               4.0 * (double(a.M) * a.K + double(a.N) * a.K + double(a.N) + double(a.M) * a.N));
    FXF_CUDA(launch_dependent(inst.kernel, dim3(unsigned(tiles * cs), unsigned((a.M + inst.rows - 1) / inst.rows)), dim3(kThreads), inst.smem, ctx.stream, cs, map, p));
    FXF_LAUNCHED(ctx);
    return 0;
}

}  // namespace fxf
