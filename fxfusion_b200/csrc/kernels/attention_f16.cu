// Tensor-core attention core for head_dim 64 on operands that are already in split form (gemm_f16.cu):
//     ctx = softmax(mask_fill(Q·K^T / scale_divisor)) · V        per (batch, head)
// Q, K and V are two fp16 planes each, written by the epilogue of their projection under a power-of-two scale per column
// (attention_scales_kernel: a pair of columns of Q and K has the same product of scales throughout a head), so both contractions are
// three kind::f16 products (hi·lo, lo·hi, hi·hi) on tiles that nothing touches between TMA and tensor core.  V needs no transposed copy: as the B operand of P·V it is read with the head columns
// contiguous (MN-major).  Semantics are those of attention.cu and attention_tc.cu (which serves the other arithmetic modes, rows
// whose size is not bounded by a LayerNorm, few rows and more than kMaxKeys keys): -inf where mask == 0, fully masked rows give NaN,
// masked keys still enter P·V with weight 0, and a block of keys is skipped only when every mask byte of it is 0 for all 128
// query rows of the CTA and its V rows are all finite.
//
// A unit of work is (128 queries, b, h); persistent CTAs of 320 threads, key blocks of BKEY = 128 (64 where there are no more keys), two CTAs per SM so
// that one's products run under the other's softmax:
//     warp 0        TMA, both planes of a tile in one load: the next K once S is done, the next V once P·V is, and the next unit's Q and
//                   first K behind the last S of this one (a unit's first loads took a quarter of its time);
//     warp 1        MMAs;
//     warps 2-9     softmax, two threads per query row, each owning half of the block's keys and 32 of the 64 output columns.
// The mask comes as bits (mask_bits_kernel: once per forward and mask, whatever the number of layers and heads that use it), with a word
// per query tile that says which key blocks any row sees.  P is split as p * 2^15 = hi + lo (the factor cancels against the row sum) and written over
// S, per 16 keys 8 columns of hi and 8 of lo: a thread only overwrites scores that it has read.  P_hi meets both planes of V in
// one instruction, 128 columns wide (65 cycles; two of 64 columns take 97), so hi·hi and the corrections have accumulators of their
// own.  Tensor memory: S / P [128 x BKEY] | O: hi·hi [128 x 64] | corrections [128 x 64].  O of a block is added to registers in fp32.
//
// Bound: the dependent chain of a key block (S 1500 cycles with a second CTA's products in between, softmax 2700, P·V 1800), of which two
// run per SM; behind it 1024 cycles of exponentials and 1560 of tensor pipe per block.  Times per layer, attention_tc.cu and here: 32 x 256
// positions, 12 heads, causal 77 and 37 us; encoder-decoder, 64 x 256, 8 heads, on average 104 and 47; 5 x 197, 12 heads 35 (the transpose of V
// included) and 14.  What it took: mask bits from one pass per forward (reading the bytes here cost 6500 of 22000 cycles per unit), a
// context that leaves by TMA (4000 cycles with 16-byte stores), the next unit's loads behind the last S.
#include <algorithm>
#include <cmath>

#include "../runtime.hpp"
#include "sm100.cuh"

namespace fxf {
namespace {

using namespace sm100;

constexpr int HD = 64, BQ = 128, kThreads = 320, kSoftWarp0 = 2;
constexpr int kMaxKeys = 2048;   // 16 blocks of 128; the words that track key blocks have room for 32, but more has not been measured against attention_tc.cu
constexpr float kLog2e = 1.4426950408889634f;
enum : int { kErrAttnF16Load = 151, kErrAttnF16S = 152, kErrAttnF16P = 153, kErrAttnF16O = 154 };

__device__ __forceinline__ float fast_exp2(float x) {   // 2^-inf = 0, NaN stays NaN
    float y;
    asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// the two softmax warps that share a quarter of the query rows
__device__ __forceinline__ void pair_sync(int quarter) { asm volatile("bar.sync %0, 64;" ::"r"(quarter + 1) : "memory"); }
__device__ __forceinline__ bool warp_all(bool ok) { return __all_sync(0xffffffffu, ok) != 0; }
// one bit per byte that is not zero
__device__ __forceinline__ uint32_t nonzero4(uint32_t w) { return (((__vcmpne4(w, 0u) & 0x01010101u) * 0x01020408u) >> 24) & 0xFu; }

template <int BKEY>
struct alignas(1024) AttnF16Smem {
    uint16_t q[2][BQ * HD];
    uint16_t k[2][BKEY * HD];
    uint16_t v[2 * BQ * HD];       // both planes of a block's V, later the context [quarter of the rows][plane]
    float vf[8][36];               // per softmax warp: the factors of its 32 columns, and AttnScales::ctx_inv
    float exch[2][2][BQ];          // row statistics exchanged between the two threads of a row, by block parity
    uint64_t bar_q, bar_k, bar_v, bar_s, bar_p, bar_o, bar_free;   // bar_free: the staged context has been read, V may be loaded
    uint32_t tmem_base;
    int abort_flag;
};

struct AttnF16Params {
    const uint32_t *bits, *need;   // MaskBits
    int64_t bit_sb, bit_sh, bit_sq, need_sb, need_sh, need_st;
    const uint32_t* bad;           // per batch: the key blocks with a projected value that is not finite
    float* ctx;
    int B, T, Tk, H, q_tiles, units;
    int q_col, k_col, v_col;
    int64_t ld_ctx;
    const float *score_inv, *v_factor, *ctx_inv;   // AttnScales; v_factor: v_ctx where split is 2, v_inv otherwise
    float score_scale;             // log2(e) / scale_divisor
    int split;                     // the context leaves by TMA: 2: as two fp16 planes, 1: as bf16; 0: fp32 in ctx
    float* so_inv;
    int* status;
};

struct MaskParams {
    const uint8_t* mask;
    int64_t sb, sh, sq, sk;
    int mh, rows, Tk, words, tiles, bkey, vec16, contiguous;
    uint32_t *bits, *need, *bad;
    int batches;
};

// sixteen mask bytes of one row as bits, keys k0 .. k0 + 15
__device__ __forceinline__ uint32_t mask16(const MaskParams& p, const uint8_t* row, int k0) {
    const int n = p.Tk - k0;   // > 0
    if (p.contiguous) {   // bytes at any address: the aligned words around them, none of which lies wholly outside the row
        const uint8_t* src = row + k0;
        const int off = int(reinterpret_cast<uintptr_t>(src) & 3), have = min(n, 16) + off;
        const uint32_t* wp = reinterpret_cast<const uint32_t*>(src - off);
        uint32_t w[5], bits = 0;
#pragma unroll
        for (int i = 0; i < 5; i++) w[i] = i * 4 < have ? wp[i] : 0u;
#pragma unroll
        for (int i = 0; i < 4; i++) bits |= nonzero4(__funnelshift_r(w[i], w[i + 1], 8 * off)) << (4 * i);
        return n < 16 ? bits & ((1u << n) - 1u) : bits;
    }
    uint32_t bits = 0;
    for (int i = 0; i < min(n, 16); i++) bits |= (row[int64_t(k0 + i) * p.sk] != 0 ? 1u : 0u) << i;
    return bits;
}

// One block per (mask batch, mask head, 128 query rows).  Bound: latency (32 x 256 x 256: 2 MB read, 0.3 written).
constexpr int kMaskThreads = 512;
__global__ void __launch_bounds__(kMaskThreads) mask_bits_kernel(MaskParams p) {
    __shared__ unsigned seen;
    if (threadIdx.x == 0) seen = 0u;
    grid_dep();
    if (blockIdx.x == 0)   // of this forward's projections nothing is known to be bad yet
        for (int i = threadIdx.x; i < p.batches; i += kMaskThreads) p.bad[i] = 0u;
    __syncthreads();
    const int tile = int(blockIdx.x) % p.tiles, bh = int(blockIdx.x) / p.tiles, r0 = tile * BQ, rows = min(BQ, p.rows - r0);
    const uint8_t* mh = p.mask + int64_t(bh / p.mh) * p.sb + int64_t(bh % p.mh) * p.sh;
    uint16_t* out = reinterpret_cast<uint16_t*>(p.bits + (int64_t(bh) * p.rows + r0) * p.words);
    const int per_row = p.words * 2, items = rows * per_row;
    unsigned mine = 0;
    for (int i = threadIdx.x; i < items; i += kMaskThreads) {
        const int rr = i / per_row, vv = i - rr * per_row;
        const uint8_t* row = mh + int64_t(r0 + rr) * p.sq;
        uint32_t w = 0;
        if (vv * 16 < p.Tk) {
            if (p.vec16) {
                const uint4 m = *reinterpret_cast<const uint4*>(row + vv * 16);
                w = nonzero4(m.x) | nonzero4(m.y) << 4 | nonzero4(m.z) << 8 | nonzero4(m.w) << 12;
            } else {
                w = mask16(p, row, vv * 16);
            }
        }
        out[i] = uint16_t(w);
        if (w) mine |= 1u << (vv * 16 / p.bkey);
    }
    mine = __reduce_or_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicOr(&seen, mine);
    __syncthreads();
    if (threadIdx.x == 0) p.need[blockIdx.x] = seen;
}

template <int BKEY>
__global__ void __launch_bounds__(kThreads, 2)
attn_f16_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_o, AttnF16Params p) {
    extern __shared__ unsigned char smem_raw[];
    using Smem = AttnF16Smem<BKEY>;
    Smem& s = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int CH = BKEY / 64;                 // 32-key chunks per softmax thread
    constexpr uint32_t kTmemCols = 256, kColO = BKEY, kTileBytes = 2 * BKEY * HD * 2;
    constexpr uint32_t kIdescS = umma_idesc_f16(BQ, BKEY), kMnB = 1u << 16;   // B of P·V is MN-major
    constexpr uint32_t kIdescO = umma_idesc_f16(BQ, HD) | kMnB, kIdescO2 = umma_idesc_f16(BQ, 2 * HD) | kMnB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int T = p.T;
    volatile int* abort_flag = &s.abort_flag;

    if (threadIdx.x == 0) {
        mbar_init(&s.bar_q, 1);
        mbar_init(&s.bar_k, 1);
        mbar_init(&s.bar_v, 1);
        mbar_init(&s.bar_s, 1);
        mbar_init(&s.bar_p, 8);
        mbar_init(&s.bar_o, 1);
        mbar_init(&s.bar_free, 4);
        s.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_kv);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s.tmem_base;
    grid_dep_wait();   // the set-up above ran under the previous kernel

    // Units are handed out back and forth, the last query tiles first: under a causal mask those are the long ones, and each CTA gets
    // its share of long and short ones.
    struct Unit { int b, h, q0; unsigned need; };
    auto unit_of = [&](int round, Unit& u) {
        const int n = (round & 1) ? (round + 1) * int(gridDim.x) - 1 - int(blockIdx.x) : round * int(gridDim.x) + int(blockIdx.x);
        if (n >= p.units) return false;
        const int per_tile = p.B * p.H, back = n / per_tile, bh = n - back * per_tile, tile = p.q_tiles - 1 - back;
        u.b = bh / p.H;
        u.h = bh - u.b * p.H;
        u.q0 = tile * BQ;
        // the key blocks that matter: those that some row sees, and those where 0 * inf has to reach the output
        u.need = __ldcg(p.need + u.b * p.need_sb + u.h * p.need_sh + tile * p.need_st) | __ldcg(p.bad + u.b);
        return true;
    };

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int t = 0;   // steps (key blocks) of all units so far
            Unit u;
            for (int r = 0; ok && unit_of(r, u); r++) {
                for (unsigned rem = u.need; ok && rem != 0; rem &= rem - 1, t++) {
                    const int blk = __ffs(rem) - 1;
                    if (t > 0) ok = mbar_wait(&s.bar_s, (t - 1) & 1, abort_flag);   // Q and K are free once S is done
                    if (!ok) break;
                    if (rem == u.need) {
                        mbar_expect_tx(&s.bar_q, uint32_t(sizeof(s.q)));
                        tma_load_4d(s.q, &map_q, p.q_col + u.h * HD, u.q0, u.b, 0, &s.bar_q);
                    }
                    mbar_expect_tx(&s.bar_k, kTileBytes);
                    tma_load_4d(s.k, &map_kv, p.k_col + u.h * HD, blk * BKEY, u.b, 0, &s.bar_k);
                    // V is free once P·V is done, and behind a unit once its context, staged there, has left
                    if (rem != u.need) ok = mbar_wait(&s.bar_o, (t - 1) & 1, abort_flag);
                    else if (r > 0) ok = mbar_wait(&s.bar_free, (r - 1) & 1, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(&s.bar_v, kTileBytes);
                    tma_load_4d(s.v, &map_kv, p.v_col + u.h * HD, blk * BKEY, u.b, 0, &s.bar_v);
                }
                if (ok && u.need == 0 && r > 0) ok = mbar_wait(&s.bar_free, (r - 1) & 1, abort_flag);   // phases are counted one by one
            }
            if (!ok) give_up(abort_flag, p.status, kErrAttnF16Load);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint64_t qd = umma_desc_k_major_bytes<128>(smem_u32(s.q[0])), kd = umma_desc_k_major_bytes<128>(smem_u32(s.k[0]));
            // V: rows of 128 bytes are keys, eight of them a group of 1024 bytes; the next 64 columns are those of the other plane
            const uint64_t vd = (umma_desc_k_major_bytes<128>(smem_u32(s.v)) & ~(uint64_t(0x3FFF) << 16)) | uint64_t(BKEY * HD * 2 >> 4) << 16;
            constexpr uint64_t kQLo = BQ * HD * 2 / 16, kKLo = BKEY * HD * 2 / 16;
            bool ok = true;
            int t = 0, q_loads = 0;
            Unit u;
            unsigned rem = 0;
            for (int r = 0; ok; t++) {
                while (rem == 0 && unit_of(r, u)) { rem = u.need; r++; }   // (a unit that sees nothing has no step)
                if (rem == 0) break;
                if (rem == u.need) ok = mbar_wait(&s.bar_q, q_loads++ & 1, abort_flag);
                rem &= rem - 1;
                ok = ok && mbar_wait(&s.bar_k, t & 1, abort_flag) && (t == 0 || mbar_wait(&s.bar_o, (t - 1) & 1, abort_flag));   // S goes where the last P was
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int kk = 0; kk < HD / 16; kk++) {   // the corrections first: fewer additions to the large sum
                    const uint64_t adv = uint64_t((kk * 32) >> 4);
                    umma_f16_ss<false>(tmem, qd + kQLo + adv, kd + adv, kIdescS, kk > 0 ? 1u : 0u);
                    umma_f16_ss<false>(tmem, qd + adv, kd + kKLo + adv, kIdescS, 1u);
                }
#pragma unroll
                for (int kk = 0; kk < HD / 16; kk++) umma_f16_ss<false>(tmem, qd + uint64_t((kk * 32) >> 4), kd + uint64_t((kk * 32) >> 4), kIdescS, 1u);
                umma_commit(&s.bar_s);
                ok = mbar_wait(&s.bar_v, t & 1, abort_flag) && mbar_wait(&s.bar_p, t & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int kk = 0; kk < BKEY / 16; kk++) {   // 16 keys = two groups of V rows = 2048 bytes
                    const uint32_t hi = tmem + uint32_t(kk * 16);
                    const uint64_t v = vd + uint64_t(kk * 2048 / 16);
                    // (the instruction descriptor names the element type)
                    umma_bf16_ts(tmem + kColO, hi, v, kIdescO2, kk > 0 ? 1u : 0u);
                    umma_bf16_ts(tmem + kColO + HD, hi + 8, v, kIdescO, 1u);
                }
                umma_commit(&s.bar_o);
            }
            if (!ok) give_up(abort_flag, p.status, kErrAttnF16P);
        }
    } else {
        const int quarter = warp & 3, half = (warp - kSoftWarp0) >> 2;   // a warp reads the lanes of tensor memory that its number names
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = uint32_t(quarter * 32) << 16;
        const uint32_t scol = tmem + lane_base + uint32_t(half * (BKEY / 2)), ocol = tmem + lane_base + kColO + uint32_t(half * 32);
        bool alive = true;   // warp-uniform; a warp that gave up keeps walking the loop so that pair_sync() stays matched
        uint32_t t = 0;
        Unit u;
        for (int r = 0; unit_of(r, u); r++) {
            const int b = u.b, h = u.h, qi = u.q0 + row;
            // on their way while the keys are walked (a round trip to L2 behind them costs 0.4 us where a CTA has one unit)
            auto fetch = [](float* dst, const float* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); };
            fetch(&s.vf[warp - kSoftWarp0][lane], p.v_factor + h * HD + half * 32 + lane);
            if (lane == 0) fetch(&s.vf[warp - kSoftWarp0][32], p.ctx_inv);
            // scores in the log2 domain; kept away from 0 and infinity, where -inf * c would not be -inf
            const float c = fminf(fmaxf(p.score_inv[h] * p.score_scale, 1.2e-38f), 3.0e38f);
            const uint32_t* row_bits = p.bits + b * p.bit_sb + h * p.bit_sh + int64_t(min(qi, T - 1)) * p.bit_sq + half * CH;
            float o[32];
#pragma unroll
            for (int j = 0; j < 32; j++) o[j] = 0.f;
            float m_run = -INFINITY, l_run = 0.f;
            for (unsigned rem = u.need; rem != 0; rem &= rem - 1, t++) {
                const uint32_t* src = row_bits + (__ffs(rem) - 1) * (BKEY / 32);
                uint32_t keep[CH];
                if constexpr (CH == 2) {
                    const uint2 k2 = *reinterpret_cast<const uint2*>(src);
                    keep[0] = k2.x; keep[CH - 1] = k2.y;
                } else {
                    keep[0] = *src;
                }
                const bool whole = warp_all((keep[0] & keep[CH - 1]) == 0xffffffffu);
                if (alive && !warp_all(mbar_wait(&s.bar_s, t & 1, abort_flag))) { give_up(abort_flag, p.status, kErrAttnF16S); alive = false; }
                // ---- pass 1: row maximum; masked scores become -inf ----
                float top = -INFINITY;
                if (alive) {
                    tc_fence_after();
#pragma unroll
                    for (int w = 0; w < CH; w++) {
                        uint32_t r[32];
                        tmem_ld32(scol + uint32_t(w * 32), r);
                        tmem_wait_ld();
                        if (!whole) {
#pragma unroll
                            for (int j = 0; j < 32; j++) r[j] = (keep[w] >> j) & 1u ? r[j] : 0xff800000u;
                            tmem_st32(scol + uint32_t(w * 32), r);
                        }
                        float t0 = -INFINITY, t1 = -INFINITY;   // NaN scores do not move the maximum; they reach the sum below
#pragma unroll
                        for (int j = 0; j < 32; j += 2) {
                            t0 = fmaxf(t0, __uint_as_float(r[j]));
                            t1 = fmaxf(t1, __uint_as_float(r[j + 1]));
                        }
                        top = fmaxf(top, fmaxf(t0, t1));
                    }
                    top *= c;
                    if (!whole) tmem_wait_st();
                }
                s.exch[t & 1][half][row] = top;
                pair_sync(quarter);
                const float m_new = fmaxf(m_run, fmaxf(top, s.exch[t & 1][half ^ 1][row]));
                const float m_safe = (m_new == -INFINITY) ? 0.f : m_new;
                const float alpha = fast_exp2(m_run - m_safe), off = 15.f - m_safe;
                // ---- pass 2: p * 2^15, its sum, and its two planes over the scores ----
                float sum0 = 0.f, sum1 = 0.f;
                if (alive) {
                    uint32_t next[16];
                    tmem_ld16(scol, next);
#pragma unroll
                    for (int w = 0; w < 2 * CH; w++) {   // sixteen keys at a time, the next sixteen on their way
                        uint32_t r[16], hi[8], lo[8];
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; j++) r[j] = next[j];
                        if (w + 1 < 2 * CH) tmem_ld16(scol + uint32_t(w * 16 + 16), next);
#pragma unroll
                        for (int j = 0; j < 16; j += 2) {
                            const float p0 = fast_exp2(fmaf(__uint_as_float(r[j]), c, off)), p1 = fast_exp2(fmaf(__uint_as_float(r[j + 1]), c, off));
                            sum0 += p0;
                            sum1 += p1;
                            split_f16x2(p0, p1, hi[j >> 1], lo[j >> 1]);
                        }
                        tmem_st8(scol + uint32_t(w * 16), hi);
                        tmem_st8(scol + uint32_t(w * 16 + 8), lo);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&s.bar_p);
                }
                l_run = fmaf(l_run, alpha, sum0 + sum1);   // this thread's share of the row sum; the two shares are added at the end
                m_run = m_new;
                if (alive && !warp_all(mbar_wait(&s.bar_o, t & 1, abort_flag))) { give_up(abort_flag, p.status, kErrAttnF16O); alive = false; }
                if (alive) {
                    tc_fence_after();
#pragma unroll
                    for (int w = 0; w < 2; w++) {
                        uint32_t r[16], e[16];
                        tmem_ld16(ocol + uint32_t(w * 16), r);
                        tmem_ld16(ocol + uint32_t(HD + w * 16), e);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; j++) o[w * 16 + j] = fmaf(o[w * 16 + j], alpha, __uint_as_float(r[j]) + __uint_as_float(e[j]));
                    }
                    tc_fence_before();
                }
            }
            if ((r + 1) * int(gridDim.x) >= p.units) grid_dep_launch();   // the last round
            s.exch[t & 1][half][row] = l_run;
            pair_sync(quarter);
            const float l_tot = s.exch[t & 1][0][row] + s.exch[t & 1][1][row];
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
            if (alive) {   // a fully masked row has o = 0 and l = 0: 0 * inf = NaN, as the reference softmax gives
                const float inv_l = 1.0f / l_tot;
                const float4* vf = reinterpret_cast<const float4*>(s.vf[warp - kSoftWarp0]);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float4 f = vf[j];
                    o[4 * j] *= inv_l * f.x; o[4 * j + 1] *= inv_l * f.y; o[4 * j + 2] *= inv_l * f.z; o[4 * j + 3] *= inv_l * f.w;
                }
                if (p.split == 0) {
                    if (qi < T) {
                        float* dst = p.ctx + (int64_t(b) * T + qi) * p.ld_ctx + int64_t(h) * HD + half * 32;
#pragma unroll
                        for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
                    }
                } else {
                    // Staged where V was (every P·V is done), 32 rows per quarter and plane, and stored by TMA, which leaves out the rows behind the
                    // last: sixteen bytes per lane and row kept the load / store unit busy for 4000 cycles.
                    char* stage = reinterpret_cast<char*>(s.v) + quarter * 8192 + lane * 128;
                    if (p.split == 2) {   // a convex combination of V rows fits the scale of V's largest column, which no masked row can move
                        if (h == 0 && half == 0 && qi < T) p.so_inv[int64_t(b) * T + qi] = s.vf[warp - kSoftWarp0][32];
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            uint4 hi, lo;
#pragma unroll
                            for (int e = 0; e < 4; e++) split_f16x2(o[8 * j + 2 * e], o[8 * j + 2 * e + 1], (&hi.x)[e], (&lo.x)[e]);
                            const int at = ((half * 4 + j) ^ (lane & 7)) << 4;
                            *reinterpret_cast<uint4*>(stage + at) = hi;
                            *reinterpret_cast<uint4*>(stage + 4096 + at) = lo;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            *reinterpret_cast<uint4*>(stage + (((half * 4 + j) ^ (lane & 7)) << 4)) =
                                make_uint4(pack_bf16x2(o[8 * j], o[8 * j + 1]), pack_bf16x2(o[8 * j + 2], o[8 * j + 3]), pack_bf16x2(o[8 * j + 4], o[8 * j + 5]), pack_bf16x2(o[8 * j + 6], o[8 * j + 7]));
                    }
                    fence_async_smem();
                }
            }
            pair_sync(quarter);
            if (half == 0 && lane == 0) {
                if (alive && p.split != 0) {
                    if (u.q0 + quarter * 32 < T) tma_store_4d(&map_o, reinterpret_cast<char*>(s.v) + quarter * 8192, h * HD, u.q0 + quarter * 32, b, 0);
                    bulk_commit();
                    bulk_wait_read<0>();
                }
                mbar_arrive(&s.bar_free);
            }
        }
        if (half == 0 && lane == 0) bulk_wait_all();
    }
    tc_fence_before();
    __syncthreads();
    let_copies_land(abort_flag);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// [planes][B][rows][cols] fp16, `ld` elements between rows; box = 64 columns (128 bytes, swizzled) x box_rows x all planes
int make_map(CUtensorMap* map, const uint16_t* base, int planes, int64_t plane, int64_t ld, int64_t rows, int64_t batches, int box_rows) {
    const auto fn = encode_tiled_fn();
    FXF_CHECK(fn != nullptr, "cuTensorMapEncodeTiled is not available from the CUDA driver");
    cuuint64_t dims[4] = {cuuint64_t(ld), cuuint64_t(rows), cuuint64_t(batches), cuuint64_t(planes)};
    cuuint64_t strides[3] = {cuuint64_t(ld) * 2, cuuint64_t(ld) * 2 * cuuint64_t(rows), cuuint64_t(planes > 1 ? plane : ld * rows * batches) * 2};
    cuuint32_t box[4] = {HD, cuuint32_t(box_rows), 1, cuuint32_t(planes)};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<uint16_t*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    FXF_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled (attention, split form) failed with code %d", int(r));
    return 0;
}

template <int BKEY>
int launch(const AttnArgs& a, const AttnSplit& sp, int Tk, AttnF16Params p, ExecCtx& ctx) {
    CUtensorMap mq, mk;
    if (make_map(&mq, sp.q, 2, sp.q_plane, a.ld_qkv, a.T, a.B, BQ)) return 1;
    if (make_map(&mk, sp.kv, 2, sp.kv_plane, a.kv ? a.ld_kv : a.ld_qkv, Tk, a.B, BKEY)) return 1;
    CUtensorMap mo = mq;
    if (p.split != 0 && make_map(&mo, a.split_ctx.planes, p.split, a.split_ctx.plane, a.ld_ctx, a.T, a.B, 32)) return 1;
    constexpr size_t smem = sizeof(AttnF16Smem<BKEY>) + 1024;
    static_assert(2 * (smem + 1024) <= 228 * 1024, "two CTAs of the attention kernel must fit one SM");
    static bool configured[64] = {};
    int dev = 0;
    FXF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        FXF_CUDA(cudaFuncSetAttribute(attn_f16_kernel<BKEY>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        FXF_CUDA(cudaFuncSetAttribute(attn_f16_kernel<BKEY>, cudaFuncAttributePreferredSharedMemoryCarveout, int(cudaSharedmemCarveoutMaxShared)));   // room for two CTAs
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    p.q_tiles = (a.T + BQ - 1) / BQ;
    p.units = p.q_tiles * a.B * a.H;
    dependent(attn_f16_kernel<BKEY>, dim3(unsigned(std::min(p.units, 2 * ctx.sm_count))), kThreads, smem, ctx)(mq, mk, mo, p);
    FXF_LAUNCHED(ctx);
    return 0;
}

}  // namespace

// The mask [.., rows, Tk] as bits: words of 32 keys, rows padded to whole key blocks; extents of 1 are not repeated.
int attention_f16_block(int64_t Tk) { return Tk > 64 ? 128 : 64; }
static void mask_extents(const FxfTensor& mask, int64_t* n) {
    for (int k = 0; k < 4; k++) n[k] = k + mask.rank >= 4 ? mask.shape[k + mask.rank - 4] : 1;
}
size_t mask_bits_bytes(const FxfTensor& mask, int64_t B, int64_t T, int64_t Tk) {
    int64_t n[4];
    mask_extents(mask, n);
    const size_t words = round_up(size_t(Tk), size_t(attention_f16_block(Tk))) / 32, tiles = n[2] == 1 ? 1 : size_t((T + BQ - 1) / BQ);
    return round_up(size_t(n[0] * n[1] * n[2]) * words * 4, 256) + round_up(size_t(n[0] * n[1]) * tiles * 4, 256) + round_up(size_t(B) * 4, 256);
}
MaskBits mask_bits_at(const FxfTensor& mask, int64_t B, int64_t T, int64_t Tk, void* area) {
    int64_t n[4];
    mask_extents(mask, n);
    const int64_t words = int64_t(round_up(size_t(Tk), size_t(attention_f16_block(Tk)))) / 32, tiles = n[2] == 1 ? 1 : (T + BQ - 1) / BQ;
    MaskBits m;
    m.batches = int(B);
    m.bits = static_cast<uint32_t*>(area);
    m.need = reinterpret_cast<uint32_t*>(static_cast<char*>(area) + round_up(size_t(n[0] * n[1] * n[2] * words) * 4, 256));
    m.bad = m.need + round_up(size_t(n[0] * n[1] * tiles) * 4, 256) / 4;
    m.bit_sq = n[2] == 1 ? 0 : words;
    m.bit_sh = n[1] == 1 ? 0 : n[2] * words;
    m.bit_sb = n[0] == 1 ? 0 : n[1] * n[2] * words;
    m.need_st = n[2] == 1 ? 0 : 1;
    m.need_sh = n[1] == 1 ? 0 : tiles;
    m.need_sb = n[0] == 1 ? 0 : n[1] * tiles;
    return m;
}
int launch_mask_bits(const FxfTensor& mask, int64_t T, int64_t Tk, const MaskBits& m, ExecCtx& ctx) {
    int64_t n[4], st[4];
    mask_extents(mask, n);
    for (int k = 0; k < 4; k++) st[k] = n[k] == 1 ? 0 : mask.stride[k + mask.rank - 4];
    MaskParams p{};
    p.mask = static_cast<const uint8_t*>(mask.ptr);
    p.sb = st[0]; p.sh = st[1]; p.sq = st[2]; p.sk = st[3];
    p.mh = int(n[1]); p.rows = int(n[2]); p.Tk = int(Tk); p.bkey = attention_f16_block(Tk);
    p.words = int(round_up(size_t(Tk), size_t(p.bkey))) / 32;
    p.tiles = n[2] == 1 ? 1 : int((T + BQ - 1) / BQ);
    p.vec16 = (p.sk == 1 && Tk % 16 == 0 && p.sb % 16 == 0 && p.sh % 16 == 0 && p.sq % 16 == 0 && aligned16(p.mask)) ? 1 : 0;
    p.contiguous = p.sk == 1 ? 1 : 0;
    p.bits = m.bits; p.need = m.need; p.bad = m.bad; p.batches = m.batches;
    const int64_t blocks = n[0] * n[1] * p.tiles;
    if (blocks == 0) return 0;
    tag_launch(ctx, "attention_mask_bits", 0, 1.125 * double(n[0] * n[1] * n[2]) * double(n[3]));
    dependent(mask_bits_kernel, dim3(unsigned(blocks)), kMaskThreads, 0, ctx)(p);
    FXF_LAUNCHED(ctx);
    return 0;
}

// Keys: as many as the bits of one word have blocks for.  A scale that is not positive would turn the order of the scores around.
bool attention_f16_ok(int64_t T, int64_t Tk, int64_t hd, float scale_divisor) {
    return hd == HD && T >= 1 && Tk >= 1 && Tk <= kMaxKeys && scale_divisor > 1e-30f && scale_divisor < 1e30f;
}

int launch_attention_f16(const AttnArgs& a, const AttnSplit& sp, ExecCtx& ctx) {
    const int Tk = a.kv ? a.Tk : a.T;
    const int64_t ldk = a.kv ? a.ld_kv : a.ld_qkv;
    FXF_CHECK(attention_f16_ok(a.T, Tk, a.hd, a.scale_divisor) && sp.q && sp.kv && aligned16(sp.q) && aligned16(sp.kv) && sp.q_plane % 8 == 0 && sp.kv_plane % 8 == 0 && a.ld_qkv % 8 == 0 &&
                  ldk % 8 == 0 && (a.q_off | a.k_off | a.v_off) % 8 == 0 && a.ld_ctx % 8 == 0 && sp.scales != nullptr && sp.mask != nullptr && sp.mask->bits != nullptr && int64_t(a.B) * a.H * ((a.T + BQ - 1) / BQ) < (1 << 30),
              "attention (split form): unsupported operands");
    FXF_CHECK(a.split_ctx.planes == nullptr || (aligned16(a.split_ctx.planes) && (a.split_ctx.plane * 2) % 16 == 0 && (a.split_bf16 || a.split_ctx.inv)), "attention: a context in split form needs 16-byte rows");
    AttnF16Params p{};
    const MaskBits& mb = *sp.mask;
    p.bits = mb.bits; p.need = mb.need;
    p.bit_sb = mb.bit_sb; p.bit_sh = mb.bit_sh; p.bit_sq = mb.bit_sq; p.need_sb = mb.need_sb; p.need_sh = mb.need_sh; p.need_st = mb.need_st;
    p.bad = mb.bad;
    p.ctx = a.ctx; p.B = a.B; p.T = a.T; p.Tk = Tk; p.H = a.H; p.ld_ctx = a.ld_ctx;
    p.q_col = int(a.q_off); p.k_col = int(a.k_off); p.v_col = int(a.v_off);
    p.split = a.split_ctx.planes == nullptr ? 0 : (a.split_bf16 ? 1 : 2);
    p.score_inv = sp.scales->score_inv; p.ctx_inv = sp.scales->ctx_inv;
    p.v_factor = p.split == 2 ? sp.scales->v_ctx : sp.scales->v_inv;
    p.score_scale = kLog2e / a.scale_divisor;
    p.so_inv = a.split_ctx.inv;
    p.status = ctx.status;
    tag_launch(ctx, "attention_f16x3_tcgen05", 4.0 * double(a.B) * a.H * double(a.T) * Tk * a.hd,
               4.0 * 2.0 * double(a.B) * (double(a.T) + Tk) * double(a.H) * a.hd + double(a.B) * a.T * Tk);
    return Tk > 64 ? launch<128>(a, sp, Tk, p, ctx) : launch<64>(a, sp, Tk, p, ctx);
}

}  // namespace fxf
