// Tensor-core GEMM for sm_100a on operands that are ALREADY in tensor-core form:
//     out[M,N] = act(x[M,K] · w[N,K]^T + bias[N])
// with fp32-grade results from three fp16 products per fp32 product ("f16x3"), or one bf16 product in the bf16 mode.
//
// Split form.  A row r of an fp32 matrix is stored as two fp16 planes and one power of two:
//     x[r,k] * s_r = hi[r,k] + lo[r,k],   s_r a power of two with max_k |x[r,k]| * s_r <= 2^15,
// hi = fp16(x * s_r), lo = fp16(x * s_r - hi): 22 significant bits for every element down to 2^-17 of the row's bound and an
// absolute error of at most 2^-39 of that bound below it (the TF32 kernels keep an exponent per element: a caller whose columns
// span more than that chooses them).  The bound is the row's maximum where the producer holds the row; a product's epilogue only
// knows max|x| * max ||w||_1 + max|b|, 2^6 to 2^8 times as much in the models here, and images share one scale over all channels.  An fp16 significand has the 11 bits of TF32, so
//     x·w = (hi·hi + hi·lo + lo·hi) / (s_x s_w)
// drops the same 2^-22 term as three TF32 products (and less than one TF32 product + two bf16 corrections, whose corrections
// are rounded at 2^-19), but a kind::f16 instruction covers K = 16 where a kind::tf32 instruction covers 8: three
// instructions per 16 K-elements instead of four or six, and 4 instead of 8 bytes per weight element.  The scales are powers
// of two, so multiplying by 1 / (s_x s_w) in the epilogue is exact.
// Both planes of [rows, K] take the bytes of the fp32 matrix: a tensor of the engine keeps its arena slot in either form.
//
// Who splits.  Weights: once per engine (split_rows_kernel, split_form.cu).  Activations: the kernel that produces them, where it knows a
// bound of each row: LayerNorm holds the row, and this kernel's own epilogue bounds its output rows by
//     |y[r,j]| <= amax_r * max_j ||w_j||_1 + max_j |b_j|
// (amax_r = max_k |x[r,k]|, kept beside the planes).  Anything else goes through split_rows_kernel first.
//
// Structure: persistent, one CTA per SM of 384 threads: warps 0-7 epilogue, warp 8 TMA producer, warp 9 MMA issuer (10 and 11
// complete the warpgroup that setmaxnreg takes registers from: a wide tile's epilogue holds 128 running sums), or 640 with sixteen
// epilogue warps (units of a single chain, see below).  Nothing
// touches an operand between TMA and the tensor core, so K-slabs are 64 deep (128-byte rows, one 3-D TMA load brings both
// planes of a tile).  PAIR: two CTAs of a cluster share a 256-row tile (cta_group::2), each staging half of the weight tile.
// Accumulation runs in chains of `chunk_slabs` K-slabs into one of two TMEM accumulators; the epilogue warps drain finished
// chains into fp32 registers (the tensor core adds with truncation: chains bound that error, see kChunkKDense).
// Launches are programmatic dependents: weight tiles of the first stages are requested before the previous kernel has
// finished, everything else waits for it.
// Every mbarrier wait is bounded; on expiry the CTA records an error in the status word and leaves.
//
// Bound: tensor pipe.  A 128 x 256 x 16 instruction takes 128 cycles, so a pair's 64-deep slab is 12 x 128 = 1536 cycles of
// tensor time against 64 KB of TMA writes and 144 KB of operand reads per SM (1625 cycles at 128 B per clock); the measured
// slab takes 1520.  Times on B200, before (one TF32 product + two bf16 corrections, operands split inside the kernel) and now:
// 8192 x 3072 x 768 133 -> 80 us (481 TFLOP/s; three times that is the library's bf16 rate under the power cap),
// 8192 x 768 x 768 57 -> 24 us, 1500 x 512 x 512 18 -> 7.8 us, 512 x 256 x 256 11 -> 4.5 us.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "../runtime.hpp"
#include "sm100.cuh"

namespace fxf {
namespace {

using namespace sm100;

constexpr int BM = 128, BK = 64;
constexpr int ACC = 2;
enum : int { kErrWaitFull = 131, kErrWaitEmpty = 133, kErrWaitAcc = 134, kErrWaitAccEmpty = 135, kErrWaitPartial = 136, kErrWaitResidual = 137, kErrWaitCluster = 138 };

// output staging buffers per epilogue warp, as far as the operand ring leaves room: a store may still be reading one (images:
// and the residual be on its way into two others)
constexpr int staging_buffers(int bn, int bnb, int stages, int npl, bool images, int warps) {
    const int room = 225 * 1024 - stages * npl * (BM + bnb) * BK * 2 - 32 * bn;
    const int fit = room / (warps * 2048), want = images ? 4 : 2;
    return fit < 1 ? 1 : (fit < want ? fit : want);
}

// BNB = weight rows held by this CTA; NPL = planes per operand (2: f16x3, 1: bf16)
template <int BN, int BNB, int STAGES, int NPL, int NSTG, int EW>
struct alignas(1024) F16Smem {
    uint16_t a[STAGES][NPL][BM * BK];
    uint16_t b[STAGES][NPL][BNB * BK];
    float stage_out[EW][NSTG][32 * 16];       // 32 rows x 16 columns per epilogue warp (64-byte rows, 64-byte swizzle)
    float col_inv[EW][BN * 4 / EW], col_bias[EW][BN * 4 / EW];   // 1 / scale and bias of a warp's columns
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
    uint64_t acc_full[ACC];
    uint64_t acc_empty[ACC];
    uint64_t res_full[EW][NSTG];
    uint64_t ready, received[EW];             // tiles cut along K inside a cluster: every CTA's products are done; a warp's partial blocks are here
    uint32_t tmem_base;
    int abort_flag;
};

// Images (IMG kernels): rows are the pixels of channels-last images, with one scale and one maximum per image (`rpi` rows)
// instead of per row; the maxima of the result are collected with atomics in so_amax[image], zeroed before the forward.
// c_slabs > 0: a convolution as an implicit GEMM.  K-slab k is input-channel slab k % c_slabs of filter tap k / c_slabs; the
// im2col mode of the TMA walks the 128 consecutive output pixels of a tile across row and image borders (stride and padding
// are in the map, the tap is the load's offset, pixels outside the image read zero), so tiles are full for any image size.
// c_slabs == 0: rows as they lie in memory (1x1 filters).
struct ImageGeom {
    unsigned rpi;
    int c_slabs, KW, WO, HO;
    int sw, sh, pw, ph, dw, dh;
    int lo_image;                 // images between the two planes of x
    const uint16_t* res;          // residual in split form, laid out like the result: res_inv / res_amax per image
    int64_t res_plane;
    const float *res_inv, *res_amax;
};

struct F16Params {
    ImageGeom im;
    const float* bias;
    const float* residual;        // optional, addressed like `out`
    const float *x_inv, *w_inv;   // 1 / scale per row of x and per row of w (NULL in bf16 mode)
    int64_t x_inv_stride;         // entries of x_inv between the rows of this product
    float* out;                   // NULL when the result leaves in split form
    int64_t M, N, K, ldo;
    int relu;
    int tma_out;                  // the result leaves through map_o (16-byte aligned rows): fp32 [M, N] or both planes of the split form
    int fast;                     // whole tiles take the short epilogue (rows in whole 32-byte sectors, of the residual too)
    int lean;                     // plain fp32 rows at any 4-byte address: whole tiles take the short epilogue for them
    int tiles_m, tiles_n, m_fastest;
    int full_tiles, tail_tiles, tail_split;   // tiles of the last round are cut along K into tail_split parts
    // > 1: a problem of one round whose tiles are cut inside clusters of that size, a part per CTA (tail_split of them).  A warp's block of the
    // tile, 32 rows x COLS columns, is finished by CTA (warp % cluster_k); the others send it theirs.
    int cluster_k;
    int chunk_slabs;
    int early_w;                  // weight tiles may be requested before the previous kernel has finished
    // Few rows against a large weight: the operands change places (map_x covers the weight, map_w the rows of x, BN = 32 or 64 of
    // them) so that the weight streams through full 128-row tiles; out[column * ldo + row], bias per row, scales as named.
    int swap;
    int64_t w_inv_stride;
    float* ws;
    int* flags;
    int* status;
    // split-form output [M, N]: planes (hi at 0, lo at so_plane), 1 / scale per row, and per row `so_parts` partial maxima
    // of |y| (one per column half of a tile); bounds of the row come from x_amax (x_parts per row) and w_bound = {max_j ||w_j||_1, max_j |b_j|}
    uint16_t* so;
    int64_t so_plane;
    float *so_inv, *so_amax;
    int so_parts;
    int so_cols;                  // columns come scaled, two fp16 planes (F16GemmArgs::col_inv)
    uint32_t* so_bad;
    int bad_rows, bad_block;
    const float *x_amax, *w_bound;
    int x_parts;
    // transposed column range (GemmArgs::vt_*)
    float* vt_out;
    unsigned char* vt_flags;
    int64_t vt_col0;
    int vt_T, vt_heads, vt_n32;
};

struct Unit { int tile, k0, k1, part, nparts, u; };
__device__ __forceinline__ Unit get_unit(const F16Params& p, int unit, int num_k) {
    Unit r;
    if (unit < p.full_tiles) {
        r.tile = unit; r.k0 = 0; r.k1 = num_k; r.part = 0; r.nparts = 1; r.u = 0;
    } else {
        r.u = unit - p.full_tiles;
        r.nparts = p.tail_split;
        r.tile = p.full_tiles + r.u / r.nparts;
        r.part = r.u % r.nparts;
        r.k0 = int(int64_t(num_k) * r.part / r.nparts);
        r.k1 = int(int64_t(num_k) * (r.part + 1) / r.nparts);
    }
    return r;
}
__device__ __forceinline__ void tile_coords(const F16Params& p, int tile, int& tm, int& tn) {
    if (p.m_fastest) {
        tm = tile % p.tiles_m;
        tn = tile / p.tiles_m;
    } else {
        tn = tile % p.tiles_n;
        tm = tile / p.tiles_n;
    }
}
// a wait counts only if it succeeded for every lane, so that a warp gives up as a whole
__device__ __forceinline__ bool warp_all(bool ok) { return __all_sync(0xffffffffu, ok) != 0; }

// v = sum[16 g ..], g known only at run time: a tree of branches (registers cannot be indexed)
template <int LO, int HI, int HALF>
__device__ __forceinline__ void pick_group(const float (&sum)[HALF], int g, float (&v)[16]) {
    if constexpr (HI - LO == 1) {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = sum[LO * 16 + j];
    } else {
        constexpr int MID = (LO + HI) / 2;
        if (g < MID) pick_group<LO, MID>(sum, g, v);
        else pick_group<MID, HI>(sum, g, v);
    }
}

template <int N>
struct Words { uint32_t w[N]; };
// 32 bytes of global memory at once: a whole sector per lane, so that lanes may own rows
__device__ __forceinline__ void load32(const void* p, Words<8>& r) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]), "=r"(r.w[7]) : "l"(p));
}
__device__ __forceinline__ void store32(void* p, const Words<8>& r) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r.w[0]), "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[3]), "r"(r.w[4]), "r"(r.w[5]), "r"(r.w[6]),
                 "r"(r.w[7]) : "memory");
}

// The larger of each half.  NaN wins among rows (a flag tells of it, and whatever reads the row is NaN); among images the finite
// maximum has to hold for the channels beside it.
template <bool IMG>
__device__ __forceinline__ __half2 larger_half2(__half2 a, __half2 b) { return IMG ? __hmax2(a, b) : __hmax2_nan(a, b); }

// 32 columns at a time (16 where the thread's registers are full of sums): the loads of a batch are in flight together
template <int HALF>
__device__ __forceinline__ void drain_chunk(uint32_t tacc, float (&sum)[HALF]) {
    constexpr int STEP = HALF <= 64 && HALF % 32 == 0 ? 32 : 16;
#pragma unroll
    for (int c = 0; c < HALF; c += STEP) {
        uint32_t r[STEP];
        tmem_ld(tacc + uint32_t(c), r);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < STEP; j++) sum[c + j] += __uint_as_float(r[j]);
    }
}

// sixteen bytes into the shared memory of a CTA of the cluster, counted on a barrier there (addresses of shared::cluster)
__device__ __forceinline__ void push16(uint32_t dst, float a, float b, float c, float d, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// EW epilogue warps: eight, or sixteen for units of a single chain, which need no registers for sums.  Those are short products
// (K <= 128) bound by the epilogue, where a scheduler with two of its warps issues an instruction every other cycle:
// 128 images of 56 x 56, 64 -> 256 channels with residual 215 -> 178 us (its bytes take 141 at 6.55 TB/s).
// CLUSTERS: tiles are cut along K inside clusters (F16Params::cluster_k); an instance of its own, because the code costs the others 0.4 us.
template <int BN, int STAGES, bool PAIR, int NPL, bool IMG, int EW, bool CLUSTERS>
__global__ void __launch_bounds__(EW * 32 + 128, 1)
gemm_f16_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_o, const __grid_constant__ CUtensorMap map_r, F16Params p) {
    extern __shared__ unsigned char smem_raw[];
    constexpr int BNB = PAIR ? BN / 2 : BN;
    constexpr int kStg = staging_buffers(BN, BNB, STAGES, NPL, IMG, EW);
    constexpr int kTmaWarp = EW, kMmaWarp = EW + 1, PARTS = EW / 4;
    using Smem = F16Smem<BN, BNB, STAGES, NPL, kStg, EW>;
    Smem& s = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr uint32_t kABytes = NPL * BM * BK * 2, kBBytes = NPL * BNB * BK * 2;
    constexpr uint32_t kIdesc = NPL == 2 ? umma_idesc_f16(PAIR ? 2 * BM : BM, BN) : umma_idesc_bf16(PAIR ? 2 * BM : BM, BN);
    static_assert(!CLUSTERS || (!PAIR && EW == 8 && NPL == 2), "instances for tiles cut inside clusters");
    constexpr uint32_t kTmemCols = ACC * BN <= 64 ? 64 : (ACC * BN <= 128 ? 128 : (ACC * BN <= 256 ? 256 : 512));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_k = int((p.K + BK - 1) / BK);
    const int num_units = p.full_tiles + p.tail_tiles * p.tail_split;
    const int chunk = p.chunk_slabs > 0 ? p.chunk_slabs : num_k;
    const int rank = PAIR ? int(cluster_ctarank()) : 0;
    const int sched_id = PAIR ? int(blockIdx.x >> 1) : int(blockIdx.x), sched_n = PAIR ? int(gridDim.x >> 1) : int(gridDim.x);
    volatile int* abort_flag = &s.abort_flag;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&s.full[i], 1);
            mbar_init(&s.empty[i], 1);
        }
        for (int i = 0; i < ACC; i++) {
            mbar_init(&s.acc_full[i], 1);
            mbar_init(&s.acc_empty[i], PAIR ? 2 * EW : EW);
        }
        if (IMG)
            for (int i = 0; i < EW * kStg; i++) mbar_init(&s.res_full[0][0] + i, 1);
        if (CLUSTERS) {
            mbar_init(&s.ready, uint32_t(p.cluster_k));
            for (int i = 0; i < EW; i++) mbar_init(&s.received[i], 1);
        }
        s.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kTmaWarp && lane == 0) {
        prefetch_tensormap(&map_x);
        prefetch_tensormap(&map_w);
        if (p.tma_out) prefetch_tensormap(&map_o);
        if (IMG && p.im.res != nullptr) prefetch_tensormap(&map_r);
    }
    if (warp == kMmaWarp) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)), "r"(kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)), "r"(kTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR || CLUSTERS) cluster_sync_all();   // the other CTA's barriers exist before anything of this CTA signals them
    tc_fence_after();
    const uint32_t tmem_base = s.tmem_base;

    // registers at launch: 384 x 168 = 256 x 208 + 128 x 88, 640 x 96 = 512 x 104 + 128 x 64
    if (warp >= EW) {
      if (BN >= 128) {
          if (EW == 16) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
          else asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
      }
      if (warp == kTmaWarp) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            int px = 0, py = 0, pn = 0;   // input position of the tile's first pixel
            auto locate = [&](int tm) {
                if (!IMG || p.im.c_slabs == 0) return;
                unsigned pix = unsigned(tm) * BM;
                if (pix >= unsigned(p.M)) pix = 0;   // the second tile of a pair may lie behind the last row: nothing of it is stored
                const unsigned n = pix / p.im.rpi, r = pix - n * p.im.rpi, oy = r / unsigned(p.im.WO), ox = r - oy * unsigned(p.im.WO);
                px = int(ox) * p.im.sw - p.im.pw;
                py = int(oy) * p.im.sh - p.im.ph;
                pn = int(n);
            };
            auto load_x = [&](int st, int k, int tm) {
                if (IMG && p.im.c_slabs > 0) {
                    const int tap = k / p.im.c_slabs, c = (k - tap * p.im.c_slabs) * BK, kh = tap / p.im.KW;
                    const uint16_t ow = uint16_t((tap - kh * p.im.KW) * p.im.dw), oh = uint16_t(kh * p.im.dh);
#pragma unroll
                    for (int pl = 0; pl < NPL; pl++) {
                        if (PAIR) tma_load_im2col_pair(s.a[st][pl], &map_x, c, px, py, pn + pl * p.im.lo_image, ow, oh, &s.full[st]);
                        else tma_load_im2col(s.a[st][pl], &map_x, c, px, py, pn + pl * p.im.lo_image, ow, oh, &s.full[st]);
                    }
                    return;
                }
                if (PAIR) tma_load_3d_pair(s.a[st], &map_x, k * BK, tm * BM, 0, &s.full[st]);
                else tma_load_3d(s.a[st], &map_x, k * BK, tm * BM, 0, &s.full[st]);
            };
            auto load_w = [&](int st, int k, int tn) {
                if (PAIR) tma_load_3d_pair(s.b[st], &map_w, k * BK, tn * BN + rank * BNB, 0, &s.full[st]);
                else tma_load_3d(s.b[st], &map_w, k * BK, tn * BN, 0, &s.full[st]);
            };
            auto announce = [&](int st) {   // the bytes of the whole stage (of both CTAs: the leader's barrier)
                if (!PAIR) mbar_expect_tx(&s.full[st], kABytes + kBBytes);
                else if (rank == 0) mbar_expect_tx(&s.full[st], 2 * (kABytes + kBBytes));
            };
            uint32_t it = 0;
            bool first = true;
            for (int unit = sched_id; unit < num_units; unit += sched_n) {
                const Unit un = get_unit(p, unit, num_k);
                int tm, tn;
                tile_coords(p, un.tile, tm, tn);
                if (PAIR) tm = tm * 2 + rank;
                locate(tm);
                int k = un.k0;
                if (first) {   // the ring is empty: fill it without waiting, the weights ahead of the previous kernel's end
                    const int pre = min(STAGES, un.k1 - un.k0);
                    if (!p.early_w) grid_dep_wait();
                    for (int i = 0; i < pre; i++) {
                        announce(i);
                        if (p.swap) load_x(i, un.k0 + i, tm);
                        else load_w(i, un.k0 + i, tn);
                    }
                    if (p.early_w) grid_dep_wait();
                    for (int i = 0; i < pre; i++) {
                        if (p.swap) load_w(i, un.k0 + i, tn);
                        else load_x(i, un.k0 + i, tm);
                    }
                    k += pre;
                    it += pre;
                    first = false;
                }
                for (; k < un.k1; k++, it++) {
                    const int st = it % STAGES;
                    if (it >= uint32_t(STAGES) && !mbar_wait(&s.empty[st], ((it / STAGES) - 1) & 1, abort_flag)) {
                        give_up(abort_flag, p.status, kErrWaitEmpty);
                        goto producer_done;
                    }
                    announce(st);
                    load_w(st, k, tn);
                    load_x(st, k, tm);
                }
            }
        producer_done:
            if (first) grid_dep_wait();
        }
      } else if (warp == kMmaWarp) {
        // ---------------- MMA issuer ----------------
        // The whole warp walks the loop, so the descriptors stay in uniform registers; one elected lane issues.
        if (rank == 0) {
            const uint32_t leader = elect_one();
            const uint64_t a0 = umma_desc_k_major_bytes<128>(smem_u32(s.a[0][0])), b0 = umma_desc_k_major_bytes<128>(smem_u32(s.b[0][0]));
            constexpr uint64_t kALo = (NPL - 1) * (BM * BK * 2 / 16), kBLo = (NPL - 1) * (BNB * BK * 2 / 16);   // lo plane, 16-byte units
            uint32_t st = 0, par = 0, ccount = 0;
            for (int unit = sched_id; unit < num_units; unit += sched_n) {
                const Unit un = get_unit(p, unit, num_k);
                for (int kc0 = un.k0; kc0 < un.k1; kc0 += chunk, ccount++) {
                    const int kc1 = min(kc0 + chunk, un.k1);
                    const uint32_t buf = ccount % ACC;
                    if (ccount >= uint32_t(ACC) &&
                        !warp_all(PAIR ? mbar_wait_cluster(&s.acc_empty[buf], ((ccount / ACC) - 1) & 1, abort_flag) : mbar_wait(&s.acc_empty[buf], ((ccount / ACC) - 1) & 1, abort_flag))) {
                        give_up(abort_flag, p.status, kErrWaitAccEmpty);
                        goto mma_done;
                    }
                    tc_fence_after();
                    const uint32_t acc = tmem_base + buf * uint32_t(BN);
                    for (int k = kc0; k < kc1; k++) {
                        if (!warp_all(mbar_wait(&s.full[st], par, abort_flag))) {
                            give_up(abort_flag, p.status, kErrWaitFull);
                            goto mma_done;
                        }
                        tc_fence_after();
                        if (leader) {
                            const uint64_t a = a0 + st * (kABytes / 16), b = b0 + st * (kBBytes / 16);
#pragma unroll
                            for (int kk = 0; kk < BK / 16; kk++) {   // 16 elements = 32 bytes per instruction inside the swizzle row
                                const uint64_t adv = uint64_t((kk * 32) >> 4);
                                const uint32_t acc_on = (k > kc0 || kk > 0) ? 1u : 0u;
                                if (NPL == 2) {
                                    umma_f16_ss<PAIR>(acc, a + kALo + adv, b + adv, kIdesc, acc_on);
                                    umma_f16_ss<PAIR>(acc, a + adv, b + kBLo + adv, kIdesc, 1u);
                                    umma_f16_ss<PAIR>(acc, a + adv, b + adv, kIdesc, 1u);
                                } else {
                                    umma_f16_ss<PAIR>(acc, a + adv, b + adv, kIdesc, acc_on);
                                }
                            }
                            if (PAIR) umma_commit_pair(&s.empty[st]);
                            else umma_commit(&s.empty[st]);
                            if (k + 1 == kc1) {
                                if (PAIR) umma_commit_pair(&s.acc_full[buf]);
                                else umma_commit(&s.acc_full[buf]);
                            }
                        }
                        if (++st == STAGES) { st = 0; par ^= 1; }
                    }
                }
            }
        mma_done:;
        }
      }
    } else {
        if (BN >= 128) {
            if (EW == 16) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
            else asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        }
        // ---------------- epilogue (warp w owns TMEM lanes 32*(w%4).. and column part w/4) ----------------
        // One thread owns one row of its warp's 32 x COLS block.  The group loop stays rolled (only picking a group's sixteen
        // running sums is spelled out): unrolled, its code missed the instruction cache at every group.  A group leaves as one
        // TMA store from a swizzled staging block; row-contiguous stores by the LSU, with the lanes re-arranged through shared
        // memory, took 250 instructions and 1900 cycles per group and bound every product of K <= 1024.
        constexpr int COLS = BN / PARTS, NSTG = kStg;
        // Narrow tiles belong to problems of a wave or two, where the store's latency counts (M = 512, N = 256, K = 256: 5.5 -> 4.4 us
        // with stores from registers); wide ones are stored by TMA, which a row per lane would keep the load / store unit busy for.
        constexpr bool DIRECT = !IMG && BN <= 64;
        static_assert(!IMG || NSTG >= 2, "a residual needs a staging buffer besides the one being stored");
        constexpr int AHEAD = NSTG >= 4 ? 2 : 1;   // images: groups between a residual's request and its use
        const int q = warp & 3, part = warp >> 2;
        const uint32_t lane_base = uint32_t(q * 32) << 16;
        float *cinv = s.col_inv[warp], *cbias = s.col_bias[warp];
        uint32_t ccount = 0, sbuf = 0, res_use = 0;   // chains, stored groups; parity of each residual buffer
        int have_tn = -1;
        const int M = int(p.M), N = int(p.N);
        grid_dep_wait();
        for (int unit = sched_id; unit < num_units; unit += sched_n) {
            const Unit un = get_unit(p, unit, num_k);
            int tm, tn;
            tile_coords(p, un.tile, tm, tn);
            if (PAIR) tm = tm * 2 + rank;
            const int owner = CLUSTERS ? warp % p.cluster_k : 0;   // of this warp's block
            const bool writes_partial = un.nparts > 1 && un.part != owner;
            const bool adds_partials = un.nparts > 1 && un.part == owner;
            const bool through_l2 = !CLUSTERS && un.nparts > 1;
            const int slot = PAIR ? un.u * 2 + rank : un.u, pstep = PAIR ? 2 : 1;
            // partial tiles: [column half][row quarter][4-column group][lane] float4, so that every access is coalesced
            float4* ws_mine = reinterpret_cast<float4*>(p.ws + size_t(slot) * size_t(BM * BN)) + warp * (COLS / 4) * 32 + lane;
            const int trow = tm * BM + q * 32, grow = trow + lane;   // first row of this warp, row of this thread
            const bool row_ok = grow < M;
            const int col_base = tn * BN + part * COLS;
            // constants of the row and of the columns, fetched while the tensor core works
            const int image = IMG ? int(unsigned(grow) / p.im.rpi) : 0;
            const int64_t sx = IMG ? image : grow * p.x_inv_stride;
            const int so_at = IMG ? image : grow;   // where the row's scales stand
            const float ri = (row_ok && p.x_inv != nullptr) ? p.x_inv[sx] : 1.f;
            const float res_inv = (IMG && p.im.res != nullptr && row_ok) ? p.im.res_inv[image] : 0.f;
            const float row_bias = (p.swap && row_ok && p.bias != nullptr) ? __ldg(p.bias + grow) : 0.f;
            float rscale = 1.f, rinv = 0.f;
            __half2 rmax = __half2half2(__ushort_as_half(0));   // largest |hi| of the row so far
            auto larger = [](__half2 a, __half2 b) { return larger_half2<IMG>(a, b); };
            if (NPL == 2 && p.so != nullptr && (IMG || !p.so_cols) && !writes_partial && row_ok) {
                float am = 0.f;
                for (int j = 0; j < p.x_parts; j++) am = fmaxf(am, p.x_amax[sx * p.x_parts + j]);
                float bound = fmaf(am, __ldg(p.w_bound), __ldg(p.w_bound + 1));
                if (IMG && p.im.res != nullptr) bound += p.im.res_amax[image];
                split_scale(bound, rscale, rinv);
                if (part == 0 && tn == 0 && (!IMG || unsigned(grow) == unsigned(image) * p.im.rpi)) p.so_inv[so_at] = rinv;
            }
            const bool fast = p.fast && !through_l2 && !writes_partial && (IMG || p.vt_out == nullptr || col_base < p.vt_col0);
            const int groups = writes_partial ? COLS / 16 : min(COLS, N - col_base + 15) / 16;   // warp-uniform; may be negative
            // the residual's next sixteen columns, requested ahead of their use: fp32 into registers, images into staging buffers
            Words<8> rn[2] = {};
            auto fetch_residual = [&](int col) {
                if (IMG || p.residual == nullptr || !row_ok || col >= N) return;
                const float* src = p.residual + int64_t(grow) * p.ldo + col;
                load32(src, rn[0]);
                load32(src + 8, rn[1]);
            };
            auto request_image = [&](int ahead) {   // lane 0: group `ahead` from the one in hand, counted over the tiles of this warp
                const uint32_t b = (sbuf + uint32_t(ahead)) % NSTG;
                bulk_wait_read<NSTG - 1 - AHEAD>();   // the store that last used the buffer has read it
                mbar_expect_tx(&s.res_full[warp][b], 2048);
                return b;
            };
            const bool image_res = IMG && fast && p.im.res != nullptr;
            if (fast) fetch_residual(col_base);
            if (image_res && lane == 0)
                for (int g = 0; g < min(AHEAD, groups); g++) {
                    const uint32_t b = request_image(g);
                    tma_load_3d(s.stage_out[warp][b], &map_r, col_base + g * 16, trow, 0, &s.res_full[warp][b]);
                }
            if (tn != have_tn) {
                __syncwarp();
                for (int j = lane; j < COLS; j += 32) {
                    const int c = col_base + j;
                    cinv[j] = (p.w_inv && c < N) ? p.w_inv[c * p.w_inv_stride] : 1.f;
                    cbias[j] = (p.bias && !p.swap && c < N) ? __ldg(p.bias + c) : 0.f;
                }
                __syncwarp();
                have_tn = tn;
            }
            // A unit of one chain is read from its accumulator group by group; of several, the sums are in registers.
            const bool single = EW == 16 || un.k1 - un.k0 <= chunk;
            const uint32_t tacc = tmem_base + (ccount % ACC) * uint32_t(BN) + lane_base + uint32_t(part * COLS);
            auto release = [&](uint32_t buf) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) mbar_arrive_leader(&s.acc_empty[buf]);
                    else mbar_arrive(&s.acc_empty[buf]);
                }
            };
            float sum[EW == 16 ? 16 : COLS];   // (a single chain keeps none)
            if (EW == 8 && !single) {
#pragma unroll
                for (int j = 0; j < COLS; j++) sum[j] = 0.f;
            }
            bool alive = true;
            for (int kc0 = un.k0; kc0 < un.k1; kc0 += chunk, ccount++) {
                const uint32_t buf = ccount % ACC;
                if (!warp_all(mbar_wait(&s.acc_full[buf], (ccount / ACC) & 1, abort_flag))) {
                    give_up(abort_flag, p.status, kErrWaitAcc);
                    alive = false;
                    break;
                }
                tc_fence_after();
                if constexpr (EW == 8) {
                    if (!single) {
                        drain_chunk<COLS>(tmem_base + buf * uint32_t(BN) + lane_base + uint32_t(part * COLS), sum);
                        release(buf);
                    }
                }
            }
            if (!alive) break;
            // The next kernel may become resident once every CTA has come to its last store; earlier, its blocks would pile up on the
            // SMs this launch leaves idle and run there one after the other.
            if (unit + sched_n >= num_units) grid_dep_launch();
            // Tiles cut inside a cluster.  The partial blocks travel into the operand ring of the CTA that finishes them, so everybody's products
            // have to be done first.  Blocks lie as [16-byte column group][lane].
            float4* inbox = nullptr;
            if constexpr (CLUSTERS) {
                constexpr uint32_t kBlock = 32 * COLS * 4;
                static_assert(12 * kBlock <= STAGES * (kABytes + kBBytes), "the operand ring holds what a CTA receives");
                const uint32_t cs = uint32_t(p.cluster_k), base = smem_u32(&s) + uint32_t(warp) / cs * (cs - 1) * kBlock;
                inbox = reinterpret_cast<float4*>(reinterpret_cast<char*>(&s) + uint32_t(warp) / cs * (cs - 1) * kBlock) + lane;
                const bool exists = trow < M && col_base < N;   // the same for every CTA of the cluster: nothing is sent of what will not be stored
                if (adds_partials && exists && lane == 0) mbar_expect_tx(&s.received[warp], (cs - 1) * kBlock);
                if (warp == 0 && uint32_t(lane) < cs) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_cta(smem_u32(&s.ready), uint32_t(lane))) : "memory");
                __syncwarp();
                bool ok = true;
                if (writes_partial) {
                    ok = warp_all(mbar_wait_cluster(&s.ready, 0, abort_flag));
                    if (ok && exists) {
                        const uint32_t slot = uint32_t(un.part) - (un.part > owner ? 1u : 0u);
                        const uint32_t dst = in_cta(base + slot * kBlock, uint32_t(owner)) + uint32_t(lane) * 16u, bar = in_cta(smem_u32(&s.received[warp]), uint32_t(owner));
                        auto send = [&](int g, float (&v)[16]) {
#pragma unroll
                            for (int j = 0; j < 4; j++) push16(dst + uint32_t(g * 4 + j) * 512u, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3], bar);
                        };
                        if (single) {
#pragma unroll 1
                            for (int g = 0; g < COLS / 16; g++) {
                                uint32_t r[16];
                                float v[16];
                                tmem_ld16(tacc + uint32_t(g * 16), r);
                                tmem_wait_ld();
#pragma unroll
                                for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
                                send(g, v);
                            }
                        } else {
#pragma unroll 1
                            for (int g = 0; g < COLS / 16; g++) {
                                float v[16];
                                pick_group<0, COLS / 16>(sum, g, v);
                                send(g, v);
                            }
                        }
                    }
                } else if (exists) {
                    ok = warp_all(mbar_wait_cluster(&s.received[warp], 0, abort_flag));
                }
                if (!ok) {
                    give_up(abort_flag, p.status, kErrWaitCluster);
                    break;
                }
                if (writes_partial) continue;   // (one unit per CTA: this ends the loop)
            }
            auto add_received = [&](int g, float (&v)[16]) {
                if constexpr (CLUSTERS) {
                    for (int r = 0; r + 1 < p.cluster_k; r++) {
                        const float4* src = inbox + r * (COLS / 4 * 32) + g * 4 * 32;
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const float4 w = src[j * 32];
                            v[4 * j] += w.x; v[4 * j + 1] += w.y; v[4 * j + 2] += w.z; v[4 * j + 3] += w.w;
                        }
                    }
                }
            };
            if (adds_partials && through_l2) {
                int ok = 1;
                if (lane == 0)
                    for (int pp = 1; pp < un.nparts && ok; pp++) ok = flag_wait(p.flags + (slot + pp * pstep) * EW + warp, abort_flag) ? 1 : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) {
                    give_up(abort_flag, p.status, kErrWaitPartial);
                    break;
                }
            }
            const bool transposes = !IMG && p.vt_out != nullptr && col_base >= p.vt_col0;
            // rows that do not start on 16-byte boundaries (a pitch like the 50257-column vocabulary): row r starts `shift` floats
            // past one and is stored as aligned 16-byte pieces, 16 columns lagging by `shift`
            float* orow = p.out + int64_t(grow) * p.ldo + col_base;
            const int shift = int((reinterpret_cast<uintptr_t>(orow) >> 2) & 3);
            float c0 = 0.f, c1 = 0.f, c2 = 0.f;   // the last three columns of the previous group
            // The common case, whole tiles that leave by TMA, without a branch but for the residual: with two warps per scheduler every
            // branch costs its latency (a group took 1500 cycles with all cases in one body).
            const float floor_at = p.relu ? 0.f : -INFINITY;
            auto finish_fast = [&](int g, float (&v)[16], auto form_tag) {
                constexpr int FORM = decltype(form_tag)::value;   // 0: fp32, 1: one bf16 plane, 2: two fp16 planes
                constexpr bool SPLIT = FORM != 0;
                const int col = col_base + g * 16;
                const Words<8> r0 = rn[0], r1 = rn[1];
                fetch_residual(g + 1 < COLS / 16 ? col + 16 : N);
                const uint32_t buf = sbuf % NSTG;
                char* stage = reinterpret_cast<char*>(s.stage_out[warp][buf]);
                if (image_res) {
                    if (lane == 0 && g + AHEAD < groups) {
                        const uint32_t b = request_image(AHEAD);
                        tma_load_3d(s.stage_out[warp][b], &map_r, col + AHEAD * 16, trow, 0, &s.res_full[warp][b]);
                    }
                    if (!warp_all(mbar_wait(&s.res_full[warp][buf], (res_use >> buf) & 1, abort_flag))) give_up(abort_flag, p.status, kErrWaitResidual);
                    res_use ^= 1u << buf;
                }
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 ci = *reinterpret_cast<const float4*>(cinv + g * 16 + j), cb = *reinterpret_cast<const float4*>(cbias + g * 16 + j);
                    // both factors are powers of two; the weight's goes first: the product of the two may leave the range of fp32
                    v[j] = fmaf(v[j] * ci.x, ri, cb.x); v[j + 1] = fmaf(v[j + 1] * ci.y, ri, cb.y);
                    v[j + 2] = fmaf(v[j + 2] * ci.z, ri, cb.z); v[j + 3] = fmaf(v[j + 3] * ci.w, ri, cb.w);
                }
                if (image_res) {
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int at = lane * 32 + ((j ^ ((lane >> 2) & 1)) << 4);
                        const uint4 hq = *reinterpret_cast<const uint4*>(stage + at), lq = *reinterpret_cast<const uint4*>(stage + 1024 + at);
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const uint32_t hw = (&hq.x)[e], lw = (&lq.x)[e];
                            const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hw)), l = __half22float2(*reinterpret_cast<const __half2*>(&lw));
                            v[8 * j + 2 * e] = fmaf(h.x + l.x, res_inv, v[8 * j + 2 * e]);
                            v[8 * j + 2 * e + 1] = fmaf(h.y + l.y, res_inv, v[8 * j + 2 * e + 1]);
                        }
                    }
                } else if (!IMG && !SPLIT && p.residual != nullptr) {
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        v[j] += __uint_as_float(r0.w[j]);
                        v[8 + j] += __uint_as_float(r1.w[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = max_keep_nan(v[j], floor_at);
                if constexpr (DIRECT) {
                    Words<8> o0, o1;
                    if constexpr (!SPLIT) {
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            o0.w[j] = __float_as_uint(v[j]);
                            o1.w[j] = __float_as_uint(v[8 + j]);
                        }
                        if (row_ok) {
                            float* dst = p.out + int64_t(grow) * p.ldo + col;
                            store32(dst, o0);
                            store32(dst + 8, o1);
                        }
                    } else if constexpr (FORM == 1) {
#pragma unroll
                        for (int j = 0; j < 8; j++) o0.w[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
                        if (row_ok) store32(p.so + int64_t(grow) * N + col, o0);
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            split_f16x2(v[2 * j] * rscale, v[2 * j + 1] * rscale, o0.w[j], o1.w[j]);
                            rmax = larger(rmax, __habs2(*reinterpret_cast<const __half2*>(&o0.w[j])));
                        }
                        if (row_ok) {
                            uint16_t* dst = p.so + int64_t(grow) * N + col;
                            store32(dst, o0);
                            store32(dst + p.so_plane, o1);
                        }
                    }
                    return;
                }
                if (!image_res) {
                    if (lane == 0) bulk_wait_read<NSTG - 1>();   // the store that used this buffer has read it
                    __syncwarp();
                }
                if constexpr (!SPLIT) {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        *reinterpret_cast<float4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                } else if constexpr (FORM == 1) {
#pragma unroll
                    for (int j = 0; j < 2; j++)
                        *reinterpret_cast<uint4*>(stage + lane * 32 + ((j ^ ((lane >> 2) & 1)) << 4)) =
                            make_uint4(pack_bf16x2(v[8 * j], v[8 * j + 1]), pack_bf16x2(v[8 * j + 2], v[8 * j + 3]), pack_bf16x2(v[8 * j + 4], v[8 * j + 5]), pack_bf16x2(v[8 * j + 6], v[8 * j + 7]));
                } else {
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        uint4 hi, lo;
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            split_f16x2(v[8 * j + 2 * e] * rscale, v[8 * j + 2 * e + 1] * rscale, (&hi.x)[e], (&lo.x)[e]);
                            rmax = larger(rmax, __habs2(*reinterpret_cast<const __half2*>(&hi.x + e)));
                        }
                        const int at = lane * 32 + ((j ^ ((lane >> 2) & 1)) << 4);
                        *reinterpret_cast<uint4*>(stage + at) = hi;
                        *reinterpret_cast<uint4*>(stage + 1024 + at) = lo;
                    }
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (trow < M) tma_store_3d(&map_o, stage, col, trow, 0);
                    bulk_commit();
                }
                sbuf++;
            };
            // The same for rows that do not start on 16-byte boundaries: row r starts `off` floats past a boundary of PIECE floats and leaves as
            // aligned pieces of that size, sixteen columns lagging by `off`; the PIECE - off first and the off last columns of the block on
            // their own.  (8192 x 50257 x 768, the logits of a 50257-word vocabulary: 1500 -> 1350 us with pieces of sixteen bytes.)  bf16
            // products, whose epilogue shows, take whole sectors: half as many stores, and none that fills a sector in part (4096 x
            // 50257 x 768 435 -> 395 us); where the products are three the longer code costs more than it gives.
            constexpr bool LEAN = !IMG && BN >= 128;   // (its code costs the one-wave problems of the narrow tiles 0.3 us)
            constexpr int PIECE = NPL == 1 ? 8 : 4, PIECES = 16 / PIECE, ROWS_AT_ONCE = 32 / PIECES;   // pieces per row and group, rows per store
            const bool lean = LEAN && p.lean && un.nparts == 1 && col_base + COLS <= N && (p.vt_out == nullptr || col_base < p.vt_col0);
            const int off = int((reinterpret_cast<uintptr_t>(orow) >> 2) & (PIECE - 1));
            float last[PIECE - 1] = {};   // the last columns of the previous group
            float* piece_at[PIECES];      // this lane's pieces of the group in hand: rows i * ROWS_AT_ONCE + lane / PIECES
            uint32_t piece_ok = 0, piece_left = 0;   // bit i: the row exists; its first piece belongs to the block on the left
            if (lean) {
#pragma unroll
                for (int i = 0; i < PIECES; i++) {
                    const int gr = trow + i * ROWS_AT_ONCE + lane / PIECES;
                    float* rp = p.out + int64_t(gr) * p.ldo + col_base;
                    const int c = (lane % PIECES) * PIECE - int((reinterpret_cast<uintptr_t>(rp) >> 2) & (PIECE - 1));
                    piece_at[i] = rp + c;
                    piece_ok |= (gr < M ? 1u : 0u) << i;
                    piece_left |= (c < 0 ? 1u : 0u) << i;
                }
            }
            auto finish_lean = [&](int g, float (&v)[16]) {
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 ci = *reinterpret_cast<const float4*>(cinv + g * 16 + j), cb = *reinterpret_cast<const float4*>(cbias + g * 16 + j);
                    v[j] = max_keep_nan(fmaf(v[j] * ci.x, ri, cb.x), floor_at); v[j + 1] = max_keep_nan(fmaf(v[j + 1] * ci.y, ri, cb.y), floor_at);
                    v[j + 2] = max_keep_nan(fmaf(v[j + 2] * ci.z, ri, cb.z), floor_at); v[j + 3] = max_keep_nan(fmaf(v[j + 3] * ci.w, ri, cb.w), floor_at);
                }
                // w[k] = column 16 g - off + k = entry k + (PIECE - 1 - off) of {the previous PIECE - 1, v}, by halving steps
                float w[16 + PIECE - 1];
                const int by = PIECE - 1 - off;
#pragma unroll
                for (int k = 0; k < PIECE - 1; k++) w[k] = last[k];
#pragma unroll
                for (int k = 0; k < 16; k++) w[PIECE - 1 + k] = v[k];
#pragma unroll
                for (int step = PIECE / 2, n = 16 + PIECE - 1; step > 0; step >>= 1) {
                    n -= step;
                    const bool move = (by & step) != 0;
#pragma unroll
                    for (int k = 0; k < n; k++) w[k] = move ? w[k + step] : w[k];
                }
#pragma unroll
                for (int k = 0; k < PIECE - 1; k++) last[k] = v[16 - (PIECE - 1) + k];
                if (row_ok && off > 0) {
                    if (g == 0) {
#pragma unroll
                        for (int k = 0; k < PIECE - 1; k++)
                            if (k < PIECE - off) orow[k] = v[k];
                    }
                    if (g + 1 == COLS / 16) {
#pragma unroll
                        for (int k = 0; k < PIECE - 1; k++)
                            if (k < off) orow[COLS - 1 - k] = v[15 - k];
                    }
                }
                char* stage = reinterpret_cast<char*>(s.stage_out[warp][0]);
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; j++)
                    *reinterpret_cast<float4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_float4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
                __syncwarp();
                const uint32_t skip = g == 0 ? piece_left : 0u;
#pragma unroll
                for (int i = 0; i < PIECES; i++) {
                    const int rr = i * ROWS_AT_ONCE + lane / PIECES, first = (lane % PIECES) * (PIECE / 4), swz = (rr >> 1) & 3;
                    if constexpr (PIECE == 4) {
                        const float4 x = *reinterpret_cast<const float4*>(stage + rr * 64 + ((first ^ swz) << 4));
                        if ((piece_ok & ~skip) >> i & 1u) *reinterpret_cast<float4*>(piece_at[i] + g * 16) = x;
                    } else {
                        const uint4 x = *reinterpret_cast<const uint4*>(stage + rr * 64 + ((first ^ swz) << 4)), y = *reinterpret_cast<const uint4*>(stage + rr * 64 + (((first + 1) ^ swz) << 4));
                        Words<8> r;
                        r.w[0] = x.x; r.w[1] = x.y; r.w[2] = x.z; r.w[3] = x.w; r.w[4] = y.x; r.w[5] = y.y; r.w[6] = y.z; r.w[7] = y.w;
                        if ((piece_ok & ~skip) >> i & 1u) store32(piece_at[i] + g * 16, r);
                    }
                }
            };
            // sixteen columns: scales, bias, residual, activation, store
            auto finish = [&](int g, float (&v)[16]) {
                const int col = col_base + g * 16;
                if (writes_partial) {   // (through L2)
#pragma unroll
                    for (int j = 0; j < 4; j++) ws_mine[(g * 4 + j) * 32] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    return;
                }
                if (adds_partials && through_l2) {
#pragma unroll 1
                    for (int pp = 1; pp < un.nparts; pp++) {
                        const float4* src = ws_mine + size_t(pp * pstep) * size_t(BM * BN / 4) + g * 4 * 32;
                        float4 w[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) w[j] = __ldcg(src + j * 32);
#pragma unroll
                        for (int j = 0; j < 4; j++) { v[4 * j] += w[j].x; v[4 * j + 1] += w[j].y; v[4 * j + 2] += w[j].z; v[4 * j + 3] += w[j].w; }
                    }
                }
                float4 r4[4];
                if (!IMG && p.residual != nullptr && p.tma_out) {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        r4[j] = (row_ok && col + 4 * j < N) ? *reinterpret_cast<const float4*>(p.residual + int64_t(grow) * p.ldo + col + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 ci = *reinterpret_cast<const float4*>(cinv + g * 16 + j), cb = *reinterpret_cast<const float4*>(cbias + g * 16 + j);
                    // both factors are powers of two; the weight's goes first: the product of the two may leave the range of fp32
                    v[j] = fmaf(v[j] * ci.x, ri, cb.x); v[j + 1] = fmaf(v[j + 1] * ci.y, ri, cb.y);
                    v[j + 2] = fmaf(v[j + 2] * ci.z, ri, cb.z); v[j + 3] = fmaf(v[j + 3] * ci.w, ri, cb.w);
                }
                if (!IMG && p.swap) {   // the 32 lanes write 32 consecutive columns of the result
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (row_ok && col + j < N) {
                            const int64_t off = int64_t(col + j) * p.ldo + grow;
                            float t = v[j] + row_bias;
                            if (p.residual != nullptr) t += p.residual[off];
                            p.out[off] = p.relu ? relu_keep_nan(t) : t;
                        }
                    return;
                }
                if (transposes) {
                    // V third of a packed QKV projection, transposed per head: the 32 lanes write 32 consecutive keys of a V^T row
                    const int b = grow / p.vt_T, t = grow - b * p.vt_T, v0 = col - int(p.vt_col0), h = v0 >> 6, d0 = v0 & 63;
                    float* dst = p.vt_out + ((int64_t(b) * p.vt_heads + h) * 64 + d0) * int64_t(p.vt_T) + t;
                    bool bad = false;
#pragma unroll
                    for (int d = 0; d < 16; d++) {
                        bad = bad || (v[d] - v[d] != 0.f);   // NaN or infinity
                        if (row_ok) dst[int64_t(d) * p.vt_T] = v[d];
                    }
                    const unsigned any_bad = __ballot_sync(0xffffffffu, row_ok && bad);
                    if (lane == 0 && row_ok) {
                        unsigned char* fl = p.vt_flags + ((int64_t(b) * p.vt_heads + h) * 2 + (d0 >> 5)) * p.vt_n32 + (t >> 5);
                        *fl = (any_bad != 0 || ((d0 & 16) && *fl != 0)) ? 1 : 0;   // two groups share a flag, in this order
                    }
                    return;
                }
                if (IMG && p.im.res != nullptr && row_ok) {
#pragma unroll
                    for (int j = 0; j < 16; j += 8)
                        if (col + j < N) {
                            const uint16_t* src = p.im.res + int64_t(grow) * N + col + j;
                            const uint4 hq = *reinterpret_cast<const uint4*>(src), lq = *reinterpret_cast<const uint4*>(src + p.im.res_plane);
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                const uint32_t hw = (&hq.x)[e], lw = (&lq.x)[e];
                                const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hw)), l = __half22float2(*reinterpret_cast<const __half2*>(&lw));
                                v[j + 2 * e] = fmaf(h.x + l.x, res_inv, v[j + 2 * e]);
                                v[j + 2 * e + 1] = fmaf(h.y + l.y, res_inv, v[j + 2 * e + 1]);
                            }
                        }
                }
                if (!IMG && p.residual != nullptr) {
                    if (p.tma_out) {
#pragma unroll
                        for (int j = 0; j < 4; j++) { v[4 * j] += r4[j].x; v[4 * j + 1] += r4[j].y; v[4 * j + 2] += r4[j].z; v[4 * j + 3] += r4[j].w; }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (row_ok && col + j < N) v[j] += p.residual[int64_t(grow) * p.ldo + col + j];
                    }
                }
                if (p.relu) {
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = relu_keep_nan(v[j]);
                }
                char* stage = reinterpret_cast<char*>(s.stage_out[warp][sbuf % NSTG]);
                if (IMG || p.tma_out) {
                    if (lane == 0) bulk_wait_read<NSTG - 1>();   // the store that used this buffer has read it
                    __syncwarp();
                    if (p.so == nullptr) {
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            *reinterpret_cast<float4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    } else if (NPL == 1 && !p.so_cols) {
#pragma unroll
                        for (int j = 0; j < 2; j++)
                            *reinterpret_cast<uint4*>(stage + lane * 32 + ((j ^ ((lane >> 2) & 1)) << 4)) =
                                make_uint4(pack_bf16x2(v[8 * j], v[8 * j + 1]), pack_bf16x2(v[8 * j + 2], v[8 * j + 3]), pack_bf16x2(v[8 * j + 4], v[8 * j + 5]), pack_bf16x2(v[8 * j + 6], v[8 * j + 7]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            uint4 hi, lo;
                            uint32_t* hp = &hi.x;
                            uint32_t* lp = &lo.x;
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                const float x = v[8 * j + 2 * e], y = v[8 * j + 2 * e + 1];
                                split_f16x2(x * rscale, y * rscale, hp[e], lp[e]);
                                rmax = larger(rmax, __habs2(*reinterpret_cast<const __half2*>(hp + e)));
                            }
                            const int at = lane * 32 + ((j ^ ((lane >> 2) & 1)) << 4);
                            *reinterpret_cast<uint4*>(stage + at) = hi;
                            *reinterpret_cast<uint4*>(stage + 1024 + at) = lo;
                        }
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (trow < M) tma_store_3d(&map_o, stage, col, trow, 0);
                        bulk_commit();
                    }
                    sbuf++;
                    return;
                }
                // ---- unaligned rows: out[k] = column 16g - shift + k of the row, by two select steps over {previous three, v} ----
                float u[18], w[16];
                {
                    const bool s1 = shift & 1, s2 = shift & 2;
                    u[0] = s1 ? c0 : c1; u[1] = s1 ? c1 : c2; u[2] = s1 ? c2 : v[0];
#pragma unroll
                    for (int k = 3; k < 18; k++) u[k] = s1 ? v[k - 3] : v[k - 2];
#pragma unroll
                    for (int k = 0; k < 16; k++) w[k] = s2 ? u[k] : u[k + 2];
                }
                if (row_ok && shift > 0) {   // the 4 - shift leading and the shift trailing columns of this block's row segment
                    if (g == 0) {
                        if (col < N) orow[0] = v[0];
                        if (shift < 3 && col + 1 < N) orow[1] = v[1];
                        if (shift < 2 && col + 2 < N) orow[2] = v[2];
                    }
                    if (g + 1 == COLS / 16 || col + 16 >= N) {
                        if (col + 15 < N) orow[g * 16 + 15] = v[15];
                        if (shift > 1 && col + 14 < N) orow[g * 16 + 14] = v[14];
                        if (shift > 2 && col + 13 < N) orow[g * 16 + 13] = v[13];
                    }
                }
                c0 = v[13]; c1 = v[14]; c2 = v[15];
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; j++)
                    *reinterpret_cast<float4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_float4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
                __syncwarp();
                const int piece = lane & 3;
#pragma unroll
                for (int i = 0; i < 4; i++) {   // 4 lanes cover a row's 64 bytes, 8 rows per instruction
                    const int rr = i * 8 + (lane >> 2);
                    const int gr = trow + rr;
                    float* rp = p.out + int64_t(gr) * p.ldo + col;
                    const int a = int((reinterpret_cast<uintptr_t>(rp) >> 2) & 3), c = piece * 4 - a;
                    const float4 x = *reinterpret_cast<const float4*>(stage + rr * 64 + ((piece ^ ((rr >> 1) & 3)) << 4));
                    if (gr >= M || (g == 0 && c < 0)) continue;   // the piece left of the block belongs to the neighbour
                    if (col + c + 3 < N) {
                        *reinterpret_cast<float4*>(rp + c) = x;
                    } else {
                        if (col + c < N) rp[c] = x.x;
                        if (col + c + 1 < N) rp[c + 1] = x.y;
                        if (col + c + 2 < N) rp[c + 2] = x.z;
                    }
                }
            };
            auto all_groups = [&](auto&& group) {
                if (single) {
                    uint32_t acc[16];
                    tmem_ld16(tacc, acc);
                    tmem_wait_ld();
#pragma unroll 1
                    for (int g = 0; g < groups; g++) {
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = __uint_as_float(acc[j]);
                        tmem_ld16(tacc + uint32_t(min(g + 1, COLS / 16 - 1) * 16), acc);   // the next group's, behind this one's work
                        if constexpr (CLUSTERS) add_received(g, v);
                        group(g, v);
                        tmem_wait_ld();
                    }
                    release((ccount - 1) % ACC);
                } else if constexpr (EW == 8) {
#pragma unroll 1
                    for (int g = 0; g < groups; g++) {
                        float v[16];
                        pick_group<0, COLS / 16>(sum, g, v);
                        if constexpr (CLUSTERS) add_received(g, v);
                        group(g, v);
                    }
                }
            };
            if (fast) {
                if (p.so == nullptr) {
                    all_groups([&](int g, float (&v)[16]) { finish_fast(g, v, std::integral_constant<int, 0>()); });
                } else if constexpr (NPL == 1) {
                    if (p.so_cols) all_groups([&](int g, float (&v)[16]) { finish_fast(g, v, std::integral_constant<int, 2>()); });
                    else all_groups([&](int g, float (&v)[16]) { finish_fast(g, v, std::integral_constant<int, 1>()); });
                } else {
                    all_groups([&](int g, float (&v)[16]) { finish_fast(g, v, std::integral_constant<int, 2>()); });
                }
            } else if (lean) {
                if constexpr (LEAN) all_groups(finish_lean);
            } else {
                all_groups(finish);
            }
            if (!IMG && p.so_cols) {
                if (row_ok && !writes_partial && p.so_bad != nullptr && !(__low2float(rmax) <= 65504.f && __high2float(rmax) <= 65504.f))
                    atomicOr(p.so_bad + grow / p.bad_rows, 1u << (grow % p.bad_rows / p.bad_block));
            } else if (NPL == 2 && p.so != nullptr && !writes_partial) {
                // hi is within 2^-11 of the value; an infinite one must not take the scale of its whole image along
                const float top = fminf(fmaxf(__low2float(rmax), __high2float(rmax)) * 1.0005f, 32768.f) * rinv;
                if (!IMG) {
                    if (row_ok) p.so_amax[int64_t(grow) * p.so_parts + tn * PARTS + part] = top;
                } else {   // one atomic per image among the warp's rows (an atomic per row: 85 us instead of 60 for 7 x 7 images)
                    const unsigned same = __match_any_sync(0xffffffffu, row_ok ? image : -1);
                    const unsigned all = __reduce_max_sync(same, __float_as_uint(top));   // non-negative floats order like integers
                    if (row_ok && lane == __ffs(same) - 1) atomicMax(reinterpret_cast<unsigned*>(p.so_amax) + image, all);
                }
            }
            if (through_l2 && writes_partial) {
                __threadfence();
                __syncwarp();
                if (lane == 0) flag_set(p.flags + slot * EW + warp, 1);
            } else if (through_l2 && adds_partials) {
                __syncwarp();
                if (lane == 0)
                    for (int pp = 1; pp < un.nparts; pp++) flag_set(p.flags + (slot + pp * pstep) * EW + warp, 0);
            }
        }
        if (p.tma_out && lane == 0) bulk_wait_all();
    }
    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    let_copies_land(abort_flag);
    if (PAIR || CLUSTERS) cluster_sync_all();   // nobody leaves while another may still send here
    if (warp == kMmaWarp) {
        tc_fence_after();
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// ---- host side -------------------------------------------------------------------------------------
int make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld, int64_t plane, int planes, int box_rows) {
    const CUresult r = encode_planes(map, base, rows, cols, ld, plane, planes, BK, box_rows);
    FXF_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled (f16) failed with code %d (rows %lld cols %lld planes %d)", int(r), (long long)rows, (long long)cols, planes);
    return 0;
}

// the result as the epilogue stores it: boxes of 32 rows x 16 columns, fp32 (64-byte rows) or split form (32-byte rows, all planes)
int make_out_map(CUtensorMap* map, const F16GemmArgs& a, int planes) {
    if (a.col_inv != nullptr) planes = 2;
    const auto fn = encode_tiled_fn();
    FXF_CHECK(fn != nullptr, "cuTensorMapEncodeTiled is not available from the CUDA driver");
    const bool split = a.split_out.planes != nullptr;
    const cuuint64_t esz = split ? 2 : 4, pitch = cuuint64_t(split ? a.N : a.ldo) * esz;
    cuuint64_t dims[3] = {cuuint64_t(a.N), cuuint64_t(a.M), cuuint64_t(split ? planes : 1)};
    cuuint64_t strides[2] = {pitch, split && planes > 1 ? cuuint64_t(a.split_out.plane) * 2 : pitch * cuuint64_t(a.M)};
    cuuint32_t box[3] = {16, 32, cuuint32_t(split ? planes : 1)};
    cuuint32_t estr[3] = {1, 1, 1};
    void* base = split ? static_cast<void*>(a.split_out.planes) : static_cast<void*>(a.out);
    CUresult r = fn(map, split ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    split ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    FXF_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled (f16 output) failed with code %d", int(r));
    return 0;
}

// K-elements per accumulation chain.  Convolutions run 50 deep without normalisation: ResNet-50's logits lie 1.1e-5 from fp64 with
// chains of 128 (5.7e-6 with 64; three TF32 products in chains of 64: 1.4e-5), and a chain of 64 drains at every slab
// (128 images of 56 x 56, 64 channels, 3x3: 136 against 114 us).
// The tensor core truncates at every addition, so chains bound the error.  Tiles of up to 64 columns drain 32 sums per thread at most:
// chains of 256 cost them nothing (us per launch in a chain, 256 against 1024: 1800 x 512 x 512 8.75 and 8.98; 16 layers of an MLP over
// 1500 rows 125 and 123), and those 16 layers lie 3.9e-7 from fp64 instead of 8.3e-7 (one TF32 product + two bf16 corrections:
// 6.9e-7).  At 128 columns 512 is the shortest chain that costs little (8192 x 768 x 768 29.1 / 26.9 / 26.6 us with 256 / 512 / 1024,
// 16384 x 1024 x 512 52.2 / 47.2 / 46.9; 14 layers of 1024 over 1565 rows 9.2e-7, 1.16e-6 with 1024, TF32 9.7e-7).  Wider tiles hold
// 96 or 128 sums and serve products whose error the rest of a transformer layer covers (8192 x 768 x 3072: 3.6e-6; TF32 5.0e-6).
// Few rows against a streamed weight ran in fp32 FFMA before: chains of 128 leave GPT-2-small over 40 positions 7.0e-7 from fp64
// (1.1e-6 with 256; fp32 7.9e-7), at 628 instead of 624 us.
constexpr int kChunkKDense = 1024, kChunkK128 = 512, kChunkKNarrow = 256, kChunkKConv = 128, kChunkKRows = 128;

// Times in microseconds as measured on B200 inside a chain of launches: `slab` per 64-deep K-slab of a tile, `gap` what every
// tile adds (its epilogue runs under the next tile's products), `drain` the exposed epilogue of the last one.
struct Variant { bool pair; int bn; double slab, gap, drain; };
const Variant kVariants[] = {
    {true, 256, 0.88, 1.5, 6.0}, {true, 192, 0.78, 0.6, 4.0}, {true, 128, 0.54, 0.4, 2.9}, {true, 64, 0.37, 0.2, 1.9},
    {false, 128, 0.64, 0.3, 2.1}, {false, 64, 0.47, 0.3, 1.3}, {false, 32, 0.39, 0.2, 0.6},
};
// Images: chains of 128, and an epilogue that often outlasts the products (it is part of `gap`).
const Variant kImageVariants[] = {
    {true, 256, 1.15, 5.0, 4.0}, {true, 192, 0.80, 4.4, 3.5}, {true, 128, 0.62, 3.2, 2.5}, {true, 64, 0.43, 2.2, 1.5},
    {false, 128, 0.74, 2.9, 2.0}, {false, 64, 0.55, 1.6, 1.0}, {false, 32, 0.46, 1.3, 0.5},
};
// bf16: a third of the products, so that the epilogue shows (in `gap`).
const Variant kBf16Variants[] = {
    {true, 256, 0.36, 1.0, 4.0}, {true, 192, 0.26, 3.0, 4.0}, {true, 128, 0.24, 1.7, 2.9}, {true, 64, 0.22, 0.4, 1.9},
    {false, 128, 0.28, 1.6, 2.1}, {false, 64, 0.24, 0.3, 1.3}, {false, 32, 0.22, 0.3, 0.6},
};
constexpr int kMaxClusterK = 8;
struct TailSplit { int64_t full, tail; int parts; double us; int cluster = 1; };
// Whole tiles first, then the remainder R = tiles % workers cut along K into s parts each (see F16Params).
TailSplit plan_tail(int64_t tiles, int num_k, const Variant& v, int workers, bool allowed, const int* clusters, double before) {
    const double tile_us = num_k * v.slab + v.gap;
    const int64_t R = tiles % workers, rounds = tiles / workers;
    TailSplit best{tiles, 0, 1, double(rounds + (R ? 1 : 0)) * tile_us + v.drain};
    const int64_t smax = allowed && R > 0 ? std::min<int64_t>(std::min<int64_t>(workers / R, num_k / 2), 8) : 1;
    for (int64_t s = 2; s <= smax; s++) {   // writing, fetching and adding partial tiles: 2 us and another one per part
        const double us = double(rounds) * tile_us + double((num_k + s - 1) / s) * v.slab + v.gap + v.drain + 1.0 + 1.0 * double(s);
        if (us < best.us) best = TailSplit{tiles - R, R, int(s), us};
    }
    // One round, cut inside clusters: the partial blocks are added through distributed shared memory in 1.8 us whatever their number (through L2,
    // flag by flag, it takes 3 to 8), and the more SMs the clusters take, and the more the launch before them does (`before`, its share), the later they start, up to 3 us each.
    // From wait to end, through L2 and so: 512 x 256 x 1024 8.1 and 5.0 us; one image of 14 x 14, 256 channels, 3x3 10.4 and 6.2; 7 x 7, 512 channels
    // 14.5 and 11.  Every pick against the same launch without clusters, pairs of products in a chain, 18 shapes of 32 to 3072 columns x 11 numbers of
    // rows from 65 to 1000: from +0.4 us (65 x 64 x 512) to -46 (128 x 32 x 8192, whose partial tiles otherwise wait for one another in L2).
    if (clusters != nullptr && !v.pair && rounds == 0)
        for (int s = 2; s <= kMaxClusterK && s <= num_k; s++) {
            if (tiles > clusters[s]) continue;
            const double us = double((num_k + s - 1) / s) * v.slab + v.gap + v.drain + 1.8 + 3.0 * double(tiles) * double(s - 1) / workers + 3.0 * before * before;
            if (us < best.us) best = TailSplit{0, tiles, s, us, s};
        }
    return best;
}

template <int BN, int STAGES, bool PAIR, int NPL, bool IMG = false, int EW = 8, bool CLUSTERS = false>
int launch_variant(const F16GemmArgs& a, F16Params p, const F16Plan& plan, ExecCtx& ctx, const CUtensorMap* im2col = nullptr) {
    constexpr int BNB = PAIR ? BN / 2 : BN;
    CUtensorMap mx, mw, mo, mr;
    if (IMG && p.im.c_slabs > 0) mx = *im2col;
    else if (make_map(&mx, a.x.planes, a.M, a.K, a.x.ld ? a.x.ld : a.K, a.x.plane, NPL, BM)) return 1;
    if (make_map(&mw, a.w.planes, a.N, a.K, a.w.ld ? a.w.ld : a.K, a.w.plane, NPL, BNB)) return 1;
    mo = mx;
    if (p.tma_out && make_out_map(&mo, a, NPL)) return 1;
    mr = mo;
    if (IMG && p.im.res != nullptr) {   // laid out like the result
        F16GemmArgs r = a;
        r.split_out.planes = const_cast<uint16_t*>(p.im.res);
        r.split_out.plane = p.im.res_plane;
        if (make_out_map(&mr, r, NPL)) return 1;
    }
    const size_t smem = sizeof(F16Smem<BN, BNB, STAGES, NPL, staging_buffers(BN, BNB, STAGES, NPL, IMG, EW), EW>) + 1024;
    static_assert(sizeof(F16Smem<BN, BNB, STAGES, NPL, staging_buffers(BN, BNB, STAGES, NPL, IMG, EW), EW>) + 1024 <= 227 * 1024, "shared memory of a CTA");
    auto kernel = gemm_f16_kernel<BN, STAGES, PAIR, NPL, IMG, EW, CLUSTERS>;
    static bool configured[64] = {};
    int dev = 0;
    FXF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        FXF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int64_t units = plan.full + plan.tail * plan.parts;
    const int grid = plan.cluster > 1 ? int(units) : int(std::min<int64_t>(units, plan.workers)) * (PAIR ? 2 : 1);
    FXF_CUDA(launch_dependent(kernel, dim3(unsigned(grid)), dim3(EW * 32 + 128), smem, ctx.stream, PAIR ? 2 : plan.cluster, mx, mw, mo, mr, p));
    FXF_LAUNCHED(ctx);
    return 0;
}

}  // namespace

bool gemm_f16_shape_ok(int64_t M, int64_t N, int64_t K) {
    return M >= 1 && N >= 1 && K >= 16 && K % 8 == 0 && M < (int64_t(1) << 31) - 512 && N < (int64_t(1) << 31) - 512 && K < (int64_t(1) << 31);
}

int gemm_f16_split_parts(int64_t N) { return int((N + 31) / 32) * 2; }

// The variant with the least modelled time.  Wide pair tiles win once they fill the machine; smaller problems take narrower
// tiles until every SM has one.
static int pick_variant(int64_t M, int64_t N, int64_t K, int sm_count, bool pairs, bool k_split, bool vt, int64_t vt_col0, const Variant* table, TailSplit* out_ts, int* out_workers,
                        const int* clusters = nullptr, bool images = false) {
    const int num_k = int((K + BK - 1) / BK);
    // An assumption about a launch that is not known here: what wrote x[M, K] had about a CTA per 128 x 64 of it (images: K counts every tap, and the maps
    // that are cut are small).  Off by all of it, it is 3 us for one variant against another.
    const double before = images ? 0.0 : std::min(1.0, double((M + BM - 1) / BM) * num_k / sm_count);
    int best = -1;
    double best_us = 0;
    for (int i = 0; i < int(sizeof(kVariants) / sizeof(kVariants[0])); i++) {
        const Variant& v = table[i];
        if (v.pair && (!pairs || M <= BM || sm_count < 2)) continue;
        if (vt && ((v.bn / 2) % 32 != 0 || vt_col0 % (v.bn / 2) != 0)) continue;   // a warp's columns: whole halves of a head
        const int rows = v.pair ? 2 * BM : BM, workers = v.pair ? sm_count / 2 : sm_count;
        const int64_t tiles = ((M + rows - 1) / rows) * ((N + v.bn - 1) / v.bn);
        const TailSplit ts = plan_tail(tiles, num_k, v, workers, k_split && !vt, vt ? nullptr : clusters, before);
        if (best < 0 || ts.us < best_us) {
            best = i;
            best_us = ts.us;
            if (out_ts) *out_ts = ts;
            if (out_workers) *out_workers = workers;
        }
    }
    return best;
}

// Which instance a product runs on, how its tiles are cut, and what it then uses of the K-split workspace: a partial tile per CTA
// of a cut tile, and one flag for each of its epilogue warps.  Where that does not fit, every tile is computed whole.
static F16Plan plan_launch(int64_t M, int64_t N, int64_t K, F16Form form, bool lean, bool vt, int64_t vt_col0, const F16Limits& lim) {
    F16Plan r;
    TailSplit ts{};
    r.variant = pick_variant(M, N, K, lim.sm_count, lim.pairs, lim.ws_bytes > 0 && lim.flag_count > 0, vt, vt_col0,
                             form == F16Form::kImages ? kImageVariants : (form == F16Form::kBf16 ? kBf16Variants : kVariants), &ts, &r.workers,
                             form == F16Form::kBf16 ? nullptr : lim.clusters, form == F16Form::kImages);
    if (r.variant < 0) return r;
    const Variant& var = kVariants[r.variant];
    // (tiles cut inside clusters are few slabs deep: the short chain costs them nothing)
    const int64_t chunk_k = lim.chunk_k > 0 ? lim.chunk_k : (form == F16Form::kImages ? kChunkKConv : (form != F16Form::kRows || var.bn > 128 ? kChunkKDense : (var.bn > 64 && ts.cluster == 1 ? kChunkK128 : kChunkKNarrow)));
    r.chunk_slabs = int(std::max<int64_t>(1, chunk_k / BK));
    r.epilogue_warps = r.variant == 0 && K <= int64_t(r.chunk_slabs) * BK && (form == F16Form::kImages || (form == F16Form::kBf16 && ts.parts == 1 && !lean)) ? 16 : 8;
    r.cluster = ts.cluster;
    const int64_t ctas = ts.cluster > 1 ? 0 : ts.tail * ts.parts * (var.pair ? 2 : 1);   // that pass partial tiles through L2
    r.ws_bytes = ts.parts > 1 ? size_t(ctas) * BM * size_t(var.bn) * sizeof(float) : 0;
    r.flags = ts.parts > 1 ? ctas * r.epilogue_warps : 0;
    if (r.ws_bytes > lim.ws_bytes || r.flags > lim.flag_count) {
        ts = TailSplit{ts.full + ts.tail, 0, 1, 0.0};
        r.ws_bytes = 0;
        r.flags = 0;
    }
    r.full = ts.full; r.tail = ts.tail; r.parts = ts.parts;
    return r;
}
F16Plan gemm_f16_plan(int64_t M, int64_t N, int64_t K, F16Form form, const F16Limits& lim) { return plan_launch(M, N, K, form, false, false, 0, lim); }

// One round of the widest single-CTA tiles at most: more tiles than SMs are more than a round.
bool gemm_f16_may_cut(int64_t M, int64_t N, int sm_count) { return (M + BM - 1) / BM * ((N + 127) / 128) < sm_count; }

std::string gemm_f16_variant_name(int64_t M, int64_t N, int64_t K, bool bf16, int sm_count) {
    const int v = pick_variant(M, N, K, sm_count, true, true, false, 0, bf16 ? kBf16Variants : kVariants, nullptr, nullptr);
    if (v < 0) return "none";
    return strfmt("%s-%dx%d%s", bf16 ? "bf16" : "f16x3", kVariants[v].pair ? 256 : 128, kVariants[v].bn, kVariants[v].pair ? "-pair" : "");
}

bool gemm_f16_vt_ok(const F16GemmArgs& a, const ExecCtx& ctx) {
    if (a.vt_out == nullptr || a.vt_flags == nullptr || a.residual != nullptr || a.relu || a.split_out.planes != nullptr) return false;
    if (a.vt_T <= 0 || a.vt_T % 32 != 0 || a.M % a.vt_T != 0 || (a.N - a.vt_col0) != int64_t(a.vt_heads) * 64) return false;
    return pick_variant(a.M, a.N, a.K, ctx.sm_count, ctx.tc_pair != 1, false, true, a.vt_col0, a.bf16 ? kBf16Variants : kVariants, nullptr, nullptr) >= 0;
}

// Clusters of `cs` CTAs, one per SM, that the device holds at once; asked once per device (a cluster lives inside one GPC, so this is not the
// number of SMs over cs: 74 of 2, 45 of 3, 33 of 4, 26 of 5, 22 of 6, 15 of 7 and 8 where there are 148).
static int clusters_resident(int cs, int* out) {
    static std::atomic<int> known[64][kMaxClusterK + 1];   // answer + 1
    int dev = 0;
    FXF_CUDA(cudaGetDevice(&dev));
    std::atomic<int>* slot = dev >= 0 && dev < 64 ? &known[dev][cs] : nullptr;
    *out = slot != nullptr ? slot->load(std::memory_order_relaxed) - 1 : -1;
    if (*out >= 0) return 0;
    auto kernel = gemm_f16_kernel<32, 4, false, 2, false, 8, true>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(cs);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(cs));
    cfg.blockDim = dim3(8 * 32 + 128);
    cfg.dynamicSmemBytes = 200 * 1024;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FXF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(cfg.dynamicSmemBytes)));
    if (cudaOccupancyMaxActiveClusters(out, kernel, &cfg) != cudaSuccess) {   // a size this device does not launch
        (void)cudaGetLastError();
        *out = 0;
    }
    if (slot != nullptr) slot->store(*out + 1, std::memory_order_relaxed);
    return 0;
}

// The launch of a product whose tiles are cut inside clusters, by the width of its tiles and the number of parts
static const char* cut_tag(bool images, int bn, int parts) {
#define FXF_CUT(name, bn) {name "_" #bn "_cut2", name "_" #bn "_cut3", name "_" #bn "_cut4", name "_" #bn "_cut5", name "_" #bn "_cut6", name "_" #bn "_cut7", name "_" #bn "_cut8"}
    static const char* const names[2][3][kMaxClusterK - 1] = {{FXF_CUT("gemm_f16x3_tcgen05", 32), FXF_CUT("gemm_f16x3_tcgen05", 64), FXF_CUT("gemm_f16x3_tcgen05", 128)},
                                                              {FXF_CUT("conv2d_f16x3_tcgen05", 32), FXF_CUT("conv2d_f16x3_tcgen05", 64), FXF_CUT("conv2d_f16x3_tcgen05", 128)}};
#undef FXF_CUT
    return names[images ? 1 : 0][bn == 32 ? 0 : (bn == 64 ? 1 : 2)][parts - 2];
}

static int launch_f16(const F16GemmArgs& a, const ImageGeom* im, const CUtensorMap* im2col, const char* tag, double flops, ExecCtx& ctx) {
    FXF_CHECK(gemm_f16_shape_ok(a.M, a.N, a.K) && a.x.planes && a.w.planes && aligned16(a.x.planes) && aligned16(a.w.planes) && (a.x.plane * 2) % 16 == 0,
              "f16 GEMM: unsupported operands (M=%lld N=%lld K=%lld)", (long long)a.M, (long long)a.N, (long long)a.K);
    const bool split = a.split_out.planes != nullptr;
    FXF_CHECK(split || a.out != nullptr, "f16 GEMM: no output");
    FXF_CHECK(!split || (a.N % 8 == 0 && a.residual == nullptr && a.vt_out == nullptr), "f16 GEMM: a split output needs N %% 8 == 0 and no residual");
    FXF_CHECK(a.col_inv == nullptr || (split && im == nullptr && a.col_bias != nullptr && a.bad_rows > 0 && a.bad_block > 0), "f16 GEMM: scaled columns are those of a split output");
    const bool tma_out = split || (a.ldo % 4 == 0 && aligned16(a.out) && (a.residual == nullptr || aligned16(a.residual)));
    const bool lean = !split && !tma_out && a.residual == nullptr;
    const F16Form form = im != nullptr ? F16Form::kImages : (a.bf16 ? F16Form::kBf16 : F16Form::kRows);
    F16Limits lim;
    lim.sm_count = ctx.sm_count; lim.pairs = ctx.tc_pair != 1; lim.chunk_k = ctx.tc_chunk_k;
    if (ctx.gemm_ws != nullptr && ctx.gemm_flags != nullptr) { lim.ws_bytes = ctx.gemm_ws_bytes; lim.flag_count = ctx.gemm_flag_count; }
    int clusters[kMaxClusterK + 1] = {};
    if (!a.bf16 && gemm_f16_may_cut(a.M, a.N, ctx.sm_count))
        for (int cs = 2; cs <= kMaxClusterK; cs++)
            if (clusters_resident(cs, &clusters[cs])) return 1;
    lim.clusters = clusters;
    const F16Plan plan = plan_launch(a.M, a.N, a.K, form, lean, a.vt_out != nullptr, a.vt_col0, lim);
    const int v = plan.variant;
    FXF_CHECK(v >= 0, "f16 GEMM: no kernel variant for M=%lld N=%lld K=%lld", (long long)a.M, (long long)a.N, (long long)a.K);
    const Variant& var = kVariants[v];
    const int rows = var.pair ? 2 * BM : BM;
    F16Params p{};
    p.bias = a.col_inv != nullptr ? a.col_bias : a.bias; p.residual = a.residual; p.out = a.out;
    p.x_inv = a.bf16 ? nullptr : a.x.inv; p.w_inv = a.col_inv != nullptr ? a.col_inv : (a.bf16 ? nullptr : a.w.inv);
    p.x_inv_stride = a.x.inv_stride;
    p.w_inv_stride = 1;
    p.M = a.M; p.N = a.N; p.K = a.K; p.ldo = split ? a.N : a.ldo;
    p.relu = a.relu ? 1 : 0;
    p.tma_out = tma_out ? 1 : 0;
    auto sector = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 31) == 0; };
    p.fast = a.N % 16 == 0 && (split ? sector(a.split_out.planes) && a.split_out.plane % 16 == 0 : a.ldo % 8 == 0 && sector(a.out)) && sector(a.residual) ? 1 : 0;
    p.lean = lean ? 1 : 0;
    p.tiles_m = int((a.M + rows - 1) / rows);
    p.tiles_n = int((a.N + var.bn - 1) / var.bn);
    p.m_fastest = a.N > a.M ? 1 : 0;
    p.status = ctx.status;
    if (im != nullptr) p.im = *im;
    p.full_tiles = int(plan.full); p.tail_tiles = int(plan.tail); p.tail_split = plan.parts; p.cluster_k = plan.cluster;
    p.chunk_slabs = plan.chunk_slabs;
    p.ws = ctx.gemm_ws; p.flags = ctx.gemm_flags;
    p.early_w = ctx.weights_settled ? 1 : 0;
    if (split) {
        p.so = a.split_out.planes; p.so_plane = a.split_out.plane; p.so_inv = a.split_out.inv; p.so_amax = a.split_out.amax;
        p.so_parts = plan.epilogue_warps / 4 * p.tiles_n;
        p.so_cols = a.col_inv != nullptr ? 1 : 0; p.so_bad = a.split_bad; p.bad_rows = a.bad_rows; p.bad_block = a.bad_block;
        if (a.split_out.parts_out) *a.split_out.parts_out = p.so_parts;
        p.x_amax = a.x.amax; p.x_parts = a.x.parts; p.w_bound = a.w.bound;
        FXF_CHECK(a.bf16 || a.col_inv != nullptr || (p.so_inv && p.so_amax && p.x_amax && p.w_bound), "f16 GEMM: a split output needs the row bounds of x and w");
    }
    if (a.vt_out != nullptr) {
        p.vt_out = a.vt_out; p.vt_flags = a.vt_flags; p.vt_col0 = a.vt_col0; p.vt_T = a.vt_T; p.vt_heads = a.vt_heads; p.vt_n32 = a.vt_n32;
    }
    tag_launch(ctx, plan.cluster > 1 ? cut_tag(im != nullptr, var.bn, plan.cluster) : tag, flops, 4.0 * (double(a.M) * a.K + double(a.N) * a.K + double(a.N) + double(a.M) * a.N));
    if (a.bf16) {
        switch (v) {
            case 0:
                if (plan.epilogue_warps == 16) return launch_variant<256, 4, true, 1, false, 16>(a, p, plan, ctx);
                return launch_variant<256, 6, true, 1>(a, p, plan, ctx);
            case 1: return launch_variant<192, 6, true, 1>(a, p, plan, ctx);
            case 2: return launch_variant<128, 6, true, 1>(a, p, plan, ctx);
            case 3: return launch_variant<64, 6, true, 1>(a, p, plan, ctx);
            case 4: return launch_variant<128, 6, false, 1>(a, p, plan, ctx);
            case 5: return launch_variant<64, 8, false, 1>(a, p, plan, ctx);
            default: return launch_variant<32, 8, false, 1>(a, p, plan, ctx);
        }
    }
    if (plan.cluster > 1) {
        if (im != nullptr)
            return v == 4 ? launch_variant<128, 2, false, 2, true, 8, true>(a, p, plan, ctx, im2col)
                          : (v == 5 ? launch_variant<64, 3, false, 2, true, 8, true>(a, p, plan, ctx, im2col) : launch_variant<32, 4, false, 2, true, 8, true>(a, p, plan, ctx, im2col));
        return v == 4 ? launch_variant<128, 3, false, 2, false, 8, true>(a, p, plan, ctx) : (v == 5 ? launch_variant<64, 4, false, 2, false, 8, true>(a, p, plan, ctx) : launch_variant<32, 4, false, 2, false, 8, true>(a, p, plan, ctx));
    }
    if (im != nullptr) {
        switch (v) {
            case 0:
                if (plan.epilogue_warps == 16) return launch_variant<256, 2, true, 2, true, 16>(a, p, plan, ctx, im2col);
                return launch_variant<256, 2, true, 2, true>(a, p, plan, ctx, im2col);
            case 1: return launch_variant<192, 3, true, 2, true>(a, p, plan, ctx, im2col);
            case 2: return launch_variant<128, 3, true, 2, true>(a, p, plan, ctx, im2col);
            case 3: return launch_variant<64, 4, true, 2, true>(a, p, plan, ctx, im2col);
            case 4: return launch_variant<128, 2, false, 2, true>(a, p, plan, ctx, im2col);
            case 5: return launch_variant<64, 3, false, 2, true>(a, p, plan, ctx, im2col);
            default: return launch_variant<32, 4, false, 2, true>(a, p, plan, ctx, im2col);
        }
    }
    switch (v) {
        case 0: return launch_variant<256, 3, true, 2>(a, p, plan, ctx);
        case 1: return launch_variant<192, 3, true, 2>(a, p, plan, ctx);
        case 2: return launch_variant<128, 4, true, 2>(a, p, plan, ctx);
        case 3: return launch_variant<64, 4, true, 2>(a, p, plan, ctx);
        case 4: return launch_variant<128, 3, false, 2>(a, p, plan, ctx);
        case 5: return launch_variant<64, 4, false, 2>(a, p, plan, ctx);
        default: return launch_variant<32, 4, false, 2>(a, p, plan, ctx);
    }
}

int launch_gemm_f16(const F16GemmArgs& a, ExecCtx& ctx) {
    if (a.M == 0 || a.N == 0) return 0;
    return launch_f16(a, nullptr, nullptr, a.bf16 ? "gemm_bf16_tcgen05" : "gemm_f16x3_tcgen05", 2.0 * double(a.M) * double(a.N) * double(a.K), ctx);
}

// The corners and offsets of a 4-D im2col map are 8-bit numbers, its strides at most 8; TMA needs 16-byte pixels and image rows.
bool conv_f16_shape_ok(int64_t n_pix, int64_t C, int64_t O, int64_t KH, int64_t KW, const int64_t* geom) {
    const int64_t sh = geom[0], sw = geom[1], ph = geom[2], pw = geom[3], dh = geom[4], dw = geom[5], groups = geom[6];
    return groups == 1 && C >= 16 && C % 8 == 0 && O % 8 == 0 && n_pix >= 1 && n_pix < (int64_t(1) << 31) - 256 && sh >= 1 && sh <= 8 && sw >= 1 && sw <= 8 && ph >= 0 && ph <= 127 &&
           pw >= 0 && pw <= 127 && dh >= 1 && dw >= 1 && (KH - 1) * dh <= 127 && (KW - 1) * dw <= 127 && KH * KW * ((C + 63) / 64) < (1 << 20);
}

int launch_conv_f16(const ConvF16Args& c, ExecCtx& ctx) {
    const int64_t pixels = int64_t(c.N) * c.HO * c.WO;
    if (pixels == 0 || c.O == 0) return 0;
    const bool rows = !c.window && c.KH == 1 && c.KW == 1 && c.str_h == 1 && c.str_w == 1 && c.pad_h == 0 && c.pad_w == 0;
    const int c_slabs = c.window ? 1 : (c.C + BK - 1) / BK, taps = c.window ? c.KH : c.KH * c.KW;
    F16GemmArgs a;
    a.x = c.x; a.w = c.w;
    a.bias = c.bias; a.out = c.out; a.split_out = c.split_out;
    a.M = pixels; a.N = c.O; a.K = rows ? c.C : int64_t(taps) * c_slabs * BK;
    a.ldo = c.O;
    a.relu = c.relu;
    FXF_CHECK(c.split_out.planes != nullptr || (c.O % 4 == 0 && aligned16(c.out)), "convolution (f16): the output needs 16-byte pixels");
    FXF_CHECK(c.res.planes == nullptr || (c.O % 8 == 0 && aligned16(c.res.planes) && (c.res.plane * 2) % 16 == 0 && c.split_out.planes != nullptr), "convolution (f16): unsupported residual");
    ImageGeom im{};
    im.rpi = unsigned(c.HO * c.WO);
    im.res = c.res.planes; im.res_plane = c.res.plane; im.res_inv = c.res.inv; im.res_amax = c.res.amax;
    CUtensorMap map;
    if (!rows) {
        im.c_slabs = c_slabs; im.KW = c.window ? 1 : c.KW; im.WO = c.WO; im.HO = c.HO;
        im.sw = c.str_w; im.sh = c.str_h; im.pw = c.pad_w; im.ph = c.pad_h; im.dw = c.dil_w; im.dh = c.dil_h;
        im.lo_image = c.N;
        const int64_t C = c.window ? BK : c.C, pitch = c.window ? 16 : c.C, W = c.window ? c.WO : c.W, row = c.window ? int64_t(c.WO + 3) * 16 : int64_t(c.W) * c.C;
        FXF_CHECK(c.x.plane == int64_t(c.N) * c.H * row, "convolution (f16): the planes of x must follow each other");
        static const auto fn = [] {
            void* q = nullptr;
            cudaDriverEntryPointQueryResult r;
            return cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &q, cudaEnableDefault, &r) == cudaSuccess && r == cudaDriverEntryPointSuccess ? reinterpret_cast<decltype(&cuTensorMapEncodeIm2col)>(q) : nullptr;
        }();
        FXF_CHECK(fn != nullptr, "cuTensorMapEncodeIm2col is not available from the CUDA driver");
        const int KW = im.KW;
        cuuint64_t dims[4] = {cuuint64_t(C), cuuint64_t(W), cuuint64_t(c.H), cuuint64_t(2) * c.N};
        cuuint64_t strides[3] = {cuuint64_t(pitch) * 2, cuuint64_t(row) * 2, cuuint64_t(row) * c.H * 2};
        int lower[2] = {-c.pad_w, -c.pad_h}, upper[2] = {c.pad_w - (KW - 1) * c.dil_w, c.pad_h - (c.KH - 1) * c.dil_h};
        cuuint32_t estr[4] = {1, cuuint32_t(c.str_w), cuuint32_t(c.str_h), 1};
        CUresult r = fn(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<uint16_t*>(c.x.planes), dims, strides, lower, upper, BK, BM, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        FXF_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeIm2col failed with code %d (%d x %d x %d x %d)", int(r), c.N, c.H, c.W, c.C);
    }
    return launch_f16(a, &im, rows ? nullptr : &map, "conv2d_f16x3_tcgen05", 2.0 * double(pixels) * c.O * c.C * c.KH * c.KW, ctx);
}

// out[M,N] for M <= 64 rows in split form and a weight of at least a tile per SM (see F16Params::swap).  The persistent kernel
// keeps its weight stream going across tiles: 32 x 50257 x 768 (154 MB) in 31 us = 4.9 TB/s.
int launch_gemm_f16_swapped(const F16GemmArgs& a, ExecCtx& ctx) {
    FXF_CHECK(a.M >= 1 && a.M <= 64 && gemm_f16_shape_ok(a.M, a.N, a.K) && !a.bf16 && a.x.planes && a.w.planes && a.out && a.split_out.planes == nullptr && a.vt_out == nullptr,
              "f16 GEMM (swapped): unsupported operands");
    F16GemmArgs t = a;
    t.x = a.w; t.w = a.x;
    t.M = a.N; t.N = a.M;
    F16Params p{};
    p.swap = 1;
    p.bias = a.bias; p.residual = a.residual; p.out = a.out;
    p.x_inv = a.w.inv; p.x_inv_stride = 1; p.w_inv = a.x.inv; p.w_inv_stride = a.x.inv_stride;
    p.M = t.M; p.N = t.N; p.K = t.K; p.ldo = a.ldo;
    p.relu = a.relu ? 1 : 0;
    p.tiles_m = int((t.M + BM - 1) / BM);
    p.tiles_n = 1;
    p.full_tiles = p.tiles_m; p.tail_split = 1;
    p.chunk_slabs = kChunkKRows / BK;
    p.early_w = ctx.weights_settled ? 1 : 0;
    p.status = ctx.status;
    tag_launch(ctx, "gemm_f16x3_swapped_tcgen05", 2.0 * double(a.M) * double(a.N) * double(a.K),
               4.0 * (double(a.M) * a.K + double(a.N) * a.K + double(a.N) + double(a.M) * a.N));
    F16Plan plan;
    plan.workers = ctx.sm_count;
    plan.full = p.tiles_m;
    return a.M <= 32 ? launch_variant<32, 4, false, 2>(t, p, plan, ctx) : launch_variant<64, 4, false, 2>(t, p, plan, ctx);
}

}  // namespace fxf
