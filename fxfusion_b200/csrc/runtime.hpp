// Runtime contracts of the B200 backend: registry, params, per-node plan and the KernelFn
// function-pointer type.  They keep the shape of the reference's contracts
// (csrc/include/runtime/tensor_registry.hpp:8-26) with LibTorch removed:
//   TensorRegistry  vector<torch::Tensor>      -> vector<FxfTensor> (raw device pointers)
//   Cache           per-node torch::empty bufs -> NodePlan: launch geometry computed once at
//                                                 build + byte counts of the shared scratch /
//                                                 persistent memory the node wants
//   KernelFn        void(*)(reg,in,out,params,cache) -> int(*)(reg,in,out,params,plan,ctx)
#pragma once
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/fxf_b200.h"

namespace fxf {

using Registry = std::vector<FxfTensor>;
using TensorIds = std::vector<uint32_t>;

struct Params {
    std::vector<int64_t> ints;
    std::vector<float> floats;
};

// One traced kernel launch (profiling mode only).
struct LaunchRecord {
    const char* name;      // kernel family, e.g. "gemm_simt128x128", "attention_fp32"
    int node;              // index of the graph node that issued it
    double flops, bytes;   // algorithmic work of this launch
    cudaEvent_t done;      // recorded right after the launch
};

// Everything a launch needs besides the registry.
// The engine allocations of all tensor-parallel ranks of a node as mapped into this process (CUDA IPC).
constexpr int kMaxTpRanks = 8;
struct PeerMap {
    char* base[kMaxTpRanks] = {};   // base[r]: rank r's allocation (own rank: the local pointer)
    size_t shared_bytes = 0;        // offsets below this mean the same tensor on every rank (the planner's arena)
    size_t flags_off = 0;           // barrier flags [peer][block] of the peer all-reduce, same offset on every rank
    size_t epoch_off = 0;           // two ints: epoch, finished-block counter
    int grid = 0;                   // blocks of the peer exchange kernels (fixes the flag layout)
    // Exchange window: a buffer outside the planner's arena (same offset on every rank, never reused for anything else) into
    // which the peers' row-parallel products store their partial sums of this rank's rows.  0 bytes: no window.
    size_t push_off = 0, push_bytes = 0;
    // wait budgets of the two peer barriers of an exchange; the first also absorbs the skew between the ranks' host threads
    unsigned long long start_budget_ns = 20000000000ull, end_budget_ns = 2000000000ull;
};

// The exchange step of a row-parallel product under tensor parallelism, fused with what follows it in a pre-LN transformer
// block: the ranks' partial [M,D] outputs are summed, the residual is added and the rows are normalised by ONE kernel over
// peer memory (kernels/tp_exchange.cu).  Set by the engine around a sharded MHA / CrossMHA / FeedForward node whose
// following Add (+ LayerNorm) or AddLayerNorm nodes were folded into it.
struct TpExchange {
    bool enabled = false;
    const float* residual = nullptr;   // the other operand of the folded Add (this rank's rows of it are read)
    float* x_out = nullptr;            // output of the folded Add: the new residual stream (NULL for AddLayerNorm)
    float* y_out = nullptr;            // output of the folded LayerNorm / AddLayerNorm (NULL: a plain Add was folded)
    const float* gamma = nullptr;
    const float* beta = nullptr;
    float eps = 0.f;
    bool replicate_x = false;          // x_out is read outside this scheme: every rank gets every row of it
    bool consumed = false;
};

// A residual Add / AddRelu node folded into the contraction that precedes it: the owner of that node's final GEMM writes
// act(acc + bias + residual) straight into the Add's output tensor.
struct EpilogueFusion {
    const float* residual = nullptr;
    float* out = nullptr;
    bool relu = false;
    bool consumed = false;
    int residual_id = -1;   // its tensor id (for a residual kept in split form)
};

// ---- split form (kernels/gemm_f16.cu): an fp32 matrix [rows, K] as two fp16 planes and a power-of-two scale per row, or as
// one bf16 plane in the bf16 mode -----------------------------------------------------------------------------------------
struct SplitMat {
    const uint16_t* planes = nullptr;   // hi plane [rows, K]; the lo plane lies `plane` elements behind it
    int64_t plane = 0;
    int64_t ld = 0;                     // elements between rows (0: dense)
    const float* inv = nullptr;         // 1 / scale per row, `inv_stride` entries apart
    int64_t inv_stride = 1;
    const float* amax = nullptr;        // activations: max_k |x[r,k]| as `parts` partial maxima per row
    int parts = 1;
    float cap = 0.f;                    // activations: no |x| exceeds it whatever the input (normalised rows); 0: unknown
    int gamma = -1, beta = -1;          // with a cap: the tensors (constants) that a LayerNorm multiplied and shifted the rows with
    const float* bound = nullptr;       // weights: {max_j ||w_j||_1, max_j |b_j|}
};
struct SplitOut {
    uint16_t* planes = nullptr;
    int64_t plane = 0;
    float* inv = nullptr;
    float* amax = nullptr;
    int* parts_out = nullptr;           // host: how many partial maxima per row the producer writes
};

// A LayerNorm folded into the product that reads it: x its input rows (dense), gamma and beta of the row's length.
struct NormInput {
    const float *x = nullptr, *gamma = nullptr, *beta = nullptr;
    float eps = 0.f;
};

// An attention mask as bits (kernels/attention_f16.cu): strides in words between batches, heads and query rows; and per batch, head
// and tile of 128 query rows a word that says which blocks of keys any of them sees.  bad: per batch the blocks of keys for which a
// projection that feeds an attention core of this forward has given a value that is not finite (F16GemmArgs::split_bad).
struct MaskBits {
    uint32_t *bits = nullptr, *need = nullptr, *bad = nullptr;
    int batches = 0;
    int64_t bit_sb = 0, bit_sh = 0, bit_sq = 0, need_sb = 0, need_sh = 0, need_st = 0;
};

struct ExecCtx {
    cudaStream_t stream = nullptr;
    void* scratch = nullptr;       // shared by all nodes of an engine; nodes run one at a time
    size_t scratch_bytes = 0;
    int* status = nullptr;         // sticky device status word (0 = ok)
    int sm_count = 148;
    int gemm_mode = FXF_GEMM_AUTO;
    int launches = 0;              // incremented by every kernel launch (host-side count)
    int tp_rank = 0, tp_size = 1;  // tensor-parallel position; tp_size > 1 needs `comm`
    void* comm = nullptr;          // fxf_comm* (NCCL communicator wrapper), owned by the caller
    const PeerMap* peers = nullptr;  // set when the ranks' allocations are mapped into each other: all-reduce over peer memory
    // Tensors in split form, by tensor id (planes == NULL: the plain fp32 tensor), and the form in which the current node has to
    // leave its output (set by the engine around the node).
    const std::vector<SplitMat>* splits = nullptr;
    SplitOut split_out;
    NormInput norm;                  // set by the engine around a node whose input 0 is the result of a folded LayerNorm
    MaskBits mask_bits;              // of the current attention node, where the engine keeps them
    EpilogueFusion fuse;             // set by the engine around a node whose following Add was folded into it
    TpExchange xchg;                 // set by the engine around a sharded node whose exchange absorbs the following Add / LayerNorm
    // workspace of the tensor-core GEMM's K-split last round: partial tiles and their ready flags (zero between
    // launches).  Without it every tile is computed whole.
    float* gemm_ws = nullptr;
    size_t gemm_ws_bytes = 0;
    int* gemm_flags = nullptr;
    int gemm_flag_count = 0;
    int tc_chunk_k = 0;            // K-elements per tensor-core accumulation chain (0 = the kernel's default)
    bool weights_settled = false;  // inside an engine after its build: weights were written long before the current kernel chain
    int tc_pair = 0;               // 0: 256-wide tensor-core GEMM tiles are computed by CTA pairs (tcgen05 cta_group::2); 1: never
    // profiling: when `trace` is set every launch appends a record carrying the current tag
    std::vector<LaunchRecord>* trace = nullptr;
    int cur_node = -1;
    const char* tag_name = "kernel";
    double tag_flops = 0, tag_bytes = 0;
};
inline void tag_launch(ExecCtx& c, const char* name, double flops, double bytes) {
    c.tag_name = name;
    c.tag_flops = flops;
    c.tag_bytes = bytes;
}
int trace_after_launch(ExecCtx& ctx);
inline const SplitMat* split_of(const ExecCtx& ctx, uint32_t id) {
    return ctx.splits != nullptr && id < ctx.splits->size() && (*ctx.splits)[id].planes != nullptr ? &(*ctx.splits)[id] : nullptr;
}
// Called by the op that owns the final GEMM of a node: redirects the output and attaches the residual of a folded Add.
// `partial`: the node is sharded over the tensor-parallel ranks and its outputs are summed afterwards, so only rank 0 adds
// the residual (like the bias); a node that is replicated on every rank adds it everywhere.
template <class Args>
inline void apply_fusion(ExecCtx& ctx, Args& g, bool partial) {
    if (ctx.fuse.out == nullptr) return;
    g.out = ctx.fuse.out;
    g.residual = (!partial || ctx.tp_rank == 0) ? ctx.fuse.residual : nullptr;
    g.relu = g.relu || ctx.fuse.relu;
    ctx.fuse.consumed = true;
}
// out = w[idx] * scale + rows, which repeat
int launch_embedding_scale_add(const FxfTensor& idx, const FxfTensor& w, float scale, const FxfTensor& rows, const FxfTensor& out, ExecCtx& ctx);
// out = act(out + residual) over n contiguous floats: the fallback when a GEMM without a fused epilogue ran
int launch_residual_epilogue(float* out, const float* residual, int64_t n, bool relu, ExecCtx& ctx);

struct NodePlan {
    virtual ~NodePlan() = default;
    // split-form activations (struct SplitMat): bit i set = input i is only ever the f16 operand of this node's products; makes_split
    // = output 0 can be written in split form, as split_rows x split_cols
    uint32_t takes_split = 0;
    bool makes_split = false;
    int64_t split_rows = 0, split_cols = 0;
    // channels-last images in split form, one scale per image (ConvF16Args): what the node can do with them
    enum ImageRole { kNoImages, kImageConv, kImageStem, kImageMaxPool, kImageGlobalAvg };
    ImageRole image_role = kNoImages;
    bool takes_norm = false;    // input 0 is read by one few-row product only, which can normalise its rows (NormInput)
    // attention nodes that may run on operands in split form: the mask's input, and the queries and keys it is for
    int mask_input = -1;
    int64_t mask_B = 0, mask_T = 0, mask_Tk = 0;
    uint32_t mask_rows_from = 0;   // the inputs that have to arrive in split form for that, a bit each
    bool scaled = false;           // found by settle(): Q, K and V have scales, the node runs so wherever the engine keeps the mask's bits
    bool images = false;        // decided by the engine before prepare(): the node runs on them
    size_t scratch_bytes = 0;   // shared scratch wanted at execute time
    size_t persist_bytes = 0;   // memory that must survive across runs (e.g. re-laid-out weights)
    void* persist = nullptr;    // assigned by the engine before prepare()
    double flops = 0, bytes = 0;  // algorithmic work of the node
    std::string variant;        // which kernel variant was chosen (for describe / profiling)
    bool tp_sharded = false;    // the node computes a partial result on each tensor-parallel rank (summed by an exchange)
    // Called once after device memory exists (constants uploaded).  May launch kernels.
    virtual int prepare(Registry&, const TensorIds&, const TensorIds&, const Params&, ExecCtx&) { return 0; }
    // Called by the engine once all of that has run on the device.
    virtual int settle() { return 0; }
};

// What a plan builder needs to know about the engine it plans for.
struct PlanEnv {
    int gemm_mode = FXF_GEMM_AUTO;
    int sm_count = 148;               // of the device that will run the plan
    int tp_rank = 0, tp_size = 1;     // tensor-parallel position of this engine
    bool shard_output_cols = false;   // this node is the graph's final Linear and its columns are sharded over the ranks
    bool tc_pairs = true;             // the engine lets CTA pairs compute the widest GEMM tiles (reported in variant names)
    // By tensor id: the tensor is a constant of the graph (NULL: a single call, whose tensors are what they are while it runs).
    // Only those may be converted at build time; a weight that the graph computes or takes as an input is read as it is.
    const std::vector<char>* constants = nullptr;
    bool is_constant(uint32_t id) const { return constants == nullptr || (id < constants->size() && (*constants)[id]); }
};

using KernelFn = int (*)(Registry&, const TensorIds&, const TensorIds&, const Params&, const NodePlan*, ExecCtx&);
using PlanFn = std::unique_ptr<NodePlan> (*)(const Registry&, const TensorIds&, const TensorIds&, const Params&, const PlanEnv&);

struct OpEntry {
    const char* name = nullptr;
    KernelFn kernel = nullptr;
    PlanFn plan = nullptr;
};

// OpCode -> {kernel, plan builder}.  Counterpart of OpRegistry (csrc/runtime/op_registry.cpp:16-106);
// there is one kernel set only — CUDA — and no CPU fallback.
const OpEntry& op_entry(int op_code);

// ---- error plumbing -------------------------------------------------------------------
void set_last_error(const std::string& msg);
const std::string& last_error();

inline std::string strfmt(const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    return std::string(buf);
}

#define FXF_FAIL(...)                                   \
    do {                                                \
        ::fxf::set_last_error(::fxf::strfmt(__VA_ARGS__)); \
        return 1;                                       \
    } while (0)

#define FXF_CHECK(cond, ...)          \
    do {                              \
        if (!(cond)) FXF_FAIL(__VA_ARGS__); \
    } while (0)

#define FXF_CUDA(expr)                                                                       \
    do {                                                                                     \
        cudaError_t _e = (expr);                                                             \
        if (_e != cudaSuccess) FXF_FAIL("CUDA error %s at %s:%d (%s)", cudaGetErrorString(_e), __FILE__, __LINE__, #expr); \
    } while (0)

// Checks the launch that has just been issued and counts it.
#define FXF_LAUNCHED(ctx)                                                                     \
    do {                                                                                      \
        cudaError_t _e = cudaPeekAtLastError();                                               \
        if (_e != cudaSuccess) FXF_FAIL("kernel launch failed: %s at %s:%d", cudaGetErrorString(_e), __FILE__, __LINE__); \
        (ctx).launches++;                                                                     \
        if ((ctx).trace && ::fxf::trace_after_launch(ctx)) return 1;                          \
    } while (0)

// ---- tensor helpers ---------------------------------------------------------------------
inline int64_t numel(const FxfTensor& t) {
    int64_t n = 1;
    for (int i = 0; i < t.rank; i++) n *= t.shape[i];
    return n;
}
inline int dtype_size(int dt) {
    switch (dt) {
        case FXF_F32: return 4;
        case FXF_F16: return 2;
        case FXF_I32: return 4;
        case FXF_I64: return 8;
        case FXF_BOOL: return 1;
        default: return 0;
    }
}
inline void set_contiguous(FxfTensor& t) {
    int64_t s = 1;
    for (int i = t.rank - 1; i >= 0; i--) {
        t.stride[i] = s;
        s *= t.shape[i];
    }
}
inline bool is_contiguous(const FxfTensor& t) {
    int64_t s = 1;
    for (int i = t.rank - 1; i >= 0; i--) {
        if (t.shape[i] != 1 && t.stride[i] != s) return false;
        s *= t.shape[i];
    }
    return true;
}
// Channels-last ("NHWC") physical layout of a logical [N,C,H,W] tensor: strides (H*W*C, 1, W*C, C).  The graph
// contract is NCHW; the engine may keep intermediate activations between layout-aware nodes channels-last
// and says so through the registry strides, the way torch's channels_last memory format does.
inline void set_channels_last(FxfTensor& t) {
    const int64_t C = t.shape[1], H = t.shape[2], W = t.shape[3];
    t.stride[0] = H * W * C;
    t.stride[1] = 1;
    t.stride[2] = W * C;
    t.stride[3] = C;
}
inline bool is_channels_last(const FxfTensor& t) {
    if (t.rank != 4 || is_contiguous(t)) return false;
    const int64_t C = t.shape[1], H = t.shape[2], W = t.shape[3];
    return (t.shape[0] == 1 || t.stride[0] == H * W * C) && (C == 1 || t.stride[1] == 1) && (H == 1 || t.stride[2] == W * C) && (W == 1 || t.stride[3] == C);
}
inline bool same_layout(const FxfTensor& a, const FxfTensor& b) {
    if (a.rank != b.rank) return false;
    for (int i = 0; i < a.rank; i++)
        if (a.shape[i] != b.shape[i] || (a.shape[i] != 1 && a.stride[i] != b.stride[i])) return false;
    return true;
}
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// ---- kernels shared between ops (defined in the .cu files) -------------------------------
// out[M,N] = act(x[M,K] · w[N,K]^T + bias[N]); row strides in elements (ldx, ldw, ldo).
// `w_hi` / `w_lo`: the weight pre-split into TF32 high and low parts for the tensor-core path
// (both null when no split exists; the fp32 SIMT kernel is used then).
struct GemmArgs {
    const float* x = nullptr;
    const float* w = nullptr;
    const float* w_hi = nullptr;
    const float* w_lo = nullptr;
    bool w_is_bf16 = false;   // bf16 mode: w_hi points to the weight as bf16 [N,K] (w_lo unused)
    bool w_mixed = false;     // mixed mode: w_hi is the TF32 high part (fp32), w_lo points to a bf16 matrix [2N,K]: bf16(w_hi) rows, then bf16(w - w_hi) rows
    const float* bias = nullptr;
    const float* residual = nullptr;   // optional [M,N] with the pitch of `out`, added after the bias and before the ReLU
    float* out = nullptr;
    int64_t M = 0, N = 0, K = 0;
    int64_t ldx = 0, ldw = 0, ldo = 0;
    bool relu = false;
    bool conv_chain = false;   // a convolution written as a GEMM: use the (shorter) accumulation chains of convolutions
    // Row-pushed output of a row-parallel product under tensor parallelism (tensor-core kernels only): rows
    // [q*push_rows, (q+1)*push_rows) of the result go to push_out[q] (rank q's exchange window, peer memory for q != rank) at
    // row push_rank*push_rows + (row - q*push_rows); `out` is not written.  push_rows == 0: the plain output.
    float* const* push_out = nullptr;
    int64_t push_rows = 0;
    int push_rank = 0;
    // Transposed column range (the V third of a packed QKV projection, tensor-core kernels only): columns [vt_col0, N) of
    // the result are not written to `out`; column vt_col0 + 64*h + d of row b*vt_T + t goes to vt_out[((b*vt_heads + h)*64 + d)
    // * vt_T + t] (V^T per batch and head, keys contiguous: the B operand of the attention's second product), and
    // vt_flags[((b*vt_heads + h)*2 + d/32)*vt_n32 + t/32] tells whether any of those values of a 32-row group and half a
    // head is NaN or infinite.
    // Ask gemm_tc_vt_ok() first.
    float* vt_out = nullptr;
    unsigned char* vt_flags = nullptr;
    int64_t vt_col0 = 0;
    int vt_T = 0, vt_heads = 0, vt_n32 = 0;
};
// Whether launch_gemm would serve the transposed column range of `a` (fields vt_* filled in) on this context.
bool gemm_tc_vt_ok(const GemmArgs& a, const ExecCtx& ctx);
int launch_gemm(const GemmArgs& a, ExecCtx& ctx);
int launch_gemm_simt(const GemmArgs& a, ExecCtx& ctx);
int launch_gemm_tc(const GemmArgs& a, ExecCtx& ctx, bool allow_few_rows = false);
// allow_few_rows: accept M < 64 (a weight-streaming problem: most rows of the 128-row tile are padding, the time is the weight read)
bool gemm_tc_supported(const GemmArgs& a, bool allow_few_rows = false);
bool gemm_tc_shape_ok(int64_t M, int64_t N, int64_t K);
// K > 0: the launch may cut the tiles of its last round along K (needs the context's GEMM workspace)
int gemm_tc_pick_bn(int64_t M, int64_t N, int sm_count, int64_t K = 0);
// Name of the tensor-core kernel variant launch_gemm_tc takes for a problem (and its tile width): the one dispatch rule.
const char* gemm_tc_variant(int64_t M, int64_t N, int64_t K, int sm_count, bool k_split, bool few_rows, int* bn_out, bool pairs = true);
const char* gemm_tc_mixed_variant(int64_t M, int64_t N, int64_t K, int sm_count, bool k_split, bool few_rows, int* bn_out, bool pairs = true);
int launch_split_tf32(const float* w, float* hi, float* lo, int64_t n, ExecCtx& ctx);
// mixed mode: hi = tf32(w) as fp32 [n], lo_bf16 = bf16(hi) [n] followed by bf16(w - hi) [n]
int launch_split_mixed(const float* w, float* hi, void* lo_bf16, int64_t n, ExecCtx& ctx);
int simt_tile_choice(int64_t M, int64_t N, int sm_count);
std::string gemm_variant_name(const GemmArgs& a, int gemm_mode, int sm_count, bool pairs = true);

struct F16GemmArgs {
    SplitMat x, w;
    bool bf16 = false;
    const float* bias = nullptr;
    const float* residual = nullptr;
    NormInput norm;                     // few-row products (x as fp32 rows): gamma != NULL: the rows are normalised first
    float* out = nullptr;               // fp32 result, or
    SplitOut split_out;                 // the result in split form (pitch N)
    // != NULL: the columns of the split result come scaled, 1 / scale of a row of w times the column's factor in col_inv, the bias times it in
    // col_bias (which stand for w.inv and bias); two fp16 planes in the bf16 mode too.  No scales or maxima of rows are written.  Where a
    // value of row r is NaN or infinite, bit r % bad_rows / bad_block of split_bad[r / bad_rows] is set.
    const float *col_inv = nullptr, *col_bias = nullptr;
    uint32_t* split_bad = nullptr;
    int bad_rows = 1, bad_block = 1;
    int64_t M = 0, N = 0, K = 0, ldo = 0;
    bool relu = false;
    float* vt_out = nullptr;            // as GemmArgs::vt_*
    unsigned char* vt_flags = nullptr;
    int64_t vt_col0 = 0;
    int vt_T = 0, vt_heads = 0, vt_n32 = 0;
};
// Convolution over channels-last images in split form with one scale per image (x.inv, x.amax: one entry per image, x.parts
// maxima each).  Filters in split form as [O, KH*KW, C padded to 64]; 1x1, stride 1, unpadded: [O, C].
// window: x is [N, H, WO + 3, 16] and a filter row covers four consecutive pixels at once, filters [O, KH, 4*16] (KW = 1).
struct ConvF16Args {
    SplitMat x, w, res;                 // res: residual, laid out like the output (planes == NULL: none)
    const float* bias = nullptr;
    float* out = nullptr;
    SplitOut split_out;                 // amax must be zero before the launch
    int N = 0, C = 0, H = 0, W = 0, O = 0, KH = 0, KW = 0, HO = 0, WO = 0;
    int pad_h = 0, pad_w = 0, dil_h = 1, dil_w = 1, str_h = 1, str_w = 1;
    bool relu = false, window = false;
};
bool conv_f16_shape_ok(int64_t n_pix, int64_t C, int64_t O, int64_t KH, int64_t KW, const int64_t* geom);   // geom: sh, sw, ph, pw, dh, dw, groups
int launch_conv_f16(const ConvF16Args& a, ExecCtx& ctx);
bool gemm_f16_shape_ok(int64_t M, int64_t N, int64_t K);
bool gemm_f16_vt_ok(const F16GemmArgs& a, const ExecCtx& ctx);
int launch_gemm_f16(const F16GemmArgs& a, ExecCtx& ctx);
std::string gemm_f16_variant_name(int64_t M, int64_t N, int64_t K, bool bf16, int sm_count);   // of tiles that are not cut inside clusters
bool gemm_f16_may_cut(int64_t M, int64_t N, int sm_count);   // the launch asks the device how many clusters it holds, and may cut
// How a product in split form is launched, and what it uses of the K-split workspace (host side, no device needed).
enum class F16Form { kRows, kBf16, kImages };
struct F16Limits {
    int sm_count = 148;
    bool pairs = true;
    int chunk_k = 0;                    // ExecCtx::tc_chunk_k
    size_t ws_bytes = 0;                // K-split workspace and its flags; 0: every tile is computed whole
    int64_t flag_count = 0;
    const int* clusters = nullptr;      // [cs]: clusters of cs CTAs (2 to 8, one per SM) that the device holds at once; NULL: tiles are not cut inside clusters
};
struct F16Plan {
    int variant = -1, epilogue_warps = 8, workers = 0, parts = 1, chunk_slabs = 1, cluster = 1;
    int64_t full = 0, tail = 0;         // whole tiles, and tiles cut along K into `parts`
    size_t ws_bytes = 0;
    int64_t flags = 0;
};
F16Plan gemm_f16_plan(int64_t M, int64_t N, int64_t K, F16Form form, const F16Limits& lim);
// The workspace an engine keeps: per SM one 128 x 256 partial tile and a flag for each epilogue warp of the instance that has most.
constexpr size_t kSplitTileBytes = size_t(128) * 256 * sizeof(float);
constexpr int kSplitFlagsPerSm = 16;
int gemm_f16_split_parts(int64_t N);    // partial maxima per row a split output of N columns needs room for
// kernels/split_form.cu.  l1_out (weights): the L1 norm of each row; bound = {largest of them, largest |bias|} (SplitMat::bound).
int launch_split_rows(const float* x, int64_t ld, int64_t M, int64_t K, bool bf16, const SplitOut& out, float* l1_out, ExecCtx& ctx);
int launch_weight_bound(const float* l1, int64_t rows, const float* bias, int64_t n, float* bound, ExecCtx& ctx);
// bound[n]: no |w_n · x + bias_n| exceeds it, x a row that a LayerNorm of width K with this gamma and beta has written
int launch_column_bounds(const float* w, int64_t rows, int64_t K, const float* gamma, const float* beta, const float* bias, float* bound, ExecCtx& ctx);
// The scales of Q, K and V in split form (kernels/attention_f16.cu), H heads of 64 columns: a power of two for each column of each.
// Arrays of 3 * 64 * H: Q's columns, K's, V's.  w_inv: 1 / scale of the weights' rows (NULL: 1), for Q, and for K and V.
struct AttnScales {
    const float *bound = nullptr, *q_winv = nullptr, *kv_winv = nullptr, *q_bias = nullptr, *kv_bias = nullptr;
    float *col_inv = nullptr, *col_bias = nullptr;   // F16GemmArgs
    float *score_inv = nullptr;                      // [H]: 1 / (scale of Q times scale of K), the same for all columns of a head
    float *v_inv = nullptr, *v_ctx = nullptr;        // [64 * H]: 1 / scale of V's columns; the same times the one scale of a context in split form
    float* ctx_inv = nullptr;                        // 1 / the latter
    int* unusable = nullptr;                         // set where a column's size is beyond what scales can serve
    int H = 0;
};
int launch_attention_scales(const AttnScales& s, ExecCtx& ctx);
// M <= 64 rows in fp32 FFMA (kernels/gemm_lanes.cu): w as the graph has it; of `a` the sizes, bias, residual, output and ReLU count
bool gemm_lanes_better(int64_t M, int64_t N, int64_t K, int sm_count);   // than the kernels on split form
int launch_gemm_lanes(const F16GemmArgs& a, const float* w, const float* x, int64_t ldx, ExecCtx& ctx);
// M <= 64 rows (kernels/gemm_rows.cu): x as fp32 rows, or NULL with a.x in split form; no split output, no transposed columns
bool gemm_rows_ok(int64_t M, int64_t N, int64_t K);
int launch_gemm_rows(const F16GemmArgs& a, const float* x, int64_t ldx, ExecCtx& ctx);
constexpr int kNormRowMax = 1024;   // longest row that the few-row kernels normalise
bool gemm_rows_streams(int64_t M, int64_t N, int sm_count);   // launch_gemm_f16_swapped (x in split form) is the better one
int launch_gemm_f16_swapped(const F16GemmArgs& a, ExecCtx& ctx);

// Launch as a programmatic dependent of the kernel before it in the stream (the kernel calls griddepcontrol.wait before it
// touches anything another kernel of the stream writes or reads).
template <class... KArgs, class... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = unsigned(cluster);
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// dependent(kernel, grid, block, smem, ctx)(args...): the same with the look of a kernel launch; errors surface in FXF_LAUNCHED.
template <class... KArgs>
struct DependentLaunch {
    void (*kernel)(KArgs...);
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
    template <class... Args>
    void operator()(Args... args) const { (void)launch_dependent(kernel, grid, block, smem, stream, 1, args...); }
};
template <class... KArgs>
inline DependentLaunch<KArgs...> dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, const ExecCtx& ctx) {
    return {kernel, grid, block, smem, ctx.stream};
}

// Convolution (stride 1 or 2) as an implicit GEMM on the tensor cores: channels-last activation x [N,H,W,C], weights
// repacked to [O, KH*KW*C] (tap-major, channel-minor) and split into TF32 hi/lo, channels-last output [N,HO,WO,O].
struct ConvTcArgs {
    const float* x = nullptr;
    const float *w_hi = nullptr, *w_lo = nullptr;
    bool w_is_bf16 = false;   // bf16 mode: w_hi points to the repacked filters as bf16
    const float* bias = nullptr;
    const float* residual = nullptr;   // optional, laid out like `out`
    float* out = nullptr;
    int N = 0, C = 0, H = 0, W = 0, O = 0, KH = 0, KW = 0, HO = 0, WO = 0;
    int pad_h = 0, pad_w = 0, dil_h = 1, dil_w = 1, str_h = 1, str_w = 1;
    bool relu = false;
};
bool conv_tc_shape_ok(int64_t n_pix, int C, int O);
// The Linear of a planned node applied to M rows that start at x_rows and lie ldx floats apart; row m of the result
// goes to out + m * ldo (+ the column offset of this rank's block when the node's output columns are sharded).
// split_rows: the same rows in split form where the tensor is kept so (x_rows is then not read).
int linear_on_rows(const NodePlan* plan, const float* x_rows, const SplitMat* split_rows, int64_t M, int64_t ldx, float* out, int64_t ldo, ExecCtx& ctx);
int launch_conv_tc(const ConvTcArgs& a, ExecCtx& ctx);
// w_oihw [O,C,KH,KW] -> TF32 hi/lo halves laid out [O,KH,KW,C]
int launch_convert_bf16(const float* w, void* out_bf16, int64_t n, ExecCtx& ctx);
int launch_conv_weight_bf16(const float* w_oihw, void* out_bf16_ohwi, int O, int C, int KH, int KW, ExecCtx& ctx);
int launch_conv_weight_split(const float* w_oihw, float* hi, float* lo, int O, int C, int KH, int KW, ExecCtx& ctx);

// Attention core on packed qkv [B,T,3D] (Q | K | V thirds, head h at columns h*hd) -> ctx [B,T,D].
struct AttnArgs {
    const float* qkv = nullptr;
    // Cross-attention: keys and values come from `kv` (rows of ld_kv floats, Tk rows per batch) while the queries
    // stay in `qkv`; self-attention leaves kv NULL and K/V are read from `qkv` with T rows.
    const float* kv = nullptr;
    int64_t ld_kv = 0;
    int Tk = 0;
    const uint8_t* mask = nullptr;
    float* ctx = nullptr;
    int B = 0, T = 0, H = 0, hd = 0;
    int64_t ld_qkv = 0;   // row stride of qkv (= 3*D of the full model, or of the local shard)
    int64_t q_off = 0, k_off = 0, v_off = 0;  // column offsets of the Q/K/V blocks inside a row
    int64_t ld_ctx = 0;
    int64_t mask_sb = 0, mask_sh = 0, mask_sq = 0, mask_sk = 0;  // mask strides (bytes): batch, head, query, key
    float scale_divisor = 1.f;
    // Tensor-core kernel only: the context in split form [B*T, H*hd] (or its bf16 plane) instead of `ctx`.  A context row is a convex
    // combination of V rows, so all of them share one scale, from |v| <= v_cap * v_bound[0] + v_bound[1].
    SplitOut split_ctx;
    bool split_bf16 = false;
    float v_cap = 0.f;                  // SplitMat::cap of the rows that V is projected from
    const float* v_bound = nullptr;     // SplitMat::bound of the projection
};
int launch_attention(const AttnArgs& a, ExecCtx& ctx);
// Sum `n` floats in place over the tensor-parallel ranks (NCCL all-reduce on ctx.stream); no-op for tp_size 1.
int tp_all_reduce_sum(float* buf, int64_t n, ExecCtx& ctx);
// Peer-memory exchanges (kernels/tp_exchange.cu) and the IPC exchange that sets them up (tp_comm.cpp).
bool p2p_all_reduce_usable(const float* buf, int64_t n, const ExecCtx& ctx);
int launch_p2p_all_reduce(float* buf, int64_t n, ExecCtx& ctx);
// sum of the ranks' partial [M,D] + residual -> x_out (own rows or all), LayerNorm of the rows -> y_out on every rank
bool tp_exchange_usable(const TpExchange& x, const float* partial, int64_t M, int64_t D, const ExecCtx& ctx);
int launch_tp_exchange(const TpExchange& x, const float* partial, int64_t M, int64_t D, ExecCtx& ctx, bool pushed = false);
// Pushed exchange: the product stores its rows straight into the owners' exchange windows (GemmArgs::push_out); `partial`
// is then unused.  Usable when the engine has a window of M*D floats and every rank owns a whole number of 128-row tiles.
bool tp_push_usable(int64_t M, int64_t D, const ExecCtx& ctx);
float* tp_push_window(int rank, const ExecCtx& ctx);
int tp_exchange_emulated(int n_ranks, const float* const* partial, const float* const* residual, float* const* x_out, float* const* y_out,
                         const float* gamma, const float* beta, float eps, int64_t M, int64_t D, int replicate_x, void* sync_mem, int budget_ms,
                         int skip_rank, cudaStream_t stream);
int tp_map_peers(void* comm, void* base, PeerMap* out);     // collective: every rank passes its own allocation
void tp_unmap_peers(void* comm, PeerMap* pm);               // collective as well
// Gather `bytes` from every rank into recv[rank * bytes ...] (NCCL all-gather on ctx.stream).
int tp_all_gather(const void* send, void* recv, int64_t bytes, ExecCtx& ctx);
// tcgen05 path (head_dim 64): needs 6*B*T*H*64 floats of scratch for the split, per-head operand copies
bool attention_tc_supported(const AttnArgs& a, int gemm_mode);
size_t attention_tc_scratch_bytes(int64_t B, int64_t T, int64_t H);
// Attention on Q, K and V in split form, a scale per column (kernels/attention_f16.cu).  The fields of AttnArgs name the layout
// (ld_qkv, ld_kv, offsets in elements of a plane; kv != NULL marks cross-attention), these the data.  The projections have put what is
// not finite into mask->bad.
struct AttnSplit {
    const uint16_t *q = nullptr, *kv = nullptr;
    int64_t q_plane = 0, kv_plane = 0;
    const AttnScales* scales = nullptr;
    const MaskBits* mask = nullptr;
};
int attention_f16_block(int64_t Tk);   // keys per block
size_t mask_bits_bytes(const FxfTensor& mask, int64_t B, int64_t T, int64_t Tk);
MaskBits mask_bits_at(const FxfTensor& mask, int64_t B, int64_t T, int64_t Tk, void* area);
int launch_mask_bits(const FxfTensor& mask, int64_t T, int64_t Tk, const MaskBits& m, ExecCtx& ctx);
bool attention_f16_ok(int64_t T, int64_t Tk, int64_t hd, float scale_divisor);
int launch_attention_f16(const AttnArgs& a, const AttnSplit& sp, ExecCtx& ctx);
// v_transposed: V^T and its finite flags are already in the scratch (written by the projection's epilogue)
int launch_attention_tc(const AttnArgs& a, float* split_scratch, ExecCtx& ctx, bool v_transposed = false);

}  // namespace fxf
