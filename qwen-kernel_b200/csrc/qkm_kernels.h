// Host-side launchers of the sm_100a kernels.  Every launcher enqueues on the
// given stream and returns the CUDA error of the launch (cudaSuccess on success);
// none of them synchronises.  `launches` (may be NULL) is incremented once per
// kernel launched.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/qk_moe.h"
#include "qkm_units.h"

namespace qkm {

struct Launch {
    cudaStream_t stream;
    uint64_t* launches;
    // programmatic dependent launch: the kernel may be scheduled while the previous kernel of the
    // stream is still running; it runs its set-up, then waits (pdl_wait) for that kernel's results
    bool pdl = false;
    void count(int n = 1) const { if (launches) *launches += (uint64_t)n; }
};

// Launch with or without the programmatic-serialization attribute.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(const Launch& L, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = L.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = L.pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// Raises a kernel's dynamic shared-memory limit, once per device (the call costs the host about as much as a launch).
template <auto Kernel>
inline cudaError_t allow_dynamic_smem(int bytes) {
    static std::atomic<uint64_t> done{0};   // a bit per device
    int dev = 0;
    if (const cudaError_t e = cudaGetDevice(&dev)) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
    return e;
}

#ifdef __CUDACC__
// Both are no-ops in a kernel launched without the attribute.  pdl_wait: every kernel this one
// depends on has finished and its stores are visible.  pdl_trigger: the next kernel of the
// stream may be scheduled now (it still waits for this one's end in its own pdl_wait).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// One unit of the prefill GEMMs: an expert, 256 rows of its matrices and up to 128 or 160
// of its pairs (pairs[pair_off .. pair_off + n)).
struct MmaItem {
    uint16_t expert;
    uint16_t rt;
    uint32_t pair_off;
    uint32_t n;
};

// ---- fused decode sequence (qkm_dec_route.cu, qkm_dec_gateup.cu, qkm_dec_down.cu) ---------------
// Several layers whose rows are at hand together go through one launch of each kernel; everything per layer lies one after the other,
// `n_tokens` (and so on) apart.
constexpr uint32_t kDecMaxLayers = 64, kDecCounters = 20;
// One expert (or the shared expert) with up to two of the tokens routed to it.  The gate/up kernel walks all n_ff rows of a group.
struct alignas(16) DecodeGroup {
    uint32_t head;     // expert | tokens (1 or 2) << 16 | shared << 24
    uint32_t pair[2];  // (token << 4) | slot; slot n_used: the shared expert
    uint32_t layer;    // of the layers that go together
    __host__ __device__ static uint32_t make_head(uint32_t expert, uint32_t ntok, uint32_t shared) { return expert | (ntok << 16) | (shared << 24); }
    __host__ __device__ uint32_t expert() const { return head & 0xFFFFu; }
    __host__ __device__ uint32_t ntok() const { return (head >> 16) & 255u; }
    __host__ __device__ bool shared() const { return (head >> 24) != 0; }
    __host__ __device__ uint32_t pair_of(uint32_t t) const { return t ? pair[1] : pair[0]; }   // t < ntok()
};
// A layer's (token, slot) pairs grouped by expert, ascending expert, then the shared expert's ceil(n_tokens / 2) groups
struct DecodeGroups {
    uint32_t* count;       // [layer]
    DecodeGroup* group;    // [layer][n_tokens * (n_used + 1)]
};
struct RouteDecodeArgs {
    struct Router { const uint8_t* w; const float* gis; } layer[kDecMaxLayers];   // [n_expert][n_embd] F32 or F16; [n_embd]
    const float* x;            // [n_tokens][n_embd] of the first layer
    uint64_t x_stride;         // floats from one layer's rows to the next one's
    qkm_sel *sel, *sel_last;   // out [layer][n_tokens]; the last layer's
    double* logits;            // scratch [layer][n_tokens][n_expert]
    uint32_t* counter;         // [layer][kDecCounters] zero words; left at zero
    int8_t* planes;            // out [layer][n_tokens][n_embd/256][8][256]: digit planes 0..3 and their negatives 4..7
    float* xscale;             // out [layer][n_tokens][n_embd/256] 2^-p
    DecodeGroups groups;       // out; NULL: none are made (one layer)
    uint32_t n_tokens, n_layers, pairs_per_block;   // the last one is the launcher's
    qkm_dims d;
};
bool route_decode_ok(const qkm_dims& d);
cudaError_t launch_route_decode(const Launch& L, uint32_t router_type, const RouteDecodeArgs& a);
// routed (IQ3_XXS) and shared (Q8_0) gate/up + SwiGLU over the groups
struct GateupDecodeArgs {
    struct Mats { const uint8_t *gate, *up, *sh_gate, *sh_up; } layer[kDecMaxLayers];   // routed experts' IQ3_XXS or IQ4_XS tiles (gateup_type), the shared expert's Q8_0 tiles
    const uint8_t* luts;            // decode_gateup_lut_bytes() bytes written by launch_decode_gateup_luts
    const int8_t* planes;
    const float* xscale;
    DecodeGroups groups;
    const qkm_sel* sel;             // one layer: its records, from which each block groups the pairs itself; NULL: the shared expert alone
    uint32_t n_tokens, n_layers;
    uint32_t gateup_type;           // QKM_TYPE_IQ3_XXS or QKM_TYPE_IQ4_XS
    float *h, *h_last;              // out [layer][n_tokens][n_used+1][n_ff]; the last layer's
    uint32_t* status;
    qkm_dims d;
};
size_t decode_gateup_lut_bytes();
cudaError_t launch_decode_gateup_luts(const Launch& L, uint8_t* luts);
bool decode_gateup_ok(const qkm_dims& d);
uint32_t decode_gateup_rows(uint32_t n_blocks);   // (layer, token) rows of several layers that go together, at most
cudaError_t launch_decode_gateup(const Launch& L, const GateupDecodeArgs& a, uint32_t n_blocks);
// routed (IQ4_XS) down + shared (Q8_0) down + weighted sum: y[t] = sum_s w_s D[ids_s] h[t][s] + w_shared DS h[t][n_used]
struct DownDecodeArgs {
    struct Mats { const uint8_t *w, *sh; } layer[kDecMaxLayers];   // routed experts' IQ4_XS or Q6_K tiles (launch_decode_down_any: NULL for the shared term alone); the
                                                                   // shared expert's Q8_0 tiles (NULL: no shared term)
    const uint8_t* lut;             // IQ4_XS form: decode_down_lut_bytes() bytes written by launch_decode_down_lut
    const float *h, *h_last;        // [layer][n_tokens][n_used+1][n_ff] f32 (encoded as int8 digit planes inside the kernels); the last layer's
    const qkm_sel *sel, *sel_last;
    float* y;                       // out [n_tokens][n_embd] of the first layer
    uint64_t y_stride;              // floats from one layer's rows to the next one's
    DecodeGroups groups;            // launch_decode_down_group; NULL: one layer, whose pairs each block groups itself
    float* contrib;                 // launch_decode_down_group: scratch [layer][n_tokens][n_used+1][n_embd]
    uint32_t n_tokens, n_layers;
    uint32_t* status;
    qkm_dims d;
};
#ifdef __CUDACC__
// layer of the batch's row `row`, and records and hidden rows of a layer
__device__ __forceinline__ uint32_t layer_of(const DownDecodeArgs& a, uint32_t row) { return a.n_layers == 1 ? 0u : row / a.n_tokens; }
__device__ __forceinline__ const qkm_sel* layer_sel(const DownDecodeArgs& a, uint32_t l) { return l + 1 == a.n_layers ? a.sel_last : a.sel + (size_t)l * a.n_tokens; }
__device__ __forceinline__ const float* layer_h(const DownDecodeArgs& a, uint32_t l) { return l + 1 == a.n_layers ? a.h_last : a.h + (size_t)l * a.n_tokens * (a.d.n_used + 1) * a.d.n_ff; }
#endif
bool decode_down_ok(const qkm_dims& d);
size_t decode_down_lut_bytes();
cudaError_t launch_decode_down_lut(const Launch& L, uint8_t* lut);
cudaError_t launch_decode_down(const Launch& L, const DownDecodeArgs& a, uint32_t n_blocks);
// the same with the routed experts as Q6_K tiles
cudaError_t launch_decode_down_q6k(const Launch& L, const DownDecodeArgs& a, uint32_t n_blocks);
// either type, other numbers of slots
bool decode_down_any_ok(const qkm_dims& d);
// either type, grouped by expert: may run, and is the faster one for n tokens
bool decode_down_group_ok(const qkm_dims& d);
bool decode_down_group_better(const qkm_dims& d, uint32_t type, uint32_t n);
cudaError_t launch_decode_down_group(const Launch& L, const DownDecodeArgs& a, uint32_t type, uint32_t n_blocks);
cudaError_t launch_decode_down_any(const Launch& L, const DownDecodeArgs& a, uint32_t type, uint32_t n_blocks);

// ---- qkm_wgemm.cu : tcgen05 GEMMs with quantised weights (batched prefill, dense projections)
constexpr uint16_t kSharedItem = 0xFFFFu;   // MmaItem::expert of the shared expert's units
size_t wgemm_table_bytes();
cudaError_t launch_wgemm_table(const Launch& L, uint8_t* out);
// x rows as f16 in the kernels' element order (0, 2, 1, 3 in every group of four), scaled per row by a power of two
// (inv_scale[row] undoes it); norm (optional): the rows' 2-norms; zero (optional): n_zero words set to zero on the way
cudaError_t launch_f16_rows(const Launch& L, const float* x, void* xh, float* inv_scale, float* norm, uint32_t n_rows, uint32_t K,
                            uint32_t* zero = nullptr, uint32_t n_zero = 0);
// rows that arrived as scaled f16 in their own element order: a copy in the kernels' order, and the norms
cudaError_t launch_f16_rows_in(const Launch& L, const void* in, const float* inv_scale, void* out, float* norm, uint32_t n_rows, uint32_t K);
// out[e] (zero before) = largest row 2-norm of matrix e (raw ggml rows), rounded up
cudaError_t launch_row_norm_max(const Launch& L, uint32_t type, const void* w, float* out, uint32_t n_mats, uint32_t rows, uint32_t K);
struct WgemmExperts {
    const void* w[2];          // routed tiles: gate and up, or down
    const void* sh[2];         // the shared expert's Q8_0 tiles
    const MmaItem* items;
    const uint32_t* n_items;   // device word
    uint32_t* ticket;          // device word, zero before the launch
    const uint32_t* pairs;
    const uint8_t* table;
    uint32_t* status;
    uint32_t n_experts;        // resident experts
    uint32_t n_sms;
    uint32_t tile;             // rows per unit that `items` were cut with
};
// h (f16, scaled per pair position, element order as above) = silu(gate x) * (up x); w_norm [2][n_experts + 1]
cudaError_t launch_wgemm_gateup(const Launch& L, const qkm_dims& d, uint32_t type, const WgemmExperts& x, const void* xrows,
                                const float* x_inv_scale, const float* x_norm, const float* w_norm, void* h, float* h_inv_scale, uint32_t max_units);
// contrib[pair position][n_embd] = routing weight * down h
cudaError_t launch_wgemm_down(const Launch& L, const qkm_dims& d, uint32_t type, const WgemmExperts& x, const void* h, uint64_t n_hrows,
                              const float* h_inv_scale, const qkm_sel* sel, float* contrib, uint32_t max_units);
// Dense quantised GEMM Y[n][M] = X[n][K] . W^T (W tile-ordered Q8_0 / IQ4_XS, M % 128 == 0, K % 256 == 0).
// Scratch: xh n*K f16, x_inv_scale n floats.  w_scale: the power of two by which the weights are multiplied as f16 operands.
cudaError_t launch_dense_gemm(const Launch& L, uint32_t type, const void* tiles, float w_scale, uint32_t M, uint32_t K, const float* x, uint32_t n_rows, float* y,
                              void* xh, float* x_inv_scale, const uint8_t* table, uint32_t n_sms, uint32_t* status);
// w_scale for a matrix whose largest |d| has the f16 bits d_bits
float dense_weight_scale(uint32_t type, uint32_t d_bits);

// ---- qkm_hrows.cu : hidden rows that the gate/up epilogue's scale served badly are made again
struct HiddenRows {
    const uint32_t *pairs, *pos_of;          // as launch_group_place writes them
    const qkm_sel* sel;
    const __half* xrows;                     // launch_f16_rows' output
    const float *x_inv_scale, *x_norm;
    const float* w_norm;                     // as for launch_wgemm_gateup
    const uint8_t *w[2], *sh[2];             // raw ggml rows: gate and up of the resident experts, of the shared expert
    __half* h;                               // in and out
    float* h_inv_scale;
    uint32_t n_tokens, n_used, n_expert, expert_first, expert_count, n_ff, n_embd;
};
cudaError_t launch_hidden_rows_check(const Launch& L, uint32_t type, const HiddenRows& a);

// ---- qkm_prefill.cu : router logits and the fold around them
cudaError_t launch_router_f16(const Launch& L, uint32_t router_type, const void* router, void* out, uint64_t n_elems);
cudaError_t launch_fold_pairs(const Launch& L, const qkm_dims& d, const float* contrib, const uint32_t* pos_of,
                              float* y, uint32_t n_tokens);

// ---- qkm_repack.cu : raw ggml -> tile layout (same bytes, see qkm_tiles.cuh)
cudaError_t launch_repack(const Launch& L, uint32_t type, const void* raw, void* out, uint32_t n_mats,
                          uint32_t rows, uint32_t K);
// *out (zero before) = largest finite |d| of a Q8_0 / IQ4_XS matrix's blocks (raw ggml rows), as f16 bits
cudaError_t launch_scale_max(const Launch& L, uint32_t type, const void* raw, uint32_t* out, uint32_t rows, uint32_t K);

// ---- qkm_gemv.cu
cudaError_t launch_dequant(const Launch& L, uint32_t type, const void* blocks, float* y, uint64_t n_elems);

// streamed form (bulk-copy ring) with the generic kernel for tail rows / unaligned tensors
cudaError_t launch_gemv_mma(const Launch& L, uint32_t type, const void* W, const float* x, float* y, uint32_t M,
                            uint32_t K, uint32_t n_sms, uint32_t* status, uint32_t* rows_done);
// 1..16 rows of x a pass, K split over a cluster of blocks (qkm_gemv_split.cu); x rows [0, *rows_done) are done
cudaError_t launch_gemv_split(const Launch& L, uint32_t type, const void* W, const float* x, float* y, uint32_t M, uint32_t K, uint32_t n,
                              uint32_t n_sms, uint32_t* rows_done);
cudaError_t launch_gemv_stream(const Launch& L, uint32_t type, const void* W, const float* x, float* y,
                               uint32_t M, uint32_t K, uint32_t n, uint32_t n_sms, uint32_t* status);

// ---- qkm_route.cu
// Scratch of launch_route_select: f32 logits (partial sums side by side) and f32 row norms, or f64
// logits for the small batches that are ranked in f64 directly.
size_t route_scratch_bytes(uint32_t n_tokens, uint32_t n_expert);
cudaError_t launch_logits(const Launch& L, const qkm_dims& d, uint32_t router_type, const void* router,
                          const float* x, float* logits, float* row_norm2, uint32_t n_tokens);
cudaError_t launch_select(const Launch& L, const qkm_dims& d, const float* logits, const float* gis,
                          const float* x, qkm_sel* sel, uint32_t n_tokens);
// norm2[e] = |router row e|^2; largest (zero before): their maximum; either may be NULL
cudaError_t launch_row_norm2(const Launch& L, const qkm_dims& d, uint32_t router_type, const void* router, float* norm2, float* largest);
struct RouteExtra {                      // all optional
    int8_t* xplanes = nullptr;           // out (at most 64 tokens): x rows as digit planes and their negatives [kb][8][256], and their scales [token][kb]
    float* xscale = nullptr;
    const void* x_f16 = nullptr;         // with these four (more than 64 tokens) the logits come from the tensor cores: rows and
    const float* x_f16_inv = nullptr;    // scales of launch_f16_rows, the router as launch_router_f16 wrote it, its rows' largest squared norm
    const void* router_f16 = nullptr;
    const float* router_norm2 = nullptr;
    uint32_t* status = nullptr;
    uint32_t* counts = nullptr;          // in zero, out: pairs per resident expert; ranks[t * n_used + s]: the pair's number inside its expert
    uint32_t* ranks = nullptr;
    uint32_t expert_first = 0, expert_count = 0;
};
cudaError_t launch_route_select(const Launch& L, const qkm_dims& d, uint32_t router_type, const void* router, const float* gis, const float* x, qkm_sel* sel,
                                uint32_t n_tokens, void* scratch, size_t scratch_bytes, const RouteExtra& extra = RouteExtra());
// ---- qkm_select.cu
struct SelectIn {
    const void* router;
    const void* logits;        // f64 (exact), or n_parts times [n_tokens][n_expert] f32 partial sums with an error bound
    const float *norm2, *gis, *x;
    int8_t* xplanes; float* xscale;
    uint32_t *counts, *ranks;
    uint32_t n_parts, n_norm, expert_first, expert_count;
    float eps_terms, eps_abs;  // |error of a logit| <= (eps_terms * |router row| + eps_abs) * |x| * 2^-24
    bool exact;
};
cudaError_t launch_select_tokens(const Launch& L, const qkm_dims& d, uint32_t router_type, const SelectIn& in, qkm_sel* sel, uint32_t n_tokens);
// counts (zero before) and ranks of records that were selected elsewhere
cudaError_t launch_group_rank(const Launch& L, const qkm_dims& d, const qkm_sel* sel, uint32_t n_tokens, uint32_t expert_first, uint32_t expert_count,
                              uint32_t* counts, uint32_t* ranks);
// work lists of the two expert GEMMs from counts and ranks
struct GroupPlace {
    const uint32_t *counts, *ranks;
    const qkm_sel* sel;
    uint32_t n_tokens, n_used, n_expert, expert_first, expert_count;   // expert_count 0: no routed pairs
    uint32_t sh_first, sh_count;                                       // rows of the shared expert
    uint32_t tile, rt_gu, rt_dn;                                       // pairs per unit; units per tile of pairs
    uint32_t *pairs, *pos_of;
    MmaItem *items_gu, *items_dn;
    uint32_t* n_items;         // out: [0], [1] units; [2], [3] zero
};
cudaError_t launch_group_place(const Launch& L, const GroupPlace& a);
#ifdef __CUDACC__
// Expert id -> index inside the resident range [expert_first, expert_first + expert_count);
// a result >= expert_count means "not here" (the subtraction wraps for ids below the range).
// With every expert resident an id past the table is clamped to the last expert, as the
// reference's moe_group_pairs.comp does; on a shard it marks an empty record that no rank
// takes (the peer-memory exchange fills unused slots with such records).
__device__ __forceinline__ uint32_t local_expert_of(uint32_t id, uint32_t n_expert, uint32_t expert_first,
                                                    uint32_t expert_count) {
    if (expert_count >= n_expert) return min(id, n_expert - 1) - expert_first;
    return id < n_expert ? id - expert_first : 0xFFFFFFFFu;
}

#endif
// f32 logits from f16 operands on the tensor cores (router_f16 as written by launch_router_f16, x_f16 / x_inv_scale by
// launch_f16_rows); |error| <= 2^-9 * |router row| * |x|.  Needs n_expert % 128 == 0 and n_embd <= 4096.
cudaError_t launch_logits_mma(const Launch& L, const qkm_dims& d, const void* router_f16,
                              const void* x_f16, const float* x_inv_scale, float* logits, uint32_t n_tokens,
                              uint32_t* status, uint32_t splits = 1)   /* splits > 1: partial logits over column ranges, [splits][n_tokens][n_expert] */;
cudaError_t launch_group_pairs(const Launch& L, const qkm_dims& d, const qkm_sel* sel, uint32_t n_tokens,
                               uint32_t* offsets, uint32_t* pairs, uint32_t expert_first,
                               uint32_t expert_count);
// ---- qkm_moe_simple.cu : one warp per output element, raw ggml layout
cudaError_t launch_gateup_tokens(const Launch& L, const qkm_dims& d, uint32_t type, const void* gate,
                                 const void* up, const float* x, const qkm_sel* sel, float* h,
                                 uint32_t n_tokens, uint32_t expert_first, uint32_t expert_count);
cudaError_t launch_gateup_pairs(const Launch& L, const qkm_dims& d, uint32_t type, const void* gate,
                                const void* up, const float* x, const uint32_t* offsets,
                                const uint32_t* pairs, float* h, uint32_t n_tokens,
                                uint32_t expert_first, uint32_t expert_count);
cudaError_t launch_shared_gateup(const Launch& L, const qkm_dims& d, const void* gate, const void* up,
                                 const float* x, float* h, uint32_t n_tokens);
cudaError_t launch_down_tokens(const Launch& L, const qkm_dims& d, uint32_t type, const void* down,
                               const float* h, const qkm_sel* sel, float* y, uint32_t n_tokens,
                               uint32_t expert_first, uint32_t expert_count,
                               const void* down_shared /* NULL: routed only */);
cudaError_t launch_down_pairs(const Launch& L, const qkm_dims& d, uint32_t type, const void* down,
                              const float* h, const qkm_sel* sel, const uint32_t* offsets,
                              const uint32_t* pairs, float* contrib, uint32_t n_tokens,
                              uint32_t expert_first, uint32_t expert_count);
// y2 = w_shared * shared down; with contrib != NULL: y2 = sum_s contrib[.][s][.] + that
cudaError_t launch_shared_down(const Launch& L, const qkm_dims& d, const void* down, const float* h,
                               const qkm_sel* sel, float* y2, uint32_t n_tokens,
                               const float* contrib = nullptr);
// y[t][o] = sum over slots (in order) of contrib[t][s][o], plus y2[t][o] when y2 != NULL
cudaError_t launch_fold_contrib(const Launch& L, const qkm_dims& d, const float* contrib, const float* y2,
                                float* y, uint32_t n_tokens);

// ---- residual adds fused with the RMS norm (qkm_tail.cu) ---------------------------------------
// mode 0: s = a + b; 1: s = a + b + c2; 2: s = a + sum_k b[row][k][:] + c2 (b = per-slot contributions).
// xn = s * w / sqrt(mean(s^2) + eps).
cudaError_t launch_add_rms(const Launch& L, int mode, const float* a, const float* b, const float* c2, const float* w,
                           float* s, float* xn, uint32_t n_rows, uint32_t n, uint32_t n_used, float eps);

// greedy token per row of logits: largest value, lowest index on ties (scratch: argmax_scratch_bytes(scratch_rows), zero before the first call)
size_t argmax_scratch_bytes(uint32_t n_rows);
cudaError_t launch_argmax(const Launch& L, const float* logits, uint32_t n_rows, uint32_t n, void* scratch, uint32_t scratch_rows, uint32_t* tok);

// ---- expert-parallel exchange helpers (qkm_ep.cu) --------------------------------------------
// counts[0..n_ranks) rows per destination rank and counts[n_ranks] their sum; send_tok the
// tokens in send order; send_pos[t][r] the row of token t among the rows sent (to rank r).
// Receive buffers of every rank as this rank sees them (its own, and the peers' mapped ones).
constexpr uint32_t kMaxPeerRanks = 16;
struct EpPeerTable {
    float* x[kMaxPeerRanks];          // [n_ranks * slot_rows][n_embd] rows pushed by the sources
    qkm_sel* sel[kMaxPeerRanks];      // their selection records
    float* back[kMaxPeerRanks];       // [n_ranks * slot_rows][n_embd] partial rows returned by the owners
    uint32_t* flags[kMaxPeerRanks];   // [n_ranks] barrier words, word s written by rank s
};
cudaError_t launch_ep_barrier(const Launch& L, const EpPeerTable& peers, uint32_t rank, uint32_t n_ranks, uint32_t epoch,
                              uint64_t limit_ns, uint32_t* status);
// xh / x_inv_scale: the rows as scaled f16 (launch_f16_rows) - then those travel instead of the f32 rows
cudaError_t launch_ep_push(const Launch& L, const qkm_dims& d, const float* x, const qkm_sel* sel, const EpPeerTable& peers,
                           uint32_t n_tokens, uint32_t slot_rows, uint32_t rank, uint32_t n_ranks, const void* xh = nullptr,
                           const float* x_inv_scale = nullptr);
cudaError_t launch_ep_row_scales(const Launch& L, const qkm_sel* selrecv, float* x_inv_scale, uint32_t n_rows);
constexpr uint32_t kSelScaleWord = 34;   // first padding word of a selection record (ids 0-15, w 16-31, w_shared, route_done, pad)
cudaError_t launch_fold_pairs_peer(const Launch& L, const qkm_dims& d, const float* contrib, const uint32_t* pos_of,
                                   const EpPeerTable& peers, uint32_t slot_rows, uint32_t rank, uint32_t n_ranks);
cudaError_t launch_ep_return(const Launch& L, const qkm_dims& d, const float* partial, const qkm_sel* selrecv,
                             const EpPeerTable& peers, uint32_t slot_rows, uint32_t rank, uint32_t n_ranks, uint32_t n_shared);
cudaError_t launch_ep_pull(const Launch& L, const qkm_dims& d, const qkm_sel* sel, const EpPeerTable& peers, const float* y2,
                           float* y, uint32_t n_tokens, uint32_t slot_rows, uint32_t rank, uint32_t n_ranks,
                           bool own_always);
cudaError_t launch_ep_plan(const Launch& L, const qkm_dims& d, const qkm_sel* sel, uint32_t n_tokens, uint32_t n_ranks,
                           uint32_t* counts, uint32_t* send_tok, uint32_t* send_pos);
cudaError_t launch_ep_pack(const Launch& L, const qkm_dims& d, const float* x, const qkm_sel* sel,
                           const uint32_t* send_tok, const uint32_t* total, uint32_t max_rows, float* xsend,
                           qkm_sel* selsend);
cudaError_t launch_ep_combine(const Launch& L, const qkm_dims& d, const float* back, const uint32_t* send_pos,
                              const float* y2, float* y, uint32_t n_tokens, uint32_t n_ranks);

}  // namespace qkm
