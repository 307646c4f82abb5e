// Quantised-weight GEMMs of batched prefill on the 5th-generation tensor cores (tcgen05 + TMEM): the experts'
// gate/up + SwiGLU, the experts' down projections and the dense projections, one persistent kernel for all formats.
//
// Replaces moe_gateup_iq3_grouped_coopmat.comp / moe_gateup_q8_coopmat.comp, moe_down_{iq4,q6k}_grouped_coopmat.comp /
// moe_down_q8_coopmat.comp and the batched projections gemm_q8_0*.comp / gemm_iq4_xs.comp.
//
// A unit of work is 256 weight rows (gate and up rows of one 128-row tile, or two consecutive row tiles of a down or
// dense matrix) times up to 128 (or 160, see qkm_units.h) activation rows.  Weights are the M = 128 operand and live in tensor memory: a
// producer thread owns one weight row, reads its quant bytes from shared memory, expands them to f16 and stores
// them with tcgen05.st; activation rows (f16, scaled per row by a power of two) are the N operand in shared memory.
//
// Who does what (32 warps, one block per SM, registers split between the warpgroups; a ticket hands out units, each role walks them on its own):
//   16 producer warps  row = lane of the four quarters x matrix x column-block parity.  The two parities work on
//                      different 256-column blocks (the k-steps of a block pair are interleaved, the order of a sum
//                      is free), so one half's look-up latency hides behind the other's
//   8 epilogue warps   TMEM -> SwiGLU / routing weight -> global; two accumulator sets while N <= 64, so the next
//                      unit's MMAs run meanwhile
//   1 MMA warp         tcgen05.mma kind::f16, A from TMEM, B from shared memory, commits free the stages
//   1 weight loader    takes the tickets; one bulk copy per matrix and 256-column block (eight consecutive 16-row tiles)
//   row loaders        activation rows into 128-byte swizzled tiles.  Scattered rows (gate/up) with 16-byte cp.async:
//                      TMA's tile::gather4 took about 60 cycles per four rows of 128 bytes and was the bound from
//                      64 rows on (588 us against 250 at 4096 tokens); consecutive rows (down, dense) by TMA boxes of 16 rows
//
// What bounds it: few rows per expert: the producers' instructions (nominally 1.5 to 3.3 per weight by format, 3.5 with
// barriers, address and scale work; issue slots 74 % busy in gate/up and 60 % in down at 77 tokens).  Measured per layer (256 experts,
// top 8), before (operands dequantised into shared memory or, for one format each, into TMEM by threads that also copied the rows)
// and now, the shared expert's units (82 us in kernels of its own before, beside the routed ones) included now:
//   gate/up IQ3_XXS   77 tokens 167 -> 88 us, 600: 176 -> 102, 4096: 301 -> 206
//   gate/up IQ4_XS    77: 340 -> 92, 600: 371 -> 107, 4096: 631 -> 214
//   down IQ4_XS       77: 133 -> 51, 600: 153 -> 62, 4096: 287 -> 150;   down Q6_K 600: 273 -> 76, 4096: 479 -> 165
//   dense 1000 x 4096 x 2048, Q8_0 and IQ4_XS: 103 -> 29 us each
//
// K order.  Inside every group of four columns the operands hold elements (0, 2, 1, 3): that is the order in which
// the bytes and nibbles of the tiles unpack to f16 pairs without a permute.  x and h rows are written in that order.
#include <cuda.h>
#include <cuda_fp16.h>

#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"
#include "qkm_tiles.cuh"
#include "qkm_umma.cuh"
#include "qkm_wait.h"

namespace qkm {

namespace wg {
constexpr int kProducerWarps = 16, kEpilogueWarps = 8;
constexpr int kMmaWarp = kProducerWarps + kEpilogueWarps, kWeightWarp = kMmaWarp + 1, kRowWarp = kMmaWarp + 2;
constexpr int kThreads = 1024;                  // eight warpgroups at 64 registers = all 65,536 of the SM
// Registers a thread after the split, producers / epilogue / others; 512 P + 256 E + 256 O must not exceed the launch's 65,536.
// (Gate/up with 160 rows: the row loaders' addresses; down: the epilogue, which is 40 % of a unit of eight k-steps, but for
// Q6_K, whose producers would spill.)
template <int FMT, int MODE, int NT> struct Regs { static constexpr int kProducer = 80, kEpilogue = 56, kOther = 40; };
template <int FMT> struct Regs<FMT, 0, 160> { static constexpr int kProducer = 72, kEpilogue = 56, kOther = 56; };
template <int NT> struct Regs<QKM_TYPE_IQ4_XS, 1, NT> { static constexpr int kProducer = 72, kEpilogue = 72, kOther = 40; };
template <int N> __device__ __forceinline__ void set_regs() {   // from the launch's 64
    static_assert(N % 8 == 0, "a multiple of eight");
    if constexpr (N > 64) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
    if constexpr (N < 64) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
constexpr int kFeed = 4;                        // units handed out ahead
// NT: activation rows per unit, 128 or 160.  Tensor memory's 512 columns hold two accumulators of NT and the A stages
constexpr int kNT = kWgemmRows, kWideNT = kWgemmRowsWide;
template <int NT> constexpr int stages() { return NT > 128 ? 3 : 4; }   // of (A: 64 TMEM columns, B: NT rows x 64 f16)
template <int NT> constexpr uint32_t b_tile() { return NT * 128; }
constexpr uint32_t kTab = 0x10000u, kTabBytes = 0x10000u, kLow = 0x1800u;
template <int FMT> constexpr bool has_table() { return FMT == QKM_TYPE_IQ3_XXS || FMT == QKM_TYPE_IQ4_XS; }
// Shared-window addresses.  With a table image (look-up addresses are byte permutes, so it has to start on a 64 KB
// boundary): all B stages but one below it, the last and the weight buffers above; else everything in one run.
template <int FMT, int NT> __device__ __forceinline__ uint32_t b_addr(uint32_t s) {
    return has_table<FMT>() && s + 1 == stages<NT>() ? kTab + kTabBytes : kLow + s * b_tile<NT>();
}
template <int FMT, int NT> constexpr uint32_t w_base() { return has_table<FMT>() ? kTab + kTabBytes + b_tile<NT>() : kLow + stages<NT>() * b_tile<NT>(); }
template <int FMT> constexpr uint32_t tile_size() {
    return FMT == QKM_TYPE_IQ3_XXS ? kTileIq3 : FMT == QKM_TYPE_IQ4_XS ? kTileIq4 : FMT == QKM_TYPE_Q6_K ? kTileQ6 : kTileQ8;
}
// Weight buffers, one per parity: 16 tiles of 256 columns, or two slots of 64 columns of the shared expert's Q8_0 tiles (those copies
// are of 1088 bytes and take about 90 cycles each, so the Q8_0 kernels load whole tiles: 41 -> 35 us at 1000 x 4096 x 2048)
template <int FMT> constexpr uint32_t q8_slots() { return FMT == QKM_TYPE_Q8_0 ? 1 : 2; }
constexpr uint32_t kQ8Slot = 16 * 1088;
template <int FMT> constexpr uint32_t w_bytes() {
    const uint32_t slots = q8_slots<FMT>() * kQ8Slot, tiles = 16u * tile_size<FMT>();
    return tiles > slots ? tiles : slots;
}
template <int FMT, int NT> constexpr uint32_t smem_end() { return w_base<FMT, NT>() + 2 * w_bytes<FMT>(); }
template <int NT> constexpr uint32_t tmem_a() { return 2 * NT; }   // accumulators first, A stages behind them
enum Mode { kGateUp = 0, kDown = 1, kDense = 2 };
template <int MODE> constexpr uint32_t warps_per_step() { return MODE == kGateUp ? 2 : 1; }   // row loaders
template <int MODE> constexpr uint32_t row_warps() { return MODE == kGateUp ? 6 : 1; }
}  // namespace wg

// ---- table image: row i (256 bytes) = IQ3_XXS grid entry i as f16 in element order (0, 2, 1, 3), 8 bytes for each of
// 16 lane columns; then the IQ4_XS pair (kvalues[i & 15], kvalues[i >> 4]) as f16, 4 bytes for each of 32 lanes.  A
// look-up of a warp never conflicts.
size_t wgemm_table_bytes() { return wg::kTabBytes; }
__global__ void wgemm_table_kernel(uint8_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;   // one 4-byte word each
    if (i >= wg::kTabBytes / 4) return;
    const uint32_t row = i >> 6, w = i & 63u;
    __half2 m;
    if (w < 32) {
        const uint32_t g = c_iq3_grid[row] >> (8 * (w & 1u));   // elements (0, 2) or (1, 3)
        m = __floats2half2_rn((float)(g & 0xFFu), (float)((g >> 16) & 0xFFu));
    } else {
        m = __floats2half2_rn((float)c_iq4_values[row & 15u], (float)c_iq4_values[row >> 4]);
    }
    reinterpret_cast<__half2*>(out)[i] = m;
}
cudaError_t launch_wgemm_table(const Launch& L, uint8_t* out) {
    wgemm_table_kernel<<<wg::kTabBytes / 4 / 256, 256, 0, L.stream>>>(out);
    L.count();
    return cudaGetLastError();
}

// ---- small helpers ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t prmt_wg(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ uint32_t lds_u16_wg(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t mul_h2(uint32_t a, __half2 s) {
    const __half2 v = __hmul2(*reinterpret_cast<const __half2*>(&a), s);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// value * (hi + lo) with one rounding to f16 that counts (value an integer below 2^8, lo = scale - hi)
struct Scale2 { __half2 hi, lo; };
__device__ __forceinline__ Scale2 split_scale(float s) {
    Scale2 r;
    const __half h = __float2half_rn(s);
    r.hi = __half2half2(h);
    r.lo = __half2half2(__float2half_rn(s - __half2float(h)));
    return r;
}
__device__ __forceinline__ uint32_t mul_h2(uint32_t a, const Scale2& s) {
    const __half2 v = *reinterpret_cast<const __half2*>(&a);
    const __half2 r = __hfma2(v, s.hi, __hmul2(v, s.lo));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t sub_h2(uint32_t a, __half2 b) {
    const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&a), b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// 32 lanes x 16 consecutive 32-bit columns of tensor memory: thread i of the warp writes lane (base lane + i)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
                 "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem]: A is 128 lanes (rows) x 8 columns (16 f16), B a K-major shared-memory tile
__device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, bool accumulate) {
    const uint32_t acc = accumulate ? 1u : 0u;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
// 16 consecutive rows x 64 columns from column x0, row r0 of the tensor map -> 2 KB at dst, swizzled
__device__ __forceinline__ void tma_rows16(uint32_t dst, const CUtensorMap* map, uint32_t x0, uint32_t r0, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x0), "r"(r0), "r"(bar) : "memory");
}

// ---- producers ---------------------------------------------------------------------------------------------
// 32 columns (one sub-block) of a thread's row -> 16 tensor-memory columns.

// IQ3_XXS: ix[t] = the index half-word of group t (in byte 0/1 or 2/3: HI), sg[t] = the sign word that covers the sub-block
// (bit positions in qkm_tiles.cuh), j = 2 (sub-block & 3).  Per 8 weights two address permutes, two loads, four packed
// multiplies by the sub-block scale, four shifts and four xor-and (16 instructions).
template <bool HI>
__device__ __forceinline__ void make_iq3(uint32_t (&o)[16], const uint32_t (&ix)[4], const uint32_t (&sg)[4], uint32_t j, __half2 s, uint32_t tab_c) {
    constexpr uint32_t s0 = HI ? 0x7624u : 0x7604u, s1 = HI ? 0x7634u : 0x7614u;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const uint2 m0 = lds64(prmt_wg(ix[t], tab_c, s0)), m1 = lds64(prmt_wg(ix[t], tab_c, s1));
        o[4 * t] = m0.x; o[4 * t + 1] = m0.y; o[4 * t + 2] = m1.x; o[4 * t + 3] = m1.y;
    }
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {   // elements 4h .. 4h+3 of the group
            const uint32_t w = sg[t], k = j + h;
            o[4 * t + 2 * h] = mul_h2(o[4 * t + 2 * h], s) ^ ((w << (8 + k)) & 0x80008000u);
            o[4 * t + 2 * h + 1] = mul_h2(o[4 * t + 2 * h + 1], s) ^ ((w << k) & 0x80008000u);
        }
}

// IQ4_XS: w[t] = quant word of group t: four look-ups of value pairs
template <class S>
__device__ __forceinline__ void make_iq4(uint32_t (&o)[16], const uint32_t (&w)[4], const S& s, uint32_t tab_c) {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        o[4 * t + 0] = lds32(prmt_wg(w[t], tab_c, 0x7604u));
        o[4 * t + 1] = lds32(prmt_wg(w[t], tab_c, 0x7614u));
        o[4 * t + 2] = lds32(prmt_wg(w[t], tab_c, 0x7624u));
        o[4 * t + 3] = lds32(prmt_wg(w[t], tab_c, 0x7634u));
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] = mul_h2(o[i], s);
}

// four unsigned bytes v -> f16 pairs (bytes 0, 2) and (1, 3) of 1024 + byte, minus `bias`, times the scale
template <class S>
__device__ __forceinline__ void bytes_to_h2(uint32_t v, __half2 bias, const S& s, uint32_t& p02, uint32_t& p13) {
    p02 = mul_h2(sub_h2((v & 0x00FF00FFu) | 0x64006400u, bias), s);
    p13 = mul_h2(sub_h2(((v >> 8) & 0x00FF00FFu) | 0x64006400u, bias), s);
}

// Q8_0: q0, q1 = the row's 32 quant bytes of a block (tile order: words t of elements 4t.. and 16 + 4t.. alternate)
template <class S>
__device__ __forceinline__ void make_q8(uint32_t (&o)[16], const uint4& q0, const uint4& q1, const S& s) {
    const __half2 bias = __float2half2_rn(1152.f);   // 1024 + 128: the bytes have their top bit flipped
    const uint32_t w[8] = {q0.x, q0.z, q1.x, q1.z, q0.y, q0.w, q1.y, q1.w};   // elements 4m .. 4m+3
#pragma unroll
    for (int i = 0; i < 8; ++i) bytes_to_h2(w[i] ^ 0x80808080u, bias, s, o[2 * i], o[2 * i + 1]);
}

// Q6_K: 32 columns: wl / wh [m] = ql / qh words of elements 4m .. 4m+3, NIB: high nibbles, hs = 2 * quarter; scales of the two 16-column groups
template <bool NIB>
__device__ __forceinline__ void make_q6(uint32_t (&o)[16], const uint32_t (&wl)[8], const uint32_t (&wh)[8], uint32_t hs, float s0, float s1) {
    const __half2 bias = __float2half2_rn(1056.f);   // 1024 + 32
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const Scale2 s = split_scale(h ? s1 : s0);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t lo = (NIB ? wl[4 * h + i] >> 4 : wl[4 * h + i]) & 0x0F0F0F0Fu;
            const uint32_t hi = (hs >= 4 ? wh[4 * h + i] >> (hs - 4) : wh[4 * h + i] << (4 - hs)) & 0x30303030u;
            bytes_to_h2(lo | hi, bias, s, o[8 * h + 2 * i], o[8 * h + 2 * i + 1]);
        }
    }
}

struct WgemmArgs {
    const uint8_t* w[2];        // routed (or dense) tiles: gate and up, or the one matrix twice
    const uint8_t* sh[2];       // the shared expert's Q8_0 tiles, likewise
    const MmaItem* items;       // expert kSharedItem: the shared expert; rt counts 128-row tiles (gate/up) or pairs of them
    const uint32_t* n_items;    // device word; unused by the dense form
    uint32_t* ticket;           // device word, zero before; NULL: units in a fixed stride
    const __half* xrows;        // gate/up: activation rows [token][K]
    const uint32_t* pairs;      // (token << 4) | slot in grouped order; unused by the dense form
    const float* x_inv_scale;   // gate/up: per token; dense: per row
    const float* x_norm;        // gate/up: 2-norm of the token's row
    const float* w_norm;        // gate/up: [2][experts + 1] largest row norm of an expert's gate / up matrix, the shared expert last
    __half* h;                  // gate/up out: [pair position][rows] f16, scaled per pair
    float* h_inv_scale;         // gate/up out, down in: per pair position
    const qkm_sel* sel;         // down: routing weights
    float* out;                 // down: contributions [pair position][rows]; dense: y [n][rows]
    const uint8_t* table;
    uint32_t* status;
    uint32_t rows, K;           // weight rows of a matrix, columns
    uint32_t n_experts, n_used; // resident experts
    uint32_t n_dense;           // dense: activation rows
    float w_scale, w_inv_scale; // dense: power of two on the weights as operands, and what undoes it
};

template <int FMT, int MODE, int NT>
__global__ void __launch_bounds__(wg::kThreads, 1)
wgemm_kernel(const WgemmArgs a, const __grid_constant__ CUtensorMap rows_map) {
    extern __shared__ __align__(1024) uint8_t smem_dyn[];
    constexpr int kSt = wg::stages<NT>();
    using R = wg::Regs<FMT, MODE, NT>;
    static_assert(wg::kProducerWarps * 32 * R::kProducer + wg::kEpilogueWarps * 32 * R::kEpilogue + (32 - wg::kProducerWarps - wg::kEpilogueWarps) * 32 * R::kOther <= wg::kThreads * 64,
                  "the shares must not exceed the launch's registers");
    static_assert(wg::tmem_a<NT>() + kSt * 64 <= 512 && (!wg::has_table<FMT>() || wg::kLow + (kSt - 1) * wg::b_tile<NT>() <= wg::kTab), "room");
    constexpr uint32_t kSlots = wg::q8_slots<FMT>(), kRowWarps = wg::row_warps<MODE>(), kPer = wg::warps_per_step<MODE>();
    static_assert(wg::kRowWarp + kRowWarps <= 32, "room");
    __shared__ __align__(8) unsigned long long s_bar[2 * kSt + 4 * kSlots + 6 + 2 * wg::kFeed];
    __shared__ MmaItem s_feed[wg::kFeed];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(16) uint32_t s_rows[MODE == wg::kGateUp ? kRowWarps : 1][NT / kPer];   // row loaders: where the unit's rows start, [row % 4][row / 4]
    __shared__ float s_col[2][2][NT];   // epilogue, per unit parity: factors of the unit's columns
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t KB = a.K / 256, RT16 = a.rows / 16;
    const uint32_t row_units = MODE == wg::kGateUp ? a.rows / 128 : (a.rows / 128 + 1) / 2;
    {   // the fixed addresses must lie inside the dynamic area
        const uint32_t dyn_base = smem_addr(smem_dyn);
        uint32_t dyn_size;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_size));
        if (dyn_base > wg::kLow || dyn_base + dyn_size < wg::smem_end<FMT, NT>()) {
            if (tid == 0) atomicExch(a.status, (uint32_t)kStatusBadLayout);
            return;
        }
    }
    const uint32_t bar = smem_addr(&s_bar[0]);
    const uint32_t bar_full = bar, bar_empty = bar + 8 * kSt, bar_wfull = bar + 16 * kSt, bar_wempty = bar_wfull + 16 * kSlots;   // [parity][slot]
    const uint32_t bar_accfull = bar_wempty + 16 * kSlots, bar_accfree = bar_accfull + 16, bar_tab = bar_accfree + 16;
    const uint32_t bar_ufull = bar_tab + 8, bar_uempty = bar_ufull + 8 * wg::kFeed;
    const uint32_t bar_cols = bar_uempty + 8 * wg::kFeed;   // the epilogue's warps among themselves
    if (tid == 0) {
        for (int s = 0; s < kSt; ++s) { mbar_init(bar_full + 8 * s, 8 + kPer); mbar_init(bar_empty + 8 * s, 1); }   // eight producer warps + the row loaders; one commit
        for (uint32_t b = 0; b < 2 * kSlots; ++b) { mbar_init(bar_wfull + 8 * b, 1); mbar_init(bar_wempty + 8 * b, 8); }
        for (int b = 0; b < wg::kFeed; ++b) { mbar_init(bar_ufull + 8 * b, 1); mbar_init(bar_uempty + 8 * b, wg::kProducerWarps + wg::kEpilogueWarps + 1 + kRowWarps); }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_accfull + 8 * b, 1); mbar_init(bar_accfree + 8 * b, wg::kEpilogueWarps);
        }
        mbar_init(bar_tab, 1);
        mbar_init(bar_cols, wg::kEpilogueWarps);
        mbar_fence_init();
        if (wg::has_table<FMT>()) {   // does not depend on the kernel before either
            mbar_expect_tx(bar_tab, wg::kTabBytes);
            for (uint32_t i = 0; i < 4; ++i) bulk_g2s(wg::kTab + i * 16384u, a.table + i * 16384u, 16384u, bar_tab);
        }
    }
    if (warp == 0) { umma::tmem_alloc(smem_addr(&s_tmem), 512); umma::tmem_relinquish(); }
    umma::fence_before_sync();
    pdl_trigger();
    // What depends on the kernel before: the work lists and everything read by their indices.  A dense matrix's units are known: its
    // weights are fetched and expanded while the kernel that writes the activation rows ends.
    if (MODE != wg::kDense) pdl_wait();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t n_units = MODE == wg::kDense ? (a.n_dense + NT - 1) / NT * row_units : *a.n_items;
    const uint32_t tmem = s_tmem;
    Waits waits;
    auto wait_bar = [&](uint32_t b, uint32_t parity) { waits.wait([&] { return mbar_wait_timed(b, parity); }); };

    auto unit_item = [&](uint32_t u) -> MmaItem {
        if (MODE != wg::kDense) return a.items[u];
        MmaItem it;
        it.expert = 0;
        it.rt = (uint16_t)(u % row_units);
        it.pair_off = (u / row_units) * NT;
        it.n = min((uint32_t)NT, a.n_dense - it.pair_off);
        return it;
    };
    // the k-th unit of this block, from the weight loader; false after the last
    auto next_unit = [&](uint32_t k, MmaItem& it) -> bool {
        const uint32_t s = k % wg::kFeed;
        if (!waits.next([&] { return mbar_wait_timed(bar_ufull + 8 * s, (k / wg::kFeed) & 1u); }, [](bool out) { return __any_sync(0xFFFFFFFFu, out) != 0; }))
            return false;   // the same for the whole warp
        it = s_feed[s];
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_uempty + 8 * s);
        return it.n != 0;
    };
    // k-step i of a unit: 256-column block and 64-column quarter.  Blocks 2p and 2p + 1 are interleaved (see above).  Of a lone last
    // block (dense matrices only) both producer groups get a copy and expand every other quarter, so that a stage always belongs to the same group.
    auto step_kb = [&](uint32_t i) -> uint32_t { return i < (KB & ~1u) * 4 ? 2 * (i >> 3) + (i & 1u) : KB - 1; };
    auto step_q = [&](uint32_t i) -> uint32_t { return i < (KB & ~1u) * 4 ? (i >> 1) & 3u : i & 3u; };
    const uint32_t KS = KB * 4;
    // stage of k-step i of a unit, and how often the stage was used earlier; `before` grows by `advance` a unit: k-steps, or rounds of four stages
    const uint32_t advance = kSt == 4 ? KB : KS;
    auto stage_of = [](uint32_t before, uint32_t i) -> uint32_t { return kSt == 4 ? i & 3u : (before + i) % kSt; };
    auto round_of = [](uint32_t before, uint32_t i) -> uint32_t { return kSt == 4 ? before + (i >> 2) : (before + i) / kSt; };

    if (warp < (uint32_t)wg::kProducerWarps) {
        // ---- producers
        wg::set_regs<R::kProducer>();
        const uint32_t lq = warp & 3u, mat = (warp >> 2) & 1u, par = warp >> 3;
        const uint32_t r = 32 * lq + lane, r16 = r & 15u, g = r16 & 7u, tl = r >> 4;   // row of the 128, row of its tile, tile
        const uint32_t a_lane = tmem + ((32 * lq) << 16) + wg::tmem_a<NT>() + mat * 32u;
        const uint32_t wbuf = wg::w_base<FMT, NT>() + par * wg::w_bytes<FMT>();
        const uint32_t tab_c = wg::kTab + (FMT == QKM_TYPE_IQ3_XXS ? (lane & 15u) * 8u : 128u + lane * 4u);
        if (FMT == QKM_TYPE_IQ3_XXS || FMT == QKM_TYPE_IQ4_XS)
            wait_bar(bar_tab, 0);
        // dense: scale and product rounded to f16 (two roundings of 2^-11 at most, a fifth fewer instructions); experts: one rounding that counts
        auto weight_scale = [&](float v) { if constexpr (MODE == wg::kDense) return __float2half2_rn(v * a.w_scale); else return split_scale(v); };
        uint32_t before = 0, wcnt = 0, qcnt = 0;   // what came before this unit; blocks and Q8_0 slots consumed
        MmaItem it;
        for (uint32_t k = 0; next_unit(k, it); ++k, before += advance) {
            const bool shared = MODE != wg::kDense && it.expert == kSharedItem;
            // A step's stores are not waited for at its end: it is announced when the next step's first values have been computed,
            // by which time they are through (waiting at once cost a tenth of the kernel).
            uint32_t pending = 0xFFFFFFFFu, st = 0;
            auto announce = [&]() {
                if (pending == 0xFFFFFFFFu) return;
                tmem_st_wait();
                umma::fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_full + 8 * pending);
            };
            auto store = [&](uint32_t i, uint32_t half, const uint32_t (&o)[16]) {   // half `half` of k-step i's 64 columns
                if (half == 0) {
                    announce();
                    const uint32_t stage = stage_of(before, i), round = round_of(before, i);   // the stage is free to be written
                    if (round) wait_bar(bar_empty + 8 * stage, (round - 1) & 1u);
                    umma::fence_after_sync();
                    st = a_lane + stage * 64u;
                    pending = stage;
                }
                tmem_st16(st + 16 * half, o);
            };
            auto w_wait = [&]() {
                // slot 0's barrier counts blocks and every kSlots-th Q8_0 slot
                wait_bar(bar_wfull + 8 * kSlots * par, (wcnt + qcnt / kSlots) & 1u);
                ++wcnt;
            };
            auto w_free = [&]() {
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_wempty + 8 * kSlots * par);
            };
            for (uint32_t kp = 0; kp < KB; kp += 2) {
                const bool lone = MODE == wg::kDense && kp + 1 == KB;
                const uint32_t i0 = lone ? kp * 4 : kp * 4 + par, istep = lone ? 1u : 2u;   // the block's k-steps: i0 + q * istep
                if (shared) {
                    // Q8_0, 64 columns a slot: two 544-byte pieces of each tile
#pragma unroll 1
                    for (uint32_t q = lone ? par : 0; q < 4; q += lone ? 2 : 1, ++qcnt) {
                        const uint32_t slot = qcnt % kSlots, bars = 8 * (kSlots * par + slot);
                        wait_bar(bar_wfull + bars, (qcnt / kSlots + (slot ? 0u : wcnt)) & 1u);
                        const uint32_t t0 = wbuf + slot * wg::kQ8Slot + (mat * 8 + tl) * 1088u;
                        uint4 v[2][2];
                        float d[2];
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            const uint32_t p = t0 + s * 544u;
                            v[s][0] = lds128(p + 32 + ((r16 >> 3) * 32 + 4 * g) * 8);
                            v[s][1] = lds128(p + 48 + ((r16 >> 3) * 32 + 4 * g) * 8);
                            d[s] = f16_bits_to_f32(lds_u16_wg(p + 2 * r16));
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_wempty + bars);
                        uint32_t o[16];
                        make_q8(o, v[0][0], v[0][1], weight_scale(d[0]));
                        store(i0 + q * istep, 0, o);
                        make_q8(o, v[1][0], v[1][1], weight_scale(d[1]));
                        store(i0 + q * istep, 1, o);
                    }
                    continue;
                }
                w_wait();
                const uint32_t tb = wbuf + (mat * 8 + tl) * wg::tile_size<FMT>();
                if constexpr (FMT == QKM_TYPE_IQ3_XXS) {
                    uint4 ix[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) ix[t] = lds128(tb + 64 * r16 + piece_at(r16, t));
                    uint32_t sg[2][4];   // [word q][t]
#pragma unroll
                    for (int tp = 0; tp < 2; ++tp) {
                        const uint4 v = lds128(tb + 1024 + 32 * r16 + 16 * (tp ^ ((r16 >> 2) & 1u)));
                        sg[0][2 * tp] = v.x; sg[1][2 * tp] = v.y; sg[0][2 * tp + 1] = v.z; sg[1][2 * tp + 1] = v.w;
                    }
                    const uint2 sc = lds64(tb + 1536 + 8 * r16);
                    const float d4 = f16_bits_to_f32(lds_u16_wg(tb + 1664 + 2 * r16)) * 0.25f;
                    w_free();
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (lone && ((q ^ par) & 1u)) continue;
                        // sub-blocks 2q, 2q + 1: scale d (2s + 1) / 4, exact in f32, one rounding to f16
                        const uint32_t w4 = q < 2 ? sc.x : sc.y, sh = 16 * (q & 1);
                        const __half2 s0 = __float2half2_rn(d4 * (float)((w4 >> sh) & 255u)), s1 = __float2half2_rn(d4 * (float)((w4 >> (sh + 8)) & 255u));
                        const uint32_t w[4] = {q == 0 ? ix[0].x : q == 1 ? ix[0].y : q == 2 ? ix[0].z : ix[0].w, q == 0 ? ix[1].x : q == 1 ? ix[1].y : q == 2 ? ix[1].z : ix[1].w,
                                               q == 0 ? ix[2].x : q == 1 ? ix[2].y : q == 2 ? ix[2].z : ix[2].w, q == 0 ? ix[3].x : q == 1 ? ix[3].y : q == 2 ? ix[3].z : ix[3].w};
                        uint32_t o[16];
                        make_iq3<false>(o, w, sg[q >> 1], 4 * (q & 1), s0, tab_c);
                        store(i0 + q * istep, 0, o);
                        make_iq3<true>(o, w, sg[q >> 1], 4 * (q & 1) + 2, s1, tab_c);
                        store(i0 + q * istep, 1, o);
                    }
                } else if constexpr (FMT == QKM_TYPE_IQ4_XS) {
                    const uint2 hd = lds64(tb + 16 * g + 8 * (r16 >> 3));   // d | scales_h << 16, scales_l
                    const float d = f16_bits_to_f32(hd.x & 0xFFFFu);
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        uint4 v[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t) v[t] = lds128(tb + 128 + 1024 * hf + 64 * r16 + piece_at(r16, t));
                        if (hf) w_free();
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            if (lone && ((q ^ par) & 1u)) continue;
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int sb = 4 * hf + 2 * q + s;
                                const int ls = (int)(((hd.y >> (4 * sb)) & 15u) | (((hd.x >> (16 + 2 * sb)) & 3u) << 4)) - 32;
                                const float dl = d * (float)ls;
                                const int c = 2 * q + s;
                                const uint32_t w[4] = {c == 0 ? v[0].x : c == 1 ? v[0].y : c == 2 ? v[0].z : v[0].w, c == 0 ? v[1].x : c == 1 ? v[1].y : c == 2 ? v[1].z : v[1].w,
                                                       c == 0 ? v[2].x : c == 1 ? v[2].y : c == 2 ? v[2].z : v[2].w, c == 0 ? v[3].x : c == 1 ? v[3].y : c == 2 ? v[3].z : v[3].w};
                                uint32_t o[16];
                                if (MODE == wg::kDown) make_iq4(o, w, __float2half2_rn(dl), tab_c);   // two roundings of 2^-12
                                else make_iq4(o, w, weight_scale(dl), tab_c);
                                store(i0 + (2 * hf + q) * istep, s, o);
                            }
                        }
                    }
                } else if constexpr (FMT == QKM_TYPE_Q6_K) {   // k-step k-step q = half q / 2, quarters 2 (q & 1) and the one after it: nibble q & 1 of both 32-byte runs
                    uint4 hq[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) hq[t] = lds128(tb + 2304 + 64 * r16 + piece_at(r16, t));
                    const uint4 sc = lds128(tb + 16 * r16);   // eight even groups, eight odd groups
                    const float d = f16_bits_to_f32(lds_u16_wg(tb + 3328 + 2 * r16));
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        uint4 v[4];
#pragma unroll
                        for (int t = 0; t < 4; ++t) v[t] = lds128(tb + 256 + 1024 * hf + 64 * r16 + piece_at(r16, t));
                        if (hf) w_free();
                        uint32_t wh[8];
#pragma unroll
                        for (int t = 0; t < 4; ++t) { wh[t] = hf ? hq[t].z : hq[t].x; wh[4 + t] = hf ? hq[t].w : hq[t].y; }
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            if (lone && ((q ^ par) & 1u)) continue;
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int qd = 2 * q + s;
                                uint32_t wl[8];
#pragma unroll
                                for (int t = 0; t < 4; ++t) { wl[t] = s ? v[t].z : v[t].x; wl[4 + t] = s ? v[t].w : v[t].y; }
                                const float f0 = d * (float)(int8_t)((hf ? sc.y : sc.x) >> (8 * qd)), f1 = d * (float)(int8_t)((hf ? sc.w : sc.z) >> (8 * qd));
                                uint32_t o[16];
                                if (q) make_q6<true>(o, wl, wh, 2 * qd, f0, f1);
                                else make_q6<false>(o, wl, wh, 2 * qd, f0, f1);
                                store(i0 + (2 * hf + q) * istep, s, o);
                            }
                        }
                    }
                } else {   // Q8_0
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const bool skip = lone && ((q ^ par) & 1u);
                        uint4 v[2][2];
                        float d[2];
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            const uint32_t p = tb + (2 * q + s) * 544u;
                            v[s][0] = lds128(p + 32 + ((r16 >> 3) * 32 + 4 * g) * 8);
                            v[s][1] = lds128(p + 48 + ((r16 >> 3) * 32 + 4 * g) * 8);
                            d[s] = f16_bits_to_f32(lds_u16_wg(p + 2 * r16));
                        }
                        if (q == 3) w_free();
                        if (skip) continue;
                        uint32_t o[16];
                        make_q8(o, v[0][0], v[0][1], weight_scale(d[0]));
                        store(i0 + q * istep, 0, o);
                        make_q8(o, v[1][0], v[1][1], weight_scale(d[1]));
                        store(i0 + q * istep, 1, o);
                    }
                }
            }
            announce();
        }
    } else if (warp < (uint32_t)wg::kMmaWarp) {
        // ---- epilogue: warps e and e + 4 read TMEM lanes 32 e .. 32 e + 31, every other 16 columns each (with four warps the drain of
        // 128 columns took 13,000 cycles a gate/up unit, a third of the time at 4096 tokens)
        wg::set_regs<R::kEpilogue>();
        if (MODE == wg::kDense) pdl_wait();
        const uint32_t e = warp & 3u, eh = (warp >> 2) & 1u, c = tid - wg::kProducerWarps * 32;   // c: the column this thread prepares
        uint32_t used[2] = {0, 0}, next = 0, iter = 0;
        MmaItem it;
        for (; next_unit(iter, it); ++iter) {
            const uint32_t n = it.n, n_mma = (n + 15u) & ~15u;
            const bool big = n_mma > 64;
            float* f0 = s_col[iter & 1u][0];
            float* f1 = s_col[iter & 1u][1];
            if (c < n) {
                const uint32_t p = it.pair_off + c;
                if (MODE == wg::kGateUp) {
                    const uint32_t tok = a.pairs[p] >> 4, ex = it.expert == kSharedItem ? a.n_experts : it.expert;
                    // |h| <= |g| |u| <= (largest gate row norm x |x|) (largest up row norm x |x|): a power of two that keeps every h below
                    // 2^15 without knowing the row.  Loose by 2^7 to 2^13 as a rule, which f16 affords (2^-14 .. 2^15 at full precision)
                    const float xn = a.x_norm[tok], bound = (a.w_norm[ex] * xn) * (a.w_norm[a.n_experts + 1 + ex] * xn);
                    int q = 0;
                    if (bound > 0.f && bound <= 3.0e38f) { int b; frexpf(bound, &b); q = max(-126, min(126, 14 - b)); }
                    f0[c] = a.x_inv_scale[tok];
                    f1[c] = ldexpf(1.0f, q);
                    if (it.rt == 0) a.h_inv_scale[p] = ldexpf(1.0f, -q);
                } else if (MODE == wg::kDown) {
                    const uint32_t pr = a.pairs[p], tok = pr >> 4, slot = pr & 15u;
                    f0[c] = (slot < a.n_used ? a.sel[tok].w[slot] : a.sel[tok].w_shared) * a.h_inv_scale[p];
                } else {
                    f0[c] = a.x_inv_scale[p] * a.w_inv_scale;
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_cols);
            wait_bar(bar_cols, iter & 1u);
            const uint32_t b = big ? 0u : next;
            wait_bar(bar_accfull + 8 * b, used[b] & 1u);
            if (big) { wait_bar(bar_accfull + 8, used[1] & 1u); ++used[0]; ++used[1]; next = 0; }
            else { ++used[b]; next ^= 1u; }
            umma::fence_after_sync();
            const uint32_t t0 = tmem + ((32 * e) << 16) + b * 128u, t1 = t0 + (big ? (uint32_t)NT : 64u);
            const uint32_t row = 32 * e + lane;
            for (uint32_t cb = 16 * eh; cb < n_mma; cb += 32) {
                uint32_t v0[16], v1[16];
                umma::tmem_ld16(t0 + cb, v0);
                umma::tmem_ld16(t1 + cb, v1);
                umma::tmem_ld_wait();
                if (MODE == wg::kGateUp) {
                    // silu with the fast exponential and division: their error (a few ulp) is far below the operands' f16 rounding
                    const uint32_t ff = it.rt * 128u + (row & ~3u) + ((row & 1u) << 1) + ((row >> 1) & 1u);   // element order 0, 2, 1, 3
                    __half* hp = a.h + (size_t)(it.pair_off + cb) * a.rows + ff;
                    auto put = [&](int i) {
                        const float us = f0[cb + i], gv = __uint_as_float(v0[i]) * us, uv = __uint_as_float(v1[i]) * us;
                        hp[(size_t)i * a.rows] = __float2half_rn(__fdividef(gv, 1.0f + __expf(-gv)) * uv * f1[cb + i]);
                    };
                    if (cb + 16 <= n) {   // without a branch per column the columns' chains overlap
#pragma unroll
                        for (int i = 0; i < 16; ++i) put(i);
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (cb + i < n) put(i);
                    }
                } else {
                    const uint32_t o0 = it.rt * 256u + row;
                    float* op = a.out + (size_t)(it.pair_off + cb) * a.rows + o0;
                    const bool second = o0 + 128 < a.rows;   // a dense matrix may end with a lone row tile
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (cb + i < n) {
                            op[(size_t)i * a.rows] = f0[cb + i] * __uint_as_float(v0[i]);
                            if (second) op[(size_t)i * a.rows + 128] = f0[cb + i] * __uint_as_float(v1[i]);
                        }
                }
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) { mbar_arrive(bar_accfree + 8 * b); if (big) mbar_arrive(bar_accfree + 8); }
        }
    } else {
    wg::set_regs<R::kOther>();
    if (warp == (uint32_t)wg::kMmaWarp) {
        // ---- MMA issue: the whole warp walks the loop, one elected lane issues
        const bool leader = umma::elect_one();
        uint32_t used[2] = {0, 0}, next = 0, before = 0;
        MmaItem it;
        for (uint32_t k = 0; next_unit(k, it); ++k, before += advance) {
            const uint32_t n_mma = (it.n + 15u) & ~15u;
            const bool big = n_mma > 64;
            const uint32_t b = big ? 0u : next, idesc = umma::instr_desc_f16(n_mma);
            // the accumulators' previous contents have been read
            if (used[b]) wait_bar(bar_accfree + 8 * b, (used[b] - 1) & 1u);
            if (big && used[1]) wait_bar(bar_accfree + 8, (used[1] - 1) & 1u);
            if (big) { ++used[0]; ++used[1]; next = 0; } else { ++used[b]; next ^= 1u; }
            umma::fence_after_sync();
            const uint32_t t0 = tmem + b * 128u, t1 = t0 + (big ? (uint32_t)NT : 64u);
            for (uint32_t i = 0; i < KS; ++i) {
                const uint32_t stage = stage_of(before, i);
                wait_bar(bar_full + 8 * stage, round_of(before, i) & 1u);
                umma::fence_after_sync();
                const uint64_t d_b = umma::smem_desc(wg::b_addr<FMT, NT>(stage));
                const uint32_t t_a = tmem + wg::tmem_a<NT>() + stage * 64u;
                if (leader) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {   // 16 columns of K further: 8 tensor-memory columns, 32 bytes of the row tile
                        const bool acc = (i | (uint32_t)j) != 0;
                        mma_f16_ts(t0, t_a + 8 * j, d_b + 2 * j, idesc, acc);
                        mma_f16_ts(t1, t_a + 32 + 8 * j, d_b + 2 * j, idesc, acc);
                    }
                    umma::commit(bar_empty + 8 * stage);
                    if (i + 1 == KS) { umma::commit(bar_accfull + 8 * b); if (big) umma::commit(bar_accfull + 8); }
                }
                __syncwarp();
            }
        }
    } else if (warp == (uint32_t)wg::kWeightWarp) {
        // ---- units and weights
        uint32_t blocks[2] = {0, 0}, slots[2] = {0, 0};   // handed out so far, per parity
        auto drained = [&](uint32_t par, uint32_t slot) {   // everything put there has been read
            const uint32_t uses = (slots[par] + kSlots - 1 - slot) / kSlots + (slot ? 0u : blocks[par]);
            if (uses) wait_bar(bar_wempty + 8 * (kSlots * par + slot), (uses - 1) & 1u);
        };
        uint32_t u = blockIdx.x;
        for (uint32_t k = 0;; ++k) {
            MmaItem it{0, 0, 0, 0};
            if (u < n_units) it = unit_item(u);
            const uint32_t s = k % wg::kFeed;
            if (k >= (uint32_t)wg::kFeed) wait_bar(bar_uempty + 8 * s, (k / wg::kFeed - 1) & 1u);
            if (__any_sync(0xFFFFFFFFu, waits.out)) break;   // the slot may still be read; the other roles' waits run out too
            if (lane == 0) {
                s_feed[s] = it;
                mbar_arrive(bar_ufull + 8 * s);
            }
            if (it.n == 0) break;
            uint32_t ticket = 0;
            if (lane == 0) ticket = a.ticket ? gridDim.x + atomicAdd(a.ticket, 1u) : u + gridDim.x;   // back by the time this unit's copies are issued
            const bool shared = MODE != wg::kDense && it.expert == kSharedItem, q8 = shared;
            const uint32_t tile = q8 ? (uint32_t)kTileQ8 : wg::tile_size<FMT>();
            auto tiles_of = [&](uint32_t m) -> const uint8_t* {   // first of the eight tiles of matrix (row tile) m, column block 0
                const uint32_t rt128 = MODE == wg::kGateUp ? it.rt : min(2u * it.rt + m, a.rows / 128 - 1);
                return (shared ? a.sh[m] : a.w[m]) + ((size_t)(shared ? 0u : it.expert) * KB * RT16 + rt128 * 8) * tile;
            };
            const uint8_t* src = q8 ? tiles_of((lane >> 3) & 1u) + (size_t)(lane & 7u) * kTileQ8 : tiles_of(lane & 1u);   // this lane's share
            for (uint32_t kp = 0; kp < KB; kp += 2) {
                const bool lone = MODE == wg::kDense && kp + 1 == KB;   // both groups get the block, of Q8_0 their quarters of it
                if (q8) {
                    for (uint32_t q = 0; q < 4; ++q)
                        for (uint32_t par = 0; par < 2; ++par) {
                            if (lone && ((q ^ par) & 1u)) continue;
                            const uint32_t slot = slots[par] % kSlots, wf = bar_wfull + 8 * (kSlots * par + slot);
                            drained(par, slot);
                            if (__any_sync(0xFFFFFFFFu, waits.out)) break;   // a barrier that still counts bytes takes no second arrival
                            ++slots[par];
                            if (lane == 0) mbar_expect_tx(wf, wg::kQ8Slot);
                            __syncwarp();
                            if (lane < 16) bulk_g2s(wg::w_base<FMT, NT>() + par * wg::w_bytes<FMT>() + slot * wg::kQ8Slot + lane * 1088u,
                                                    src + (size_t)(lone ? kp : kp + par) * RT16 * kTileQ8 + q * 1088u, 1088u, wf);
                        }
                } else {
                    for (uint32_t par = 0; par < 2; ++par) {
                        const uint32_t wf = bar_wfull + 8 * kSlots * par;
                        for (uint32_t slot = 0; slot < kSlots; ++slot) drained(par, slot);   // a block covers them all
                        if (__any_sync(0xFFFFFFFFu, waits.out)) break;
                        ++blocks[par];
                        if (lane == 0) mbar_expect_tx(wf, 16 * tile);
                        __syncwarp();
                        if (lane < 2) bulk_g2s(wg::w_base<FMT, NT>() + par * wg::w_bytes<FMT>() + lane * 8 * tile, src + (size_t)(lone ? kp : kp + par) * RT16 * tile, 8 * tile, wf);
                    }
                }
            }
            u = __shfl_sync(0xFFFFFFFFu, ticket, 0);
        }
    } else if (MODE == wg::kGateUp && warp < wg::kRowWarp + wg::row_warps<MODE>()) {
        // ---- scattered activation rows: six warps; two, which take every other 16 rows, copy a step (four rows x 64 columns per
        // instruction), wait for its arrival and announce it, and three pairs take the steps in turn.  A copy issues every 55 cycles or
        // so, and from about 100 rows on that is what a stage waits for: gate/up at 4096 tokens, tiles of 160, 236 us with one warp
        // a step, 227 with more registers for the addresses (56 a thread), 213 with two; 3200 tokens, tiles of 128, 189 -> 181.
        // (Two warps that shared every step and announced it two steps later, so as not to wait, kept two stages in flight: the
        // producers waited 40 to 60 % of their time for a free stage.)
        // Past the unit's end: the last row again (nobody reads those columns)
        const uint32_t wi = warp - wg::kRowWarp, w = wi % 3u, part = wi / 3u, rr = lane >> 3, c = lane & 7u;   // groups of 16 rows: part, part + kPer, ...
        const uint32_t d0 = part * 2048u + rr * 128u + ((c ^ rr) << 4), d1 = part * 2048u + (rr + 4) * 128u + ((c ^ (rr + 4)) << 4);
        const uint32_t rows = smem_addr(&s_rows[wi][rr * (NT / 4 / kPer)]);
        uint32_t before = 0, first = w;   // first: this warp's first step of the unit
        MmaItem it;
        for (uint32_t k = 0; next_unit(k, it); ++k, before += advance) {
            const uint32_t groups = ((it.n + 15u) & ~15u) / 4;   // of four rows, a multiple of four
            for (uint32_t r = lane; r < 4 * groups; r += 32)
                if (kPer == 1 || (r >> 4) % kPer == part)
                    s_rows[wi][(r & 3u) * (NT / 4 / kPer) + (r >> 4) / kPer * 4 + ((r >> 2) & 3u)] = (a.pairs[it.pair_off + min(r, it.n - 1)] >> 4) * (a.K / 8);   // in 16-byte pieces
            __syncwarp();
            uint32_t i = first;
            for (; i < KS; i += 3) {
                const uint32_t stage = stage_of(before, i), round = round_of(before, i), dst = wg::b_addr<FMT, NT>(stage);
                if (round) wait_bar(bar_empty + 8 * stage, (round - 1) & 1u);
                const uint4* src = reinterpret_cast<const uint4*>(a.xrows) + step_kb(i) * 32u + step_q(i) * 8u + c;
#pragma unroll
                for (int b = 0; b < NT / 16 / (int)kPer; ++b)
                    if (4u * (kPer * b + part) < groups) {
                        const uint4 o4 = lds128(rows + 16 * b);
                        const uint32_t o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + ((j & 1) ? d1 : d0) + (2 * kPer * b + (j >> 1)) * 1024u), "l"(src + o[j]) : "memory");
                    }
                asm volatile("cp.async.wait_all;" ::: "memory");
                umma::fence_smem_to_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_full + 8 * stage);
            }
            first = i - KS;
            __syncwarp();   // every lane is done with this unit's offsets
        }
    } else if (MODE != wg::kGateUp && warp == (uint32_t)wg::kRowWarp) {
        // ---- consecutive activation rows: boxes of 16
        if (MODE == wg::kDense) pdl_wait();
        uint32_t gs = 0;
        MmaItem it;
        for (uint32_t k = 0; next_unit(k, it); ++k) {
            const uint32_t boxes = (it.n + 15u) / 16;
            for (uint32_t i = 0; i < KS; ++i, ++gs) {
                const uint32_t stage = gs % kSt;
                if (gs >= kSt) wait_bar(bar_empty + 8 * stage, (gs / kSt - 1) & 1u);
                if (__any_sync(0xFFFFFFFFu, waits.out)) break;   // a barrier that still counts bytes takes no second arrival
                if (lane == 0) mbar_expect_tx(bar_full + 8 * stage, boxes * 2048u);
                __syncwarp();
                if (lane < boxes) tma_rows16(wg::b_addr<FMT, NT>(stage) + lane * 2048u, &rows_map, step_kb(i) * 256u + step_q(i) * 64u, it.pair_off + 16 * lane, bar_full + 8 * stage);
            }
        }
    }
    }
    umma::fence_before_sync();
    const int any_timed_out = __syncthreads_or(waits.out ? 1 : 0);   // any role's wait that ran out counts
    if (any_timed_out) for (int i = 0; i < 100; ++i) __nanosleep(1000);   // copies and MMAs still under way end long before this does
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
    if (any_timed_out && tid == 0) atomicExch(a.status, (uint32_t)kStatusWaitTimeout);
}

// ---- activation rows ---------------------------------------------------------------------------------------
// x -> f16 rows in the kernels' element order, each scaled by a power of two so that the largest finite |x| lands in
// [2^13, 2^14) (infinities and NaN stay what they are), the inverse scale and (optional) the row's 2-norm.  WARPS warps per row, which hold it in registers (up to four float4 a thread; a longer
// row is read twice): one trip to memory.  (A warp per row that read it twice: 1000 x 2048 8.0 us, 4096 rows 11.5.)
template <int WARPS>
__global__ void __launch_bounds__(256)
f16_rows_kernel(const float* x, __half* __restrict__ xh, float* __restrict__ inv_scale, float* __restrict__ norm, uint32_t n_rows, uint32_t K, uint32_t* __restrict__ zero,
                uint32_t n_zero) {
    __shared__ float s_m[8], s_ss[8];
    constexpr uint32_t kT = WARPS * 32;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, sub = threadIdx.x / kT, lt = threadIdx.x % kT, t = blockIdx.x * (256 / kT) + sub;
    pdl_trigger();
    pdl_wait();
    if (blockIdx.x == 0)
        for (uint32_t i = threadIdx.x; i < n_zero; i += 256) zero[i] = 0;
    const bool live = t < n_rows;
    const float4* xt = reinterpret_cast<const float4*>(x + (size_t)(live ? t : 0) * K);
    const uint32_t K4 = K / 4;
    float m = 0.f, ss = 0.f;
    auto finite_abs = [](float v) { const float a = fabsf(v); return a <= 3.402823466e38f ? a : 0.f; };
    auto take = [&](const float4& v) {
        m = fmaxf(fmaxf(m, fmaxf(finite_abs(v.x), finite_abs(v.y))), fmaxf(finite_abs(v.z), finite_abs(v.w)));
        ss += v.x * v.x; ss += v.y * v.y; ss += v.z * v.z; ss += v.w * v.w;
    };
    float4 r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = live && lt + i * kT < K4 ? xt[lt + i * kT] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) take(r[i]);
    if (live)
        for (uint32_t k = lt + 4 * kT; k < K4; k += kT) take(xt[k]);
    m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));   // non-negative floats order like their bits
    ss = warp_sum(ss);
    if (WARPS > 1) {
        if (lane == 0) { s_m[warp] = m; s_ss[warp] = ss; }
        __syncthreads();
        m = ss = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) { m = fmaxf(m, s_m[sub * WARPS + w]); ss += s_ss[sub * WARPS + w]; }
    }
    if (!live) return;
    int p = 0;
    if (m > 0.f) { int e; frexpf(m, &e); p = min(14 - e, 126); }   // m * 2^p in [2^13, 2^14)
    const float up = ldexpf(1.0f, p);
    uint2* dst = reinterpret_cast<uint2*>(xh + (size_t)t * K);
    auto put = [&](uint32_t k, const float4& v) {
        const __half2 a = __floats2half2_rn(v.x * up, v.z * up), b = __floats2half2_rn(v.y * up, v.w * up);
        dst[k] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    };
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (lt + i * kT < K4) put(lt + i * kT, r[i]);
    for (uint32_t k = lt + 4 * kT; k < K4; k += kT) put(k, xt[k]);
    if (lt == 0) {
        inv_scale[t] = ldexpf(1.0f, -p);
        if (norm) norm[t] = sqrtf(ss);
    }
}
cudaError_t launch_f16_rows(const Launch& L, const float* x, void* xh, float* inv_scale, float* norm, uint32_t n_rows, uint32_t K, uint32_t* zero, uint32_t n_zero) {
    if (n_rows == 0) return cudaSuccess;
    if (K % 4) return cudaErrorInvalidValue;
    const Launch P{L.stream, nullptr, true};
    cudaError_t e;
    // as many warps a row as hold 512 columns each
    if (K <= 512) e = launch_kernel(P, f16_rows_kernel<1>, dim3((n_rows + 7) / 8), dim3(256), 0, x, (__half*)xh, inv_scale, norm, n_rows, K, zero, n_zero);
    else if (K <= 2048) e = launch_kernel(P, f16_rows_kernel<4>, dim3((n_rows + 1) / 2), dim3(256), 0, x, (__half*)xh, inv_scale, norm, n_rows, K, zero, n_zero);
    else e = launch_kernel(P, f16_rows_kernel<8>, dim3(n_rows), dim3(256), 0, x, (__half*)xh, inv_scale, norm, n_rows, K, zero, n_zero);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}
// rows that arrived as scaled f16 (expert parallel): their 2-norms, and a copy in the kernels' element order
__global__ void __launch_bounds__(256)
f16_rows_in_kernel(const __half* __restrict__ in, const float* __restrict__ inv_scale, __half* __restrict__ out, float* __restrict__ norm, uint32_t n_rows, uint32_t K) {
    const uint32_t t = (blockIdx.x * 256u + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (t >= n_rows) return;
    const uint4* xt = reinterpret_cast<const uint4*>(in + (size_t)t * K);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)t * K);
    float ss = 0.f;
    for (uint32_t k = lane; k < K / 8; k += 32) {
        const uint4 v = xt[k];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            ss += f.x * f.x; ss += f.y * f.y;
        }
        dst[k] = make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x5410), __byte_perm(v.z, v.w, 0x7632));
    }
    ss = warp_sum(ss);
    if (lane == 0) norm[t] = sqrtf(ss) * inv_scale[t];
}
cudaError_t launch_f16_rows_in(const Launch& L, const void* in, const float* inv_scale, void* out, float* norm, uint32_t n_rows, uint32_t K) {
    if (n_rows == 0) return cudaSuccess;
    f16_rows_in_kernel<<<(n_rows + 7) / 8, 256, 0, L.stream>>>((const __half*)in, inv_scale, (__half*)out, norm, n_rows, K);
    L.count();
    return cudaGetLastError();
}
// out[e] = largest row 2-norm of expert e's matrix [rows][K] (raw ggml rows; at upload), rounded up a little.
// out has to be zero before (the maximum is taken on the bits of non-negative floats).
// A warp per row, a 32-column sub-block per lane; squares of codebook entries from a table in shared memory.
template <int TYPE>
__global__ void __launch_bounds__(256)
row_norm_max_kernel(const uint8_t* __restrict__ w, float* __restrict__ out, uint32_t rows, uint32_t K) {
    __shared__ float s_sq[256];   // IQ3_XXS: a grid entry's four magnitudes squared and summed; IQ4_XS: a byte's two values
    const uint32_t tid = threadIdx.x, lane = tid & 31u, e = blockIdx.y;
    if (TYPE == QKM_TYPE_IQ3_XXS) {
        const uint32_t g = c_iq3_grid[tid];
        s_sq[tid] = (float)__dp4a(g, g, 0u);
    } else if (TYPE == QKM_TYPE_IQ4_XS) {
        const float a = (float)c_iq4_values[tid & 15u], b = (float)c_iq4_values[tid >> 4];
        s_sq[tid] = a * a + b * b;
    }
    __syncthreads();
    const size_t rb = row_bytes(TYPE, K);
    float best = 0.f;
    for (uint32_t r = blockIdx.x * 8 + (tid >> 5); r < rows; r += gridDim.x * 8) {
        const uint8_t* row = w + ((size_t)e * rows + r) * rb;
        float ss = 0.f;
        for (uint32_t sb = lane; sb < K / 32; sb += 32) {
            const uint8_t* b = row + (size_t)(sb >> 3) * Fmt<TYPE>::kBytes;
            const uint32_t ib = sb & 7u;
            float sum = 0.f, sc;
            if (TYPE == QKM_TYPE_IQ3_XXS) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t q = ld_u16(b + 2 + 8 * ib + 2 * i);
                    sum += s_sq[q & 255u] + s_sq[q >> 8];
                }
                sc = f16_bits_to_f32(ld_u16(b)) * (0.5f + (float)(ld_u32_a2(b + 66 + 4 * ib) >> 28)) * 0.5f;
            } else if (TYPE == QKM_TYPE_IQ4_XS) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t q = *reinterpret_cast<const uint32_t*>(b + 8 + 16 * ib + 4 * i);
                    sum += (s_sq[q & 255u] + s_sq[(q >> 8) & 255u]) + (s_sq[(q >> 16) & 255u] + s_sq[q >> 24]);
                }
                const uint32_t ls = (((uint32_t)b[4 + (ib >> 1)] >> (4 * (ib & 1u))) & 15u) | (((ld_u16(b + 2) >> (2 * ib)) & 3u) << 4);
                sc = f16_bits_to_f32(ld_u16(b)) * (float)((int)ls - 32);
            } else {   // Q8_0: a block of 34 bytes per sub-block
                const uint8_t* q8 = row + (size_t)sb * 34;
                int s = 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int q = (int)ld_u32_a2(q8 + 2 + 4 * i);
                    s = __dp4a(q, q, s);
                }
                sum = (float)s;
                sc = f16_bits_to_f32(ld_u16(q8));
            }
            ss += sum * sc * sc;
        }
        best = fmaxf(best, warp_sum(ss));
    }
    if (lane == 0 && best > 0.f) atomicMax(reinterpret_cast<uint32_t*>(out + e), __float_as_uint(sqrtf(best) * 1.001f));
}
cudaError_t launch_row_norm_max(const Launch& L, uint32_t type, const void* w, float* out, uint32_t n_mats, uint32_t rows, uint32_t K) {
    const dim3 grid((rows + 63) / 64, n_mats);   // eight rows a warp
    const uint8_t* p = (const uint8_t*)w;
    switch (type) {
        case QKM_TYPE_IQ3_XXS: row_norm_max_kernel<QKM_TYPE_IQ3_XXS><<<grid, 256, 0, L.stream>>>(p, out, rows, K); break;
        case QKM_TYPE_IQ4_XS: row_norm_max_kernel<QKM_TYPE_IQ4_XS><<<grid, 256, 0, L.stream>>>(p, out, rows, K); break;
        case QKM_TYPE_Q8_0: row_norm_max_kernel<QKM_TYPE_Q8_0><<<grid, 256, 0, L.stream>>>(p, out, rows, K); break;
        default: return cudaErrorInvalidValue;
    }
    L.count();
    return cudaGetLastError();
}

// ---- launchers ---------------------------------------------------------------------------------------------
// tensor map over f16 rows [n_rows][K]: boxes of 16 rows x 64 columns, 128-byte swizzle
static bool rows_tensor_map(CUtensorMap* map, const void* rows, uint64_t n_rows, uint32_t K) {
    typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const EncodeFn encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess ? (EncodeFn)fn : (EncodeFn) nullptr;
    }();
    if (!encode) return false;
    const cuuint64_t dim[2] = {K, n_rows}, stride[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {64, 16}, estride[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(rows), dim, stride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int FMT, int MODE, int NT = wg::kNT>
static cudaError_t wgemm_launch(const Launch& L, const WgemmArgs& a, const void* rows, uint64_t n_rows, uint32_t max_units, uint32_t n_sms) {
    if (max_units == 0) return cudaSuccess;
    if (MODE != wg::kDense && a.K % 512) return cudaErrorInvalidValue;   // a lone last column block is compiled for dense matrices only
    if (const cudaError_t e = allow_dynamic_smem<wgemm_kernel<FMT, MODE, NT>>((int)wg::smem_end<FMT, NT>())) return e;
    CUtensorMap map{};
    if (((uintptr_t)rows & 15u) || (MODE != wg::kGateUp && !rows_tensor_map(&map, rows, n_rows, a.K))) return cudaErrorInvalidValue;
    const cudaError_t e = launch_kernel(Launch{L.stream, nullptr, true}, wgemm_kernel<FMT, MODE, NT>, dim3(max_units < n_sms ? max_units : n_sms), dim3(wg::kThreads),
                                        wg::smem_end<FMT, NT>(), a, map);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_wgemm_gateup(const Launch& L, const qkm_dims& d, uint32_t type, const WgemmExperts& x, const void* xrows,
                                const float* x_inv_scale, const float* x_norm, const float* w_norm, void* h, float* h_inv_scale, uint32_t max_units) {
    WgemmArgs a{};
    a.w[0] = (const uint8_t*)x.w[0]; a.w[1] = (const uint8_t*)x.w[1]; a.sh[0] = (const uint8_t*)x.sh[0]; a.sh[1] = (const uint8_t*)x.sh[1];
    a.items = x.items; a.n_items = x.n_items; a.ticket = x.ticket; a.pairs = x.pairs; a.x_inv_scale = x_inv_scale; a.x_norm = x_norm; a.w_norm = w_norm;
    a.xrows = (const __half*)xrows; a.h = (__half*)h; a.h_inv_scale = h_inv_scale; a.table = x.table; a.status = x.status; a.rows = d.n_ff; a.K = d.n_embd;
    a.n_experts = x.n_experts; a.n_used = d.n_used;
    if (type == QKM_TYPE_IQ3_XXS)
        return x.tile > wg::kNT ? wgemm_launch<QKM_TYPE_IQ3_XXS, wg::kGateUp, wg::kWideNT>(L, a, xrows, 0, max_units, x.n_sms) : wgemm_launch<QKM_TYPE_IQ3_XXS, wg::kGateUp>(L, a, xrows, 0, max_units, x.n_sms);
    if (type == QKM_TYPE_IQ4_XS)
        return x.tile > wg::kNT ? wgemm_launch<QKM_TYPE_IQ4_XS, wg::kGateUp, wg::kWideNT>(L, a, xrows, 0, max_units, x.n_sms) : wgemm_launch<QKM_TYPE_IQ4_XS, wg::kGateUp>(L, a, xrows, 0, max_units, x.n_sms);
    return cudaErrorInvalidValue;
}

cudaError_t launch_wgemm_down(const Launch& L, const qkm_dims& d, uint32_t type, const WgemmExperts& x, const void* h, uint64_t n_hrows,
                              const float* h_inv_scale, const qkm_sel* sel, float* contrib, uint32_t max_units) {
    if (d.n_embd % 256) return cudaErrorInvalidValue;
    WgemmArgs a{};
    a.w[0] = a.w[1] = (const uint8_t*)x.w[0]; a.sh[0] = a.sh[1] = (const uint8_t*)x.sh[0];
    a.items = x.items; a.n_items = x.n_items; a.ticket = x.ticket; a.pairs = x.pairs; a.h_inv_scale = const_cast<float*>(h_inv_scale); a.sel = sel; a.out = contrib;
    a.table = x.table; a.status = x.status; a.rows = d.n_embd; a.K = d.n_ff; a.n_experts = x.n_experts; a.n_used = d.n_used;
    if (type == QKM_TYPE_IQ4_XS)
        return x.tile > wg::kNT ? wgemm_launch<QKM_TYPE_IQ4_XS, wg::kDown, wg::kWideNT>(L, a, h, n_hrows, max_units, x.n_sms) : wgemm_launch<QKM_TYPE_IQ4_XS, wg::kDown>(L, a, h, n_hrows, max_units, x.n_sms);
    if (type == QKM_TYPE_Q6_K)
        return x.tile > wg::kNT ? wgemm_launch<QKM_TYPE_Q6_K, wg::kDown, wg::kWideNT>(L, a, h, n_hrows, max_units, x.n_sms) : wgemm_launch<QKM_TYPE_Q6_K, wg::kDown>(L, a, h, n_hrows, max_units, x.n_sms);
    return cudaErrorInvalidValue;
}

// A weight is at most 128 |d| (Q8_0) or 32 * 127 |d| (IQ4_XS); where that would pass f16's 65504 the matrix's weights are scaled
// to at most 2^15.  Downwards nothing is needed: d is a multiple of 2^-24, the sub-block scales and codebook values are integers,
// so a scale or weight below f16's normal range (2^-14) is a multiple of 2^-24 too and exact as a subnormal.
float dense_weight_scale(uint32_t type, uint32_t d_bits) {
    const int e = (int)(d_bits >> 10);
    const float d = e ? ldexpf(1024.f + (float)(d_bits & 1023u), e - 25) : ldexpf((float)d_bits, -24);
    const float most = d * (type == QKM_TYPE_Q8_0 ? 128.f : 32.f * 127.f);
    if (most < 65504.f) return 1.f;
    int b;
    frexpf(most, &b);   // most < 2^b
    return ldexpf(1.f, 15 - b);
}

// Y[n][M] = X[n][K] . W^T: x rows to scaled f16, then one launch
cudaError_t launch_dense_gemm(const Launch& L, uint32_t type, const void* tiles, float w_scale, uint32_t M, uint32_t K, const float* x, uint32_t n_rows, float* y,
                              void* xh, float* x_inv_scale, const uint8_t* table, uint32_t n_sms, uint32_t* status) {
    if (n_rows == 0) return cudaSuccess;
    if (M % 128 || K % 256 || M / 128 > 65535) return cudaErrorInvalidValue;
    if (const cudaError_t e = launch_f16_rows(L, x, xh, x_inv_scale, nullptr, n_rows, K)) return e;
    WgemmArgs a{};
    a.w[0] = a.w[1] = (const uint8_t*)tiles;
    a.x_inv_scale = x_inv_scale; a.out = y; a.table = table; a.status = status; a.rows = M; a.K = K; a.n_dense = n_rows;
    a.w_scale = w_scale; a.w_inv_scale = 1.f / w_scale;
    const uint32_t units = (n_rows + wg::kNT - 1) / wg::kNT * ((M / 128 + 1) / 2);
    if (type == QKM_TYPE_Q8_0) return wgemm_launch<QKM_TYPE_Q8_0, wg::kDense>(L, a, xh, n_rows, units, n_sms);
    if (type == QKM_TYPE_IQ4_XS) return wgemm_launch<QKM_TYPE_IQ4_XS, wg::kDense>(L, a, xh, n_rows, units, n_sms);
    return cudaErrorInvalidValue;
}

}  // namespace qkm
