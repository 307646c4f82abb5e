// Gate/up + SwiGLU of the fused decode sequence: routed experts (IQ3_XXS) and the shared
// expert (Q8_0) in one persistent launch.
//
// Replaces moe_gateup_iq3.comp / moe_gateup_iq3_rowtile.comp and moe_gateup_q8.comp /
// moe_gateup_q8_64.comp for decode-sized batches; every selected expert is streamed once for
// up to two of the tokens that chose it (the reference's "live expert union" of multi-slot
// decode), and the shared expert rides in the same work list as groups of its own.
//
// Several layers whose rows are at hand together go through one launch: the list of work runs over all of them, so start-up, first
// tiles and the uneven end are paid once (12 to 13 us of each kernel did not depend on the work: one layer of 16 tokens 38 us, 40 layers
// together 26 us each).  A layer on its own takes a form without the other layers' bookkeeping.
//
// Work: the flat list of (layer, group, 16-row tile) - a group is an expert with up to two
// tokens, n_ff / 16 tiles each - is cut evenly and contiguously over teams of KB = n_embd / 256
// warps; warp kb of a team streams column block kb of every tile of the team's range through
// a private two-stage ring of bulk copies (TMA, no tensor map, no multicast).
//
// IQ3_XXS inner step (one 32-column sub-block of 16 rows = one int8 MMA of weights):
//   * the lane's two grid indices are already bytes of one register; a byte-permute drops
//     each into bits 8..15 of a table address whose other bytes are lane constants (the grid
//     table has a 256-byte stride per entry and sits at a 64 KB boundary), so a lookup
//     address costs one instruction;
//   * the tiles hold signs as bits at places where a shift brings four of them to the top of their
//     bytes, and a byte permute in sign mode turns those into 0xFF / 0x00 masks;
//   * magnitudes ^ mask is -m-1 where the element is negative; a second MMA of the masks
//     (-1 / 0) with the negated digit planes adds the missing +1 * x, so no per-element
//     sign arithmetic remains;
//   * the 4-bit sub-block scale stays an integer (2s + 1) and multiplies the exact int32
//     partial sums; d * 0.25 and the digit weights are applied once per tile in f32.
// Q8_0 tiles are cut into quarters (two 32-column blocks) so that a stage of the same ring
// holds them.
//
// IQ4_XS gate/up tensors (moe_gateup_iq4.comp) take the same kernel, instantiated with the inner
// step of the decode down kernel: the 16-entry codebook in four registers, looked up with byte
// permutes, the 6-bit sub-block scales as integers.  No table image: the rings (4352 bytes per
// stage) lie in one run at the start of shared memory.
#include "qkm_dec_rank.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"
#include "qkm_tiles.cuh"

namespace qkm {

namespace dg {
constexpr int kWarps = 16;
constexpr int kStages = 2;
constexpr int kStageBytes = 2 * kTileIq3;          // gate tile + up tile (3392); a Q8_0 quarter pair needs 2176
constexpr int kRingBytes = kStages * kStageBytes;
constexpr int kStageBytes4 = 2 * kTileIq4;         // the IQ4_XS form: 4352
constexpr int kRingBytes4 = kStages * kStageBytes4;
constexpr uint32_t kTab = 65536, kTabBytes = 65536;   // absolute shared-window address (64 KB aligned) and size
constexpr int kLowRingWarps = 9;                    // rings below the table; the others above it
constexpr int kGroupTiles = 4;                      // tiles between two team-wide reductions
constexpr int kRedFloats = kGroupTiles * 16 * 2 * 2;   // per warp and buffer: tile, row, token, matrix
constexpr uint32_t kHigh = kTab + kTabBytes;
constexpr uint32_t kRed = kHigh + (kWarps - kLowRingWarps) * kRingBytes;
constexpr uint32_t kRedBytes = kWarps * 2 * kRedFloats * 4, kListBytes = rk::kMaxGroups * sizeof(DecodeGroup);   // the list: of a layer's groups, or of those in the teams' shares
constexpr uint32_t kList = kRed + kRedBytes;
static_assert(sizeof(OwnScratch) <= kRedBytes, "the grouping's working set lies where the partial sums come later");
// IQ4_XS form, offsets from the (128-byte aligned) start of the dynamic area: barriers, rings, scratch
constexpr uint32_t kRings4 = 1024;
constexpr uint32_t kRed4 = kRings4 + kWarps * kRingBytes4;
constexpr uint32_t kList4 = kRed4 + kRedBytes;
constexpr int kQ8Quarter = 2 * 544;                 // two 32-column blocks of a Q8_0 tile: d and quants of 16 rows each
// Relative time of a routed / a shared tile.  11 instead of 10 changes layers that go together by -2.5 to +1.1 % (mostly less than two runs
// differ) and a layer on its own by -1.3 to +0.4 %, but one token's from 23.5 to 25.2 us.
constexpr uint32_t kCostRouted = 8, kCostShared = 10;
}  // namespace dg

size_t decode_gateup_lut_bytes() { return dg::kTabBytes; }

// The table image: row i (256 B) = grid entry i for 32 lanes (4 B each); the upper 128 B are not read.
__global__ void decode_gateup_lut_kernel(uint8_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;   // one 4-byte word each
    if (i >= dg::kTabBytes / 4) return;
    reinterpret_cast<uint32_t*>(out)[i] = (i & 63u) < 32 ? c_iq3_grid[i >> 6] : 0u;
}

cudaError_t launch_decode_gateup_luts(const Launch& L, uint8_t* luts) {
    decode_gateup_lut_kernel<<<dg::kTabBytes / 4 / 256, 256, 0, L.stream>>>(luts);
    L.count();
    return cudaGetLastError();
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// One IQ3_XXS tile (16 rows x 256 columns) of one matrix against the warp's B operand.
// acc[0..1]: row g, columns 2t and 2t+1; acc[2..3]: row g+8.  Integer, exact.
__device__ __forceinline__ void iq3_tile(uint32_t tb, uint32_t i_off, uint32_t s_off, uint32_t g, uint32_t grid_c,
                                         const uint32_t (&b0)[8], const uint32_t (&b1)[8],
                                         const uint32_t (&n0)[8], const uint32_t (&n1)[8], int (&acc)[4]) {
    const uint4 ia = lds128(tb + i_off), ib = lds128(tb + i_off + 512);                          // rows g and g+8: 2 index bytes per sub-block
    const uint2 sa = lds64(tb + 1024 + s_off), sb2 = lds64(tb + 1280 + s_off);                    // signs
    const uint2 ca = lds64(tb + 1536 + 8 * g), cb = lds64(tb + 1600 + 8 * g);                     // scales 2 s + 1
    const uint32_t idx_a[4] = {ia.x, ia.y, ia.z, ia.w}, idx_b[4] = {ib.x, ib.y, ib.z, ib.w};
    acc[0] = acc[1] = acc[2] = acc[3] = 0;
#pragma unroll
    for (int sb = 0; sb < 8; ++sb) {
        const uint32_t wa = idx_a[sb >> 1], wb = idx_b[sb >> 1];
        const uint32_t s_lo = (sb & 1) ? 0x7624u : 0x7604u, s_hi = (sb & 1) ? 0x7634u : 0x7614u;
        const uint32_t ga0 = lds32(prmt(wa, grid_c, s_lo)), ga1 = lds32(prmt(wa, grid_c, s_hi));
        const uint32_t gb0 = lds32(prmt(wb, grid_c, s_lo)), gb1 = lds32(prmt(wb, grid_c, s_hi));
        // 0xFF bytes where negative: the top bits of the shifted sign word's bytes, replicated (the shift is a multiply's pipe, not the ALU's)
        const uint32_t va = (sb < 4 ? sa.x : sa.y), vb = (sb < 4 ? sb2.x : sb2.y);
        const uint32_t ma0 = prmt(va * (1u << (2 * (sb & 3))), 0u, 0xBA98u), ma1 = prmt(va * (2u << (2 * (sb & 3))), 0u, 0xBA98u);
        const uint32_t mb0 = prmt(vb * (1u << (2 * (sb & 3))), 0u, 0xBA98u), mb1 = prmt(vb * (2u << (2 * (sb & 3))), 0u, 0xBA98u);
        int c[4];
        mma_s8_first(c, ga0 ^ ma0, gb0 ^ mb0, ga1 ^ ma1, gb1 ^ mb1, b0[sb], b1[sb]);
        mma_s8(c, ma0, mb0, ma1, mb1, n0[sb], n1[sb]);
        const uint32_t sel = 0x4440u + (uint32_t)(sb & 3);
        const int qa = (int)prmt(sb < 4 ? ca.x : ca.y, 0u, sel), qb = (int)prmt(sb < 4 ? cb.x : cb.y, 0u, sel);
        acc[0] += qa * c[0]; acc[1] += qa * c[1];
        acc[2] += qb * c[2]; acc[3] += qb * c[3];
    }
}

// Eight IQ4_XS weights of one quant word (elements e0 .. e7 = 8t .. 8t+7 of a sub-block, see qkm_tiles.cuh) as
// two int8 A-operand registers: lo = (e0, e2, e1, e3), hi = (e4, e6, e5, e7).
__device__ __forceinline__ void iq4_word_gu(uint32_t w, uint32_t& lo, uint32_t& hi) {
    const uint32_t T0 = 0xBFAD9881u, T1 = 0xF6EADDCFu, T2 = 0x26190D01u, T3 = 0x71594535u;   // kvalues_iq4nl as int8
    const uint32_t s = w & 0x77777777u, s2 = s >> 16, w4 = w << 4;
    const uint32_t m_lo = prmt(w4, w, 0xD9C8u), m_hi = prmt(w4, w, 0xFBEAu);   // 0xFF where a nibble's top bit is set
    const uint32_t a_lo = prmt(T0, T1, s), b_lo = prmt(T2, T3, s);
    const uint32_t a_hi = prmt(T0, T1, s2), b_hi = prmt(T2, T3, s2);
    lo = (a_lo & ~m_lo) | (b_lo & m_lo);
    hi = (a_hi & ~m_hi) | (b_hi & m_hi);
}
// the eight sub-block scales ls - 32 of one row as int8: sub-blocks 0,2,4,6 in ev, 1,3,5,7 in od
__device__ __forceinline__ void iq4_scales_gu(uint32_t sl, uint32_t sh, uint32_t& ev, uint32_t& od) {
    const uint32_t r = prmt(sh, 0u, 0x1100u);
    const uint32_t he = ((r << 4) & 0x00300030u) | (r & 0x30003000u);
    const uint32_t ho = ((r << 2) & 0x00300030u) | ((r >> 2) & 0x30003000u);
    const uint32_t te = ((sl & 0x0F0F0F0Fu) | he) ^ 0x20202020u;
    const uint32_t to = (((sl >> 4) & 0x0F0F0F0Fu) | ho) ^ 0x20202020u;
    ev = (te & 0x20202020u) * 6u + te;
    od = (to & 0x20202020u) * 6u + to;
}
// One IQ4_XS tile against the warp's B operand (elements in iq4_word_gu's order).  acc as in iq3_tile;
// hd: the headers of rows g (x: d | scales_h << 16, y: scales_l) and g+8 (z, w).
__device__ __forceinline__ void iq4_tile_gu(uint32_t tb, uint32_t i_off, uint32_t g, const uint32_t (&b0)[8],
                                            const uint32_t (&b1)[8], int (&acc)[4], uint4& hd) {
    hd = lds128(tb + 16 * g);
    uint32_t ea, oa, eb, ob;
    iq4_scales_gu(hd.y, hd.x >> 16, ea, oa);
    iq4_scales_gu(hd.w, hd.z >> 16, eb, ob);
    acc[0] = acc[1] = acc[2] = acc[3] = 0;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
        const uint4 qa4 = lds128(tb + 128 + hf * 1024 + i_off), qb4 = lds128(tb + 640 + hf * 1024 + i_off);
        const uint32_t wa[4] = {qa4.x, qa4.y, qa4.z, qa4.w}, wb[4] = {qb4.x, qb4.y, qb4.z, qb4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int sb = 4 * hf + j;
            uint32_t a0, a1, a2, a3;
            iq4_word_gu(wa[j], a0, a2);
            iq4_word_gu(wb[j], a1, a3);
            int c[4];
            mma_s8_first(c, a0, a1, a2, a3, b0[sb], b1[sb]);
            const uint32_t sel = 0x8880u + (uint32_t)(sb >> 1) * 0x1111u;   // byte sb / 2, sign-extended
            const int la = (int)prmt((sb & 1) ? oa : ea, 0u, sel), lb = (int)prmt((sb & 1) ? ob : eb, 0u, sel);
            acc[0] += la * c[0]; acc[1] += la * c[1]; acc[2] += lb * c[2]; acc[3] += lb * c[3];
        }
    }
}

// Two Q8_0 blocks (a quarter tile) of one matrix: q points at two 544-byte pieces [d 32 B][quants 512 B].
__device__ __forceinline__ void q8_quarter(uint32_t q, uint32_t lane, uint32_t g, uint32_t b0a, uint32_t b1a, uint32_t b0b,
                                           uint32_t b1b, float wcol0, float wcol1, float& fa, float& fb) {
#pragma unroll
    for (int bb = 0; bb < 2; ++bb) {
        const uint32_t pb = q + 544 * bb;
        const uint2 qa = lds64(pb + 32 + lane * 8);
        const uint2 qb = lds64(pb + 32 + 256 + lane * 8);
        int c[4];
        mma_s8_first(c, qa.x, qb.x, qa.y, qb.y, bb ? b0b : b0a, bb ? b1b : b1a);
        const uint32_t dw = lds32(pb + 2 * (g & ~1u));
        const uint32_t dw8 = lds32(pb + 2 * (8 + (g & ~1u)));
        const float da = f16_bits_to_f32((dw >> (16 * (g & 1u))) & 0xFFFFu);
        const float db = f16_bits_to_f32((dw8 >> (16 * (g & 1u))) & 0xFFFFu);
        fa += da * ((float)c[0] * wcol0 + (float)c[1] * wcol1);
        fb += db * ((float)c[2] * wcol0 + (float)c[3] * wcol1);
    }
}

// ONE: one layer, whose pairs the block groups itself (from a.sel; NULL: the shared expert's groups only); else the router kernel's lists
template <bool IQ4, bool ONE>
__global__ void __launch_bounds__(dg::kWarps * 32, 1)
decode_gateup_kernel(const __grid_constant__ GateupDecodeArgs a) {
    constexpr int kTileR = IQ4 ? kTileIq4 : kTileIq3;                       // routed tile bytes
    constexpr int kStageB = IQ4 ? dg::kStageBytes4 : dg::kStageBytes, kRingB = IQ4 ? dg::kRingBytes4 : dg::kRingBytes;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ LayerCuts s_cuts;
    const uint32_t base = smem_addr(smem_raw);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    const qkm_dims d = a.d;
    const uint32_t KB = d.n_embd / 256;           // warps per team (2, 4 or 8)
    const uint32_t n_teams = dg::kWarps / KB;
    const uint32_t team = warp / KB, kb = warp - team * KB;
    const uint32_t RT = d.n_ff / 16;              // tiles per group
    const uint32_t team_threads = KB * 32, lt = tid - team * team_threads;

    const uint32_t base4 = (base + 127u) & ~127u;                        // IQ4_XS form: everything relative to here
    const uint32_t bar_base = IQ4 ? base4 : (base + 15u) & ~15u;         // kWarps * kStages ring barriers, then the table's
    const uint32_t tab_bar = bar_base + dg::kWarps * dg::kStages * 8;
    const uint32_t low_ring = (tab_bar + 8 + 127u) & ~127u;
    if (!IQ4 && low_ring + dg::kLowRingWarps * dg::kRingBytes > dg::kTab) {   // layout assumption broken
        if (tid == 0) atomicExch(a.status, (uint32_t)kStatusBadLayout);
        return;
    }
    const uint32_t ring = IQ4 ? base4 + dg::kRings4 + warp * kRingB
                        : warp < (uint32_t)dg::kLowRingWarps ? low_ring + warp * dg::kRingBytes
                                                             : dg::kHigh + (warp - dg::kLowRingWarps) * dg::kRingBytes;
    float* red = reinterpret_cast<float*>(smem_raw + ((IQ4 ? base4 + dg::kRed4 : dg::kRed) - base));
    DecodeGroup* own_list = reinterpret_cast<DecodeGroup*>(smem_raw + ((IQ4 ? base4 + dg::kList4 : dg::kList) - base));
    OwnScratch& own = *reinterpret_cast<OwnScratch*>(red);
    const uint32_t my_bar = bar_base + warp * dg::kStages * 8;
    bool timed_out = false;

    if (ONE) own.mask[tid] = 0ull;
    if (lane == 0) {
        for (int s = 0; s < dg::kStages; ++s) mbar_init(my_bar + 8 * s, 1);
        if (warp == 0) mbar_init(tab_bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (!IQ4 && tid == 0) {   // the 64 KB table image comes from global memory (L2 after the first block) in four bulk copies
        mbar_expect_tx(tab_bar, dg::kTabBytes);
        for (uint32_t i = 0; i < 4; ++i) bulk_g2s(dg::kTab + i * 16384u, a.luts + i * 16384u, 16384u, tab_bar);
    }

    const uint32_t teams_total = gridDim.x * n_teams, team_global = blockIdx.x * n_teams + team;
    const uint32_t n_layers = ONE ? 1 : a.n_layers;
    const Divisor by_teams(teams_total), by_tiles(RT), by_shared(dg::kCostShared);

    // Up to here nothing depended on the router kernel, so a block scheduled early (programmatic
    // dependent launch) has its barriers and table copy under way while that kernel's tail runs.  The
    // next kernel is released only now: what it reads before its own wait (the selection) is then final.
    pdl_wait();
    pdl_trigger();

    // This team's contiguous share of the flat list.  A shared-expert (Q8_0) tile takes longer
    // than a routed one (four ring stages, each a round trip), so the cut is made in cost units:
    // kCostRouted per routed tile, kCostShared per shared tile (a layer's shared groups come last).
    if (ONE) {
        own_groups<dg::kWarps * 32>(own, own_list, s_cuts, a.sel, d, a.n_tokens, dg::kCostRouted, dg::kCostShared);
    } else {
        if (warp == 0) layer_cuts(s_cuts, a.groups, a.n_tokens, n_layers, dg::kCostRouted, dg::kCostShared);
        __syncthreads();
    }
    uint32_t left;   // tiles still to do
    const ListPlace at = list_share(s_cuts, a.n_tokens, n_layers, by_tiles, dg::kCostRouted, by_shared, team_global, by_teams, left);
    uint32_t rt = at.rt;   // the consumers' tile in its group
    DecodeGroup* my_list = own_list + (ONE ? 0 : team * (rk::kMaxGroups / n_teams));   // ONE: the layer's groups; else the share's
    if (!ONE) {   // they fit: decode_gateup_rows
        const uint32_t first = s_cuts.groups[at.l] + at.gi, n = left ? by_tiles(rt + left + RT - 1) : 0;
        for (uint32_t i = lt; i < n; i += team_threads) {
            uint32_t l = at.l;
            while (s_cuts.groups[l + 1] <= first + i) ++l;
            reinterpret_cast<uint4*>(my_list)[i] = __ldcg(reinterpret_cast<const uint4*>(decode_group_at(a.groups, a.n_tokens, d.n_used, l, first + i - s_cuts.groups[l])));
        }
        asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(team_threads) : "memory");
    }
    // (read again where it is needed: a record in registers costs the IQ3_XXS form spills, 50 us of 1950 at 40 layers of 16 tokens)
    const uint32_t recs = smem_addr(my_list);
    auto record = [&](uint32_t i) {
        const uint4 v = lds128(recs + 16 * i);
        return DecodeGroup{v.x, {v.y, v.z}, v.w};
    };
    // (a record's place is computed when a group begins: counters cost the IQ3_XXS form spills, 2.5 % of its time)
    const uint32_t total = (ONE ? at.gi * RT : 0) + rt + left;
    const size_t mat_tiles = (size_t)KB * RT;

    // producer cursor over (tile, quarter); lane 0 only.  A routed tile is one stage, a shared
    // tile four (its quarters).
    uint32_t p_left = left, p_q = 0;
    uint32_t p_rt = rt;
    bool p_new = true;                            // the group record must be (re)loaded
    // Next tile of the gate and the up matrix, routed or shared: pointers, or ONE: its number, since the matrices are the parameters' first then
    // (with pointers the IQ3_XXS form spills, 4 % of its time; of several layers the number and the layer cost 5 %).
    const uint8_t* p_g = nullptr;
    const uint8_t* p_u = nullptr;
    uint32_t p_tile = 0;
    bool p_shared = false;
    auto issue = [&](uint32_t stage) {
        if (p_left == 0) return;
        if (p_new) {   // first call, or the previous group is finished
            p_new = false;
            const DecodeGroup r = record((total - p_left) / RT);
            const GateupDecodeArgs::Mats& m = a.layer[ONE ? 0 : r.layer];
            p_shared = r.shared();
            if (ONE) {
                p_tile = (p_shared ? 0 : r.expert() * (uint32_t)mat_tiles) + kb * RT + p_rt;
            } else if (!p_shared) {
                const size_t tile = (size_t)r.expert() * mat_tiles + (size_t)kb * RT + p_rt;
                p_g = m.gate + tile * kTileR; p_u = m.up + tile * kTileR;
            } else {
                const size_t tile = (size_t)kb * RT + p_rt;
                p_g = m.sh_gate + tile * kTileQ8; p_u = m.sh_up + tile * kTileQ8;
            }
        }
        auto next_tile = [&]() {
            --p_left;
            if (++p_rt == RT) { p_rt = 0; p_new = true; }
        };
        const uint32_t bar = my_bar + 8 * stage, dst = ring + stage * kStageB;
        if (!p_shared) {
            mbar_expect_tx(bar, 2 * kTileR);
            bulk_g2s(dst, ONE ? a.layer[0].gate + (size_t)p_tile * kTileR : p_g, kTileR, bar);
            bulk_g2s(dst + kTileR, ONE ? a.layer[0].up + (size_t)p_tile * kTileR : p_u, kTileR, bar);
            if (ONE) { ++p_tile; } else { p_g += kTileR; p_u += kTileR; }
            next_tile();
        } else {
            mbar_expect_tx(bar, 2 * dg::kQ8Quarter);   // a quarter = two 32-column blocks = one 1088-byte piece
            bulk_g2s(dst, (ONE ? a.layer[0].sh_gate + (size_t)p_tile * kTileQ8 : p_g) + dg::kQ8Quarter * p_q, dg::kQ8Quarter, bar);
            bulk_g2s(dst + dg::kQ8Quarter, (ONE ? a.layer[0].sh_up + (size_t)p_tile * kTileQ8 : p_u) + dg::kQ8Quarter * p_q, dg::kQ8Quarter, bar);
            if (++p_q == 4) {
                p_q = 0;
                if (ONE) { ++p_tile; } else { p_g += kTileQ8; p_u += kTileQ8; }
                next_tile();
            }
        }
    };
    if (lane == 0)
        for (int s = 0; s < dg::kStages; ++s) issue(s);

    const uint32_t grid_c = dg::kTab + lane * 4;
    const uint32_t i_off = 64 * g + piece_at(g, t), s_off = 32 * g + 16 * ((t >> 1) ^ ((g >> 2) & 1u)) + 8 * (t & 1u);   // this lane's pieces of row g (rows g+8 alike)
    uint32_t cnt = 0;   // stages consumed by this warp
    uint32_t b0[8], b1[8], n0[8], n1[8];
    float wcol0 = 0.f, wcol1 = 0.f;   // digit weights of the two C columns of this lane (2t, 2t+1)
    bool shared = false;   // the group is one of the shared expert's
    uint32_t e_n = 0, e_buf = 0;   // tiles waiting for the team-wide reduction (the last e_n up to rt): count, buffer
    bool new_group = true;
    float* h = nullptr;   // where this thread's reduction outputs of the current group go: (token, slot) of token slot lt & 1; null: none

    if (!IQ4 && !mbar_wait_bounded(tab_bar, 0)) timed_out = true;   // every thread observes the table's arrival itself

    for (; left; --left) {
        if (new_group) {
            new_group = false;
            const DecodeGroup rec = record((total - left) / RT);
            shared = rec.shared();
            const uint32_t row0 = ONE ? 0 : rec.layer * a.n_tokens;   // the layer's first row of the planes
            {
                const uint32_t ets = lt & 1u;   // the reduction below gives this thread token slot (j & 1) == (lt & 1)
                h = nullptr;
                if (ets < rec.ntok()) {
                    const uint32_t pr = rec.pair_of(ets), tok = pr >> 4, slot = pr & 15u;
                    h = (ONE || rec.layer + 1 == n_layers ? a.h_last : a.h + (size_t)row0 * (d.n_used + 1) * d.n_ff) + ((size_t)tok * (d.n_used + 1) + slot) * d.n_ff;
                }
            }
            // B operand: column g of the MMA = (token slot g >> 2, digit g & 3); this warp's 256 columns
            const uint32_t ts = g >> 2, dgt = g & 3u;
            if (ts < rec.ntok()) {
                const uint32_t row = row0 + (rec.pair_of(ts) >> 4);
                const int8_t* pl = a.planes + (((size_t)row * KB + kb) * 8 + dgt) * 256;
#pragma unroll
                for (int sb = 0; sb < 8; ++sb) {
                    if (IQ4 && !rec.shared()) {   // iq4_word_gu's order
                        const uint2 v = *reinterpret_cast<const uint2*>(pl + 32 * sb + 8 * t);
                        b0[sb] = prmt(v.x, 0u, 0x3120u); b1[sb] = prmt(v.y, 0u, 0x3120u);
                    } else if (!rec.shared()) {   // lane t owns elements 8t .. 8t+7 of each sub-block
                        const uint2 v = *reinterpret_cast<const uint2*>(pl + 32 * sb + 8 * t);
                        const uint2 n = *reinterpret_cast<const uint2*>(pl + 1024 + 32 * sb + 8 * t);
                        b0[sb] = v.x; b1[sb] = v.y; n0[sb] = n.x; n1[sb] = n.y;
                    } else {               // elements 4t .. 4t+3 and 16+4t .. 16+4t+3
                        b0[sb] = *reinterpret_cast<const uint32_t*>(pl + 32 * sb + 4 * t);
                        b1[sb] = *reinterpret_cast<const uint32_t*>(pl + 32 * sb + 16 + 4 * t);
                    }
                }
            } else {
#pragma unroll
                for (int sb = 0; sb < 8; ++sb) { b0[sb] = 0; b1[sb] = 0; n0[sb] = 0; n1[sb] = 0; }
            }
            const uint32_t cts = t >> 1;   // token slot of C columns 2t, 2t+1
            wcol0 = 0.f; wcol1 = 0.f;
            if (cts < rec.ntok()) {
                const float sc = a.xscale[(row0 + (rec.pair_of(cts) >> 4)) * KB + kb];
                const float w0 = (t & 1u) ? 16384.f : 1.f;   // 128^(2 * (t & 1))
                wcol0 = sc * w0;
                wcol1 = sc * w0 * 128.f;
            }
        }
        float ga, gb, ua, ub;
        // the token's other two digits sit in lane t^1
        auto both_halves = [&]() {
            ga += __shfl_xor_sync(0xFFFFFFFFu, ga, 1); gb += __shfl_xor_sync(0xFFFFFFFFu, gb, 1);
            ua += __shfl_xor_sync(0xFFFFFFFFu, ua, 1); ub += __shfl_xor_sync(0xFFFFFFFFu, ub, 1);
        };
        if (!shared) {
            const uint32_t stage = cnt % dg::kStages, parity = (cnt / dg::kStages) & 1u;
            if (!mbar_wait_bounded(my_bar + 8 * stage, parity)) timed_out = true;
            const uint32_t sbase = ring + stage * kStageB;
            int ig[4], iu[4];
            if (IQ4) {
                uint4 hg, hu;
                iq4_tile_gu(sbase, i_off, g, b0, b1, ig, hg);
                iq4_tile_gu(sbase + kTileIq4, i_off, g, b0, b1, iu, hu);
                ga = f16_bits_to_f32(hg.x & 0xFFFFu) * ((float)ig[0] * wcol0 + (float)ig[1] * wcol1);
                gb = f16_bits_to_f32(hg.z & 0xFFFFu) * ((float)ig[2] * wcol0 + (float)ig[3] * wcol1);
                ua = f16_bits_to_f32(hu.x & 0xFFFFu) * ((float)iu[0] * wcol0 + (float)iu[1] * wcol1);
                ub = f16_bits_to_f32(hu.z & 0xFFFFu) * ((float)iu[2] * wcol0 + (float)iu[3] * wcol1);
            } else {
            iq3_tile(sbase, i_off, s_off, g, grid_c, b0, b1, n0, n1, ig);
            iq3_tile(sbase + kTileIq3, i_off, s_off, g, grid_c, b0, b1, n0, n1, iu);
            const uint32_t dwa = lds32(sbase + 1664 + 2 * (g & ~1u)), dwb = lds32(sbase + 1664 + 2 * ((g + 8) & ~1u));
            const uint32_t uwa = lds32(sbase + kTileIq3 + 1664 + 2 * (g & ~1u)), uwb = lds32(sbase + kTileIq3 + 1664 + 2 * ((g + 8) & ~1u));
            const uint32_t sh = 16 * (g & 1u);
            // d * 0.25 * (2s+1) * m  ==  d * (0.5 + s) * 0.5 * m
            ga = (f16_bits_to_f32((dwa >> sh) & 0xFFFFu) * 0.25f) * ((float)ig[0] * wcol0 + (float)ig[1] * wcol1);
            gb = (f16_bits_to_f32((dwb >> sh) & 0xFFFFu) * 0.25f) * ((float)ig[2] * wcol0 + (float)ig[3] * wcol1);
            ua = (f16_bits_to_f32((uwa >> sh) & 0xFFFFu) * 0.25f) * ((float)iu[0] * wcol0 + (float)iu[1] * wcol1);
            ub = (f16_bits_to_f32((uwb >> sh) & 0xFFFFu) * 0.25f) * ((float)iu[2] * wcol0 + (float)iu[3] * wcol1);
            }
            both_halves();
            stage_read();
            __syncwarp();
            if (lane == 0) issue(stage);
            ++cnt;
        } else {
            ga = gb = ua = ub = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t stage = cnt % dg::kStages, parity = (cnt / dg::kStages) & 1u;
                if (!mbar_wait_bounded(my_bar + 8 * stage, parity)) timed_out = true;
                const uint32_t sbase = ring + stage * kStageB;
                q8_quarter(sbase, lane, g, b0[2 * q], b1[2 * q], b0[2 * q + 1], b1[2 * q + 1], wcol0, wcol1, ga, gb);
                q8_quarter(sbase + dg::kQ8Quarter, lane, g, b0[2 * q], b1[2 * q], b0[2 * q + 1], b1[2 * q + 1], wcol0, wcol1, ua, ub);
                stage_read();
                __syncwarp();
                if (lane == 0) issue(stage);
                ++cnt;
            }
            both_halves();
        }
        float* my_red = red + (warp * 2 + e_buf) * dg::kRedFloats;
        if ((t & 1u) == 0) {
            const uint32_t ts = t >> 1;   // [tile][row 16][token 2][matrix 2]
            *reinterpret_cast<float2*>(my_red + (((e_n * 16 + g) * 2 + ts) * 2)) = make_float2(ga, ua);
            *reinterpret_cast<float2*>(my_red + (((e_n * 16 + g + 8) * 2 + ts) * 2)) = make_float2(gb, ub);
        }
        ++e_n;
        if (e_n == dg::kGroupTiles || (rt & (dg::kGroupTiles - 1)) == dg::kGroupTiles - 1 || left == 1) {
            // team-wide: sum the KB column-block partials, SwiGLU, store.  The scratch is double
            // buffered, so one barrier per reduction is enough.
            asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(team_threads) : "memory");
            for (uint32_t j = lt; j < e_n * 32; j += team_threads) {   // team_threads is even: j & 1 == lt & 1
                const uint32_t ts = j & 1u, row = j >> 1;   // row within the waiting tiles
                if (h) {
                    float gsum = 0.f, usum = 0.f;
                    for (uint32_t w = 0; w < KB; ++w) {
                        const float2 r = *reinterpret_cast<const float2*>(red + ((team * KB + w) * 2 + e_buf) * dg::kRedFloats + (row * 2 + ts) * 2);
                        gsum += r.x; usum += r.y;
                    }
                    const float hv = swiglu(gsum, usum);
                    h[(rt + 1 - e_n) * 16 + row] = hv;
                }
            }
            e_n = 0;
            e_buf ^= 1u;
        }
        if (++rt == RT) { rt = 0; new_group = true; }
    }
    if (timed_out && lane == 0) atomicExch(a.status, (uint32_t)kStatusWaitTimeout);
}

bool decode_gateup_ok(const qkm_dims& d) {
    const uint32_t KB = d.n_embd / 256;
    return d.n_embd % 256 == 0 && KB >= 2 && KB <= 8 && (KB & (KB - 1)) == 0 && d.n_ff % 64 == 0 && d.n_used <= 15;
}

template <bool IQ4, bool ONE>
static cudaError_t gateup_launch(const Launch& L, const GateupDecodeArgs& a, uint32_t n_blocks) {
    const size_t smem = (IQ4 ? dg::kList4 + 128 : dg::kList) + dg::kListBytes;   // IQ3_XXS: the dynamic area must reach the list's end from wherever it starts
    if (const cudaError_t e = cudaFuncSetAttribute(decode_gateup_kernel<IQ4, ONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) return e;
    const cudaError_t e = launch_kernel(L, decode_gateup_kernel<IQ4, ONE>, dim3(n_blocks), dim3(dg::kWarps * 32), smem, a);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}
// The records of a team's share of several layers find room in its part of the list: at most so many (layer, token) rows.  (A row has up to 16
// groups, and a share of routed tiles, the cheaper ones, has the most: one of n_teams * n_blocks shares gets at most
// 16 rows * kCostShared / (n_teams * n_blocks * kCostRouted) groups and two begun ones, with 8 rows a block 160 / n_teams + 2 of 800 / n_teams.)
uint32_t decode_gateup_rows(uint32_t n_blocks) { return 8 * n_blocks; }

cudaError_t launch_decode_gateup(const Launch& L, const GateupDecodeArgs& a, uint32_t n_blocks) {
    if (!decode_gateup_ok(a.d) || a.n_tokens > rk::kMaxTokens || a.n_layers > kDecMaxLayers) return cudaErrorInvalidValue;
    if (a.n_layers != 1 && (!a.groups.group || a.n_layers * a.n_tokens > decode_gateup_rows(n_blocks))) return cudaErrorInvalidValue;
    if (a.gateup_type != QKM_TYPE_IQ3_XXS && a.gateup_type != QKM_TYPE_IQ4_XS) return cudaErrorInvalidValue;
    if (a.gateup_type == QKM_TYPE_IQ4_XS) return a.n_layers == 1 ? gateup_launch<true, true>(L, a, n_blocks) : gateup_launch<true, false>(L, a, n_blocks);
    return a.n_layers == 1 ? gateup_launch<false, true>(L, a, n_blocks) : gateup_launch<false, false>(L, a, n_blocks);
}

}  // namespace qkm
