// Down projection of the fused decode sequence for larger batches, expert major: routed experts (IQ4_XS or Q6_K) and the shared
// expert (Q8_0), then a fold of the weighted contributions in slot order:
//   contrib[t][s] = w_s * D[ids_s] . h[t][s],   y[t] = sum_s contrib[t][s]   (s = n_used: the shared expert).
//
// Replaces moe_down_iq4.comp / moe_down_q6k.comp + moe_down_q8b.comp and the slot-order sum of add_rms3_grouped.comp:22-27.
//
// The token-major kernels unpack an expert's weights once for every token that chose it.  Here the pairs are grouped by expert as in
// the gate/up kernel (of several layers the router kernel's lists, of one by every block itself), a group is an expert with up to two of its tokens, and a
// team of two warps (one per 256 columns) walks 16-row tiles of a contiguous share of the (group, tile) list: at 64 tokens of 256 experts,
// top 8, 317 groups instead of 512 pairs.  The price is the grouping, the contribution rows' way through the L2 and a second
// launch, about 7 us together.
//
// Bound by instruction issue, as the token-major kernels are.  Layer time on the B200, IQ3_XXS gate/up, token major -> grouped:
//   IQ4_XS, 256 experts, top 8:  24 tokens 91.0 -> 91.9 us, 32: 110.9 -> 109.4, 40: 130.2 -> 126.7, 64: 187.0 -> 173.7
//   IQ4_XS, 512 experts, top 10: 32 tokens 143.3 -> 144.4, 40: 169.0 -> 167.6, 64: 245.0 -> 232.4
//   Q6_K,   256 experts, top 8:  40 tokens 127.5 -> 131.2, 64: 183.3 -> 180.6;  128 experts, top 4, 64: 125.2 -> 108.7
// Q6_K gains less: its multiplies, 16 MMAs and 64 integer multiply-adds for two tokens, outweigh the unpacking that is shared.
//
// Arithmetic as in the token-major kernels: h as four int8 digit planes per 256 columns (28-bit fixed point), exact integer sums;
// an IQ4_XS or Q8_0 tile takes both tokens in one MMA (four columns each), a Q6_K tile one MMA per token (its 16-column
// scales take the other four columns).
#include "qkm_dec_rank.cuh"
#include "qkm_dec_tiles.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"
#include "qkm_tiles.cuh"

namespace qkm {

namespace dp {
constexpr int kWarps = 16;
constexpr uint32_t kHalfQ8 = kTileQ8 / 2;           // a stage of the shared expert: four of a tile's eight block columns
constexpr uint32_t kStages = 3;
constexpr uint32_t kGroupTiles = 4;                 // tiles between two sums over a team
constexpr uint32_t kTab = 0x10000u, kTabBytes = 0x10000u, kHigh = kTab + kTabBytes;   // IQ4_XS table image, absolute shared-window address
template <bool Q6> struct Cfg {
    static constexpr uint32_t kTile = Q6 ? kTileQ6 : kTileIq4, kRing = kStages * kTile;   // 10080, 6528; a Q8_0 half fits a stage
    static constexpr uint32_t kLow = 9;                                                   // IQ4_XS: rings below the table, up against it; the others above
    static constexpr uint32_t kScratch = Q6 ? kWarps * kRing : kHigh + (kWarps - kLow) * kRing;   // Q6_K: from the aligned start
    static constexpr uint32_t kRed = kScratch + kWarps * 1024;                            // digits of a warp's 256 columns, one token at a time
    static constexpr uint32_t kRedBytes = kWarps * 2 * kGroupTiles * 16 * 2 * 4;          // [warp][buffer][tile][row][token]
    static constexpr uint32_t kList = kRed + kRedBytes;                                   // groups of a layer on its own
    static constexpr uint32_t kEnd = kList + rk::kMaxGroups * sizeof(DecodeGroup);
    static_assert(sizeof(OwnScratch) <= kRedBytes, "the grouping's working set lies where the partial sums come later");
    static constexpr uint32_t kDyn = Q6 ? kEnd + 128 : kEnd - 1024;                       // the first KB of the window is the system's
};
static_assert(Cfg<true>::kDyn <= 231000 && Cfg<false>::kDyn <= 231000 && kHalfQ8 <= kTileIq4, "with the static part at most 227 KB");
}  // namespace dp

// ONE: one layer, whose pairs the block groups itself; else the router kernel's lists
template <bool Q6, bool ONE>
__global__ void __launch_bounds__(dp::kWarps * 32, 1)
decode_down_group_kernel(const __grid_constant__ DownDecodeArgs a) {
    using C = dp::Cfg<Q6>;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) unsigned long long s_bar[dp::kWarps * dp::kStages + 1];
    __shared__ LayerCuts s_cuts;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    const qkm_dims d = a.d;
    const uint32_t n_slots = d.n_used + 1, KB = 2, RT = d.n_embd / 16;
    const uint32_t n_teams = dp::kWarps / KB, team = warp / KB, kb = warp - team * KB, team_threads = KB * 32, lt = tid - team * team_threads;
    const uint32_t win0 = smem_addr(smem_raw), base = Q6 ? (win0 + 127u) & ~127u : 0u;
    if (!Q6) {   // the fixed addresses must lie inside the dynamic area
        uint32_t dyn_size;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_size));
        if (win0 > dp::kTab - C::kLow * C::kRing || win0 + dyn_size < C::kEnd) {
            if (tid == 0) atomicExch(a.status, (uint32_t)kStatusBadLayout);
            return;
        }
    }
    const uint32_t ring = Q6 ? base + warp * C::kRing : warp < C::kLow ? dp::kTab - (warp + 1) * C::kRing : dp::kHigh + (warp - C::kLow) * C::kRing;
    const uint32_t my_dig = base + C::kScratch + warp * 1024;
    uint8_t* dig = smem_raw + (my_dig - win0);
    float* red = reinterpret_cast<float*>(smem_raw + (base + C::kRed - win0));
    DecodeGroup* own_list = reinterpret_cast<DecodeGroup*>(smem_raw + (base + C::kList - win0));
    OwnScratch& own = *reinterpret_cast<OwnScratch*>(red);
    const uint32_t n_layers = ONE ? 1 : a.n_layers;
    const uint32_t my_bar = smem_addr(&s_bar[warp * dp::kStages]), bar_tab = smem_addr(&s_bar[dp::kWarps * dp::kStages]);
    bool timed_out = false;

    if (ONE) own.mask[tid] = 0ull;
    if (lane == 0) {
        for (uint32_t s = 0; s < dp::kStages; ++s) mbar_init(my_bar + 8 * s, 1);
        if (warp == 0) mbar_init(bar_tab, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (!Q6 && tid == 0) {
        mbar_expect_tx(bar_tab, dp::kTabBytes);
        for (uint32_t i = 0; i < 4; ++i) bulk_g2s(dp::kTab + i * 16384u, a.lut + i * 16384u, 16384u, bar_tab);
    }
    const uint32_t teams_total = gridDim.x * n_teams, team_global = blockIdx.x * n_teams + team;
    const Divisor by_teams(teams_total), by_tiles(RT);

    // the selection and its groups were final before the gate/up kernel released this one
    if (ONE) {
        own_groups<dp::kWarps * 32>(own, own_list, s_cuts, layer_sel(a, 0), d, a.n_tokens, 1, 1);
    } else {
        if (warp == 0) layer_cuts(s_cuts, a.groups, a.n_tokens, n_layers, 1, 1);
        __syncthreads();
    }
    uint32_t left;   // tiles still to do
    ListPlace at = list_share(s_cuts, a.n_tokens, n_layers, by_tiles, 1, Divisor(1), team_global, by_teams, left);
    auto group = [&](const ListPlace& p) {
        const uint4 v = ONE ? reinterpret_cast<const uint4*>(own_list)[p.gi] : __ldcg(reinterpret_cast<const uint4*>(decode_group_at(a.groups, a.n_tokens, d.n_used, p.l, p.gi)));
        return DecodeGroup{v.x, {v.y, v.z}, v.w};
    };
    const size_t mat_tiles = (size_t)KB * RT;

    // producer cursor; lane 0 only.  A routed tile is one stage, a shared tile two.
    uint32_t p_left = left, p_half = 0;
    ListPlace p_at = at;
    bool p_new = true;                     // the group record must be (re)loaded
    const uint8_t* p_src = nullptr;
    bool p_shared = false;
    auto issue = [&](uint32_t stage) {
        if (p_left == 0 || timed_out) return;
        if (p_new) {
            p_new = false;
            const DecodeGroup r = group(p_at);
            p_shared = r.shared();
            const DownDecodeArgs::Mats& m = a.layer[ONE ? 0 : p_at.l];
            p_src = p_shared ? m.sh + ((size_t)kb * RT + p_at.rt) * kTileQ8 : m.w + ((size_t)r.expert() * mat_tiles + (size_t)kb * RT + p_at.rt) * C::kTile;
        }
        const uint32_t n = p_shared ? dp::kHalfQ8 : C::kTile;
        mbar_expect_tx(my_bar + 8 * stage, n);
        bulk_g2s(ring + stage * C::kTile, p_src, n, my_bar + 8 * stage);
        p_src += n;
        if (p_shared && !p_half) { p_half = 1; return; }
        p_half = 0;
        --p_left;
        if (++p_at.rt == RT) { p_at.rt = 0; p_at.next_group(s_cuts); p_new = true; }
    };
    if (lane == 0)
        for (uint32_t s = 0; s < dp::kStages; ++s) issue(s);
    pdl_wait();   // h is the gate/up kernel's output
    pdl_trigger();
    if (!Q6 && !mbar_wait_bounded(bar_tab, 0)) timed_out = true;   // every thread observes the table's arrival itself

    const uint32_t i_off = 64 * g + piece_at(g, t), tab_c = dp::kTab + lane * 4;
    uint32_t stage = 0, phase = 0, e_n = 0, e_buf = 0;   // tiles waiting for the team's sum (the last e_n up to at.rt): count, buffer
    bool new_group = true, live = false;
    DecodeGroup rec{}, rec_next{};
    if (!ONE && left) rec_next = group(at);   // a group's record is read while the group before is worked on
    size_t out = 0;                          // where this thread's sums of the current group go: (token, slot) of token slot lt & 1
    constexpr int NB = Q6 ? 2 : 1;
    uint32_t b0[NB][8], b1[NB][8];           // B operands (Q6_K: per token)
    float w0 = 0.f, w1 = 0.f;                // weights of this lane's two C columns (Q6_K: of the two tokens)
    auto next = [&]() {
        stage_read();
        __syncwarp();
        if (lane == 0) issue(stage);
        if (++stage == dp::kStages) { stage = 0; phase ^= 1u; }
    };
    for (; left; --left) {
        if (new_group) {
            new_group = false;
            if (ONE) {
                rec = group(at);
            } else {
                rec = rec_next;
                ListPlace after = at;
                after.next_group(s_cuts);
                if (after.l < n_layers) rec_next = group(after);
            }
            const bool shared = rec.shared();
            const float* h = layer_h(a, ONE ? 0 : at.l);
            const qkm_sel* sel = layer_sel(a, ONE ? 0 : at.l);
            live = (lt & 1u) < rec.ntok();
            if (live) {
                const uint32_t pr = rec.pair_of(lt & 1u);
                out = ((size_t)((ONE ? 0 : at.l * a.n_tokens) + (pr >> 4)) * n_slots + (pr & 15u)) * d.n_embd;
            }
            float wt[2] = {0.f, 0.f};        // routing weight x plane scale
            float4 hv4[2][2];
#pragma unroll
            for (int ts = 0; ts < 2; ++ts) {
                const uint32_t pr = rec.pair_of((uint32_t)ts < rec.ntok() ? ts : 0), tok = pr >> 4, slot = pr & 15u;
                const float* hs = h + ((size_t)tok * n_slots + slot) * d.n_ff + 256 * kb + 8 * lane;
                hv4[ts][0] = *reinterpret_cast<const float4*>(hs); hv4[ts][1] = *reinterpret_cast<const float4*>(hs + 4);
                if ((uint32_t)ts < rec.ntok()) wt[ts] = slot < d.n_used ? sel[tok].w[slot] : sel[tok].w_shared;
            }
#pragma unroll
            for (int ts = 0; ts < 2; ++ts) {
                const float hv[8] = {hv4[ts][0].x, hv4[ts][0].y, hv4[ts][0].z, hv4[ts][0].w, hv4[ts][1].x, hv4[ts][1].y, hv4[ts][1].z, hv4[ts][1].w};
                float m = 0.f;
                bool bad = false;
#pragma unroll
                for (int i = 0; i < 8; ++i) { m = fmaxf(m, fabsf(hv[i])); bad |= !(fabsf(hv[i]) <= 3.0e38f); }
                m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));   // non-negative floats order like their bits
                const bool any_bad = __any_sync(0xFFFFFFFFu, bad), off = (uint32_t)ts >= rec.ntok();
                const int p = any_bad ? 0 : digit_exponent(m);
                const float up = ldexpf(1.0f, p);
                uint32_t dg[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) dg[i] = any_bad || off ? 0u : digits4(__float2int_rn(hv[i] * up));
                wt[ts] *= any_bad ? __int_as_float(0x7FC00000) : ldexpf(Q6 && !shared ? 0.25f : 1.0f, -p);
                const bool perm = !Q6 && !shared;   // iq4_word's order 0, 2, 1, 3; else as they come
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; ++j) {   // plane j of elements 8 lane .. 8 lane + 7
                    const uint32_t sel = 0x4040u + 0x1111u * j;   // byte j of a, byte j of b, twice
                    const uint32_t p0 = prmt_dec(dg[0], perm ? dg[2] : dg[1], sel), p1 = prmt_dec(perm ? dg[1] : dg[2], dg[3], sel);
                    const uint32_t p2 = prmt_dec(dg[4], perm ? dg[6] : dg[5], sel), p3 = prmt_dec(perm ? dg[5] : dg[6], dg[7], sel);
                    *reinterpret_cast<uint2*>(dig + 256 * j + 8 * lane) = make_uint2(prmt_dec(p0, p1, 0x5410u), prmt_dec(p2, p3, 0x5410u));
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t at = my_dig + (g & 3u) * 256 + 32 * j;
                    if (Q6 && !shared) {   // lanes g < 4: digit g of the first 16-column group in b0; g >= 4: digit g - 4 of the second in b1
                        const uint32_t v = lds32(at + 16 * (g >> 2) + 4 * t);
                        b0[ts % NB][j] = g < 4 ? v : 0u;
                        b1[ts % NB][j] = g < 4 ? 0u : v;
                    } else if ((g >> 2) == (uint32_t)ts) {   // column g: digit g & 3 of token g >> 2
                        if (perm) { const uint2 v = lds64(at + 8 * t); b0[0][j] = v.x; b1[0][j] = v.y; }
                        else { b0[0][j] = lds32(at + 4 * t); b1[0][j] = lds32(at + 16 + 4 * t); }
                    }
                }
            }
            if (Q6 && !shared) { w0 = wt[0]; w1 = wt[1]; }
            else {
                w0 = ((t >> 1) ? wt[1] : wt[0]) * ((t & 1u) ? 16384.f : 1.f);   // digits 2 (t & 1), + 1 of token t >> 1
                w1 = w0 * 128.f;
            }
        }
        float va = 0.f, vb = 0.f, va1 = 0.f, vb1 = 0.f;   // rows g, g + 8 (Q6_K tiles: of tokens 0 and 1)
        if (!rec.shared()) {
            if (!mbar_wait_bounded(my_bar + 8 * stage, phase)) timed_out = true;
            const uint32_t tb = ring + stage * C::kTile;
            if (Q6) {
                // the eight scales of this lane's groups (even groups for t < 2, odd for t >= 2), rows g and g+8
                const uint2 scA = lds64(tb + 16 * g + 8 * (t >> 1)), scB = lds64(tb + 16 * (g + 8) + 8 * (t >> 1));
                const uint4 hA = lds128(tb + 2304 + i_off), hB = lds128(tb + 2816 + i_off);
                int acc[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const uint4 qA = lds128(tb + 256 + hf * 1024 + i_off), qB = lds128(tb + 768 + hf * 1024 + i_off);
                    uint32_t a0[4], a2[4], a1[4], a3[4];
                    q6k_words(qA.x, qA.z, hf ? hA.z : hA.x, a0);   // row g, l = 4t..
                    q6k_words(qA.y, qA.w, hf ? hA.w : hA.y, a2);   // row g, l = 16 + 4t..
                    q6k_words(qB.x, qB.z, hf ? hB.z : hB.x, a1);   // row g + 8
                    q6k_words(qB.y, qB.w, hf ? hB.w : hB.y, a3);
#pragma unroll
                    for (int qd = 0; qd < 4; ++qd) {
                        const int j = 4 * hf + qd;
                        const uint32_t sel = 0x8880u + (uint32_t)(j & 3) * 0x1111u;   // byte j & 3, sign-extended
                        const int sa = (int)prmt_dec(hf ? scA.y : scA.x, 0u, sel), sb = (int)prmt_dec(hf ? scB.y : scB.x, 0u, sel);
#pragma unroll
                        for (int ts = 0; ts < NB; ++ts) {
                            int c[4];
                            mma_s8_first(c, a0[qd], a1[qd], a2[qd], a3[qd], b0[ts][j], b1[ts][j]);
                            acc[ts][0] += sa * c[0]; acc[ts][1] += sa * c[1]; acc[ts][2] += sb * c[2]; acc[ts][3] += sb * c[3];
                        }
                    }
                }
                const uint32_t d2 = lds32(tb + 3328 + 2 * (g & ~1u)), d8 = lds32(tb + 3328 + 16 + 2 * (g & ~1u));
                const float da = f16_bits_to_f32((d2 >> (16 * (g & 1u))) & 0xFFFFu), db = f16_bits_to_f32((d8 >> (16 * (g & 1u))) & 0xFFFFu);
                const float q0 = (t & 1u) ? 16384.f : 1.f, q1 = q0 * 128.f;   // columns 2t, 2t+1: digits 2 (t & 1), + 1 of group t / 2
                va = w0 * (da * ((float)acc[0][0] * q0 + (float)acc[0][1] * q1)); vb = w0 * (db * ((float)acc[0][2] * q0 + (float)acc[0][3] * q1));
                va1 = w1 * (da * ((float)acc[1][0] * q0 + (float)acc[1][1] * q1)); vb1 = w1 * (db * ((float)acc[1][2] * q0 + (float)acc[1][3] * q1));
                va += __shfl_xor_sync(0xFFFFFFFFu, va, 2); vb += __shfl_xor_sync(0xFFFFFFFFu, vb, 2);
                va1 += __shfl_xor_sync(0xFFFFFFFFu, va1, 2); vb1 += __shfl_xor_sync(0xFFFFFFFFu, vb1, 2);
                if (t >> 1) { va = va1; vb = vb1; }   // lanes t >> 1: token
            } else {
                const uint4 hd = lds128(tb + 16 * g);   // row g (x: d | scales_h << 16, y: scales_l), row g+8 (z, w)
                uint32_t ea, oa, eb, ob;
                iq4_scales(hd.y, hd.x >> 16, ea, oa);
                iq4_scales(hd.w, hd.z >> 16, eb, ob);
                int acc[4] = {0, 0, 0, 0};
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const uint4 qa4 = lds128(tb + 128 + hf * 1024 + i_off), qb4 = lds128(tb + 640 + hf * 1024 + i_off);
                    const uint32_t wa[4] = {qa4.x, qa4.y, qa4.z, qa4.w}, wb[4] = {qb4.x, qb4.y, qb4.z, qb4.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int sb = 4 * hf + j;
                        uint32_t a0, a1, a2, a3;
                        iq4_word(wa[j], tab_c, a0, a2);
                        iq4_word(wb[j], tab_c, a1, a3);
                        int c[4];
                        mma_s8_first(c, a0, a1, a2, a3, b0[0][sb], b1[0][sb]);
                        const uint32_t sel = 0x8880u + (uint32_t)(sb >> 1) * 0x1111u;   // byte sb / 2, sign-extended
                        const int la = (int)prmt_dec((sb & 1) ? oa : ea, 0u, sel), lb = (int)prmt_dec((sb & 1) ? ob : eb, 0u, sel);
                        acc[0] += la * c[0]; acc[1] += la * c[1]; acc[2] += lb * c[2]; acc[3] += lb * c[3];
                    }
                }
                va = f16_bits_to_f32(hd.x & 0xFFFFu) * ((float)acc[0] * w0 + (float)acc[1] * w1);
                vb = f16_bits_to_f32(hd.z & 0xFFFFu) * ((float)acc[2] * w0 + (float)acc[3] * w1);
            }
        } else {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (!mbar_wait_bounded(my_bar + 8 * stage, phase)) timed_out = true;
                const uint32_t tb = ring + stage * C::kTile;
#pragma unroll
                for (int bb = 0; bb < 4; ++bb) {
                    const uint32_t q = tb + 544 * bb;
                    const uint2 qa = lds64(q + 32 + lane * 8), qc = lds64(q + 32 + 256 + lane * 8);   // rows g, g+8: qs[4t..4t+3], qs[16+4t..16+4t+3]
                    int c[4];
                    mma_s8_first(c, qa.x, qc.x, qa.y, qc.y, b0[0][4 * half + bb], b1[0][4 * half + bb]);
                    const uint32_t dw = lds32(q + 2 * (g & ~1u)), dw8 = lds32(q + 2 * (8 + (g & ~1u)));
                    va += f16_bits_to_f32((dw >> (16 * (g & 1u))) & 0xFFFFu) * ((float)c[0] * w0 + (float)c[1] * w1);
                    vb += f16_bits_to_f32((dw8 >> (16 * (g & 1u))) & 0xFFFFu) * ((float)c[2] * w0 + (float)c[3] * w1);
                }
                next();
            }
        }
        // the token's other two digits sit in lane t^1
        va += __shfl_xor_sync(0xFFFFFFFFu, va, 1); vb += __shfl_xor_sync(0xFFFFFFFFu, vb, 1);
        if (!rec.shared()) next();
        if ((t & 1u) == 0) {
            float* r = red + ((warp * 2 + e_buf) * dp::kGroupTiles + e_n) * 32 + (t >> 1);
            r[2 * g] = va; r[2 * (g + 8)] = vb;
        }
        ++e_n;
        if (e_n == dp::kGroupTiles || at.rt + 1 == RT || left == 1) {
            // team-wide: add the column blocks, store.  The scratch is double buffered: one barrier a sum
            asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(team_threads) : "memory");
            for (uint32_t j = lt; j < e_n * 32; j += team_threads)   // team_threads is even: j & 1 == lt & 1
                if (live) {
                    float v = 0.f;
                    for (uint32_t w = 0; w < KB; ++w) v += red[((team * KB + w) * 2 + e_buf) * dp::kGroupTiles * 32 + j];
                    a.contrib[out + (size_t)(at.rt + 1 - e_n) * 16 + (j >> 1)] = v;
                }
            e_n = 0;
            e_buf ^= 1u;
        }
        if (++at.rt == RT) { at.rt = 0; at.next_group(s_cuts); new_group = true; }
    }
    if (timed_out && lane == 0) atomicExch(a.status, (uint32_t)kStatusWaitTimeout);
}

// y[layer][t] = the contributions' sum in slot order
__global__ void __launch_bounds__(256)
decode_fold_kernel(const float* contrib, float* y, uint64_t y_stride, uint32_t n_slots, uint32_t n_embd, uint32_t n_tokens, uint32_t n) {
    const uint32_t i = blockIdx.x * 256 + threadIdx.x, n4 = n_embd / 4;   // a float4 of y each
    pdl_trigger();
    pdl_wait();
    if (i >= n) return;
    const uint32_t row = i / n4, o = i - row * n4, l = row / n_tokens, t = row - l * n_tokens;
    const float4* c = reinterpret_cast<const float4*>(contrib) + (size_t)row * n_slots * n4 + o;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (uint32_t s = 0; s < n_slots; ++s) {
        const float4 q = __ldcg(c + (size_t)s * n4);
        v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
    }
    reinterpret_cast<float4*>(y + l * y_stride)[(size_t)t * n4 + o] = v;
}

// IQ4_XS: from 40 tokens on for every expert count and number of slots that was measured (some cross over at 12 to 37); Q6_K: only
// where an expert also has two tokens on average, since half a pair costs it as much as a whole one.
// With more than ten slots, beyond the token-major kernel's warps, it is the only one (60 experts, top 15: 8 tokens 835 -> 61 us,
// 64 tokens 6483 -> 223 us against the kernels on the raw layout).
bool decode_down_group_better(const qkm_dims& d, uint32_t type, uint32_t n) {
    if (!decode_down_any_ok(d)) return true;
    return n >= 40 && (type != QKM_TYPE_Q6_K || n * d.n_used >= 2 * d.n_expert);
}
bool decode_down_group_ok(const qkm_dims& d) { return d.n_ff == 512 && d.n_used <= 15 && d.n_embd % 64 == 0 && d.n_expert <= rk::kMaxExperts; }

template <bool Q6, bool ONE>
static cudaError_t group_launch(const Launch& L, const DownDecodeArgs& a, uint32_t n_blocks) {
    const size_t smem = dp::Cfg<Q6>::kDyn;
    if (const cudaError_t e = allow_dynamic_smem<decode_down_group_kernel<Q6, ONE>>((int)smem)) return e;
    if (const cudaError_t e = launch_kernel(L, decode_down_group_kernel<Q6, ONE>, dim3(n_blocks), dim3(dp::kWarps * 32), smem, a)) return e;
    const uint32_t n = a.n_layers * a.n_tokens * (a.d.n_embd / 4);
    const cudaError_t e = launch_kernel(L, decode_fold_kernel, dim3((n + 255) / 256), dim3(256), 0, (const float*)a.contrib, a.y, a.y_stride, a.d.n_used + 1, a.d.n_embd, a.n_tokens, n);
    L.count(2);
    return e != cudaSuccess ? e : cudaGetLastError();
}
cudaError_t launch_decode_down_group(const Launch& L, const DownDecodeArgs& a, uint32_t type, uint32_t n_blocks) {
    if (!decode_down_group_ok(a.d) || !a.contrib || (a.n_layers != 1 && !a.groups.group) || a.n_tokens > rk::kMaxTokens) return cudaErrorInvalidValue;
    if (a.n_tokens == 0) return cudaSuccess;
    if (type == QKM_TYPE_Q6_K) return a.n_layers == 1 ? group_launch<true, true>(L, a, n_blocks) : group_launch<true, false>(L, a, n_blocks);
    if (type != QKM_TYPE_IQ4_XS || !a.lut) return cudaErrorInvalidValue;
    return a.n_layers == 1 ? group_launch<false, true>(L, a, n_blocks) : group_launch<false, false>(L, a, n_blocks);
}

}  // namespace qkm
