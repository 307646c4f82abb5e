// Down projection of the fused decode sequence for shapes whose (slot, 256-column block) pairs are not exactly the sixteen
// warps of the two specialised kernels (n_ff = 512 with eight slots): any number of slots up to twenty pairs (ten slots),
// IQ4_XS or Q6_K, n_ff = 512:  y[t] = sum_s w_s * D[ids_s] . h[t][s]  +  w_shared * DS . h[t][n_used].
//
// Replaces moe_down_iq4.comp / moe_down_q6k.comp + moe_down_q8b.comp + the "routed + shared" add for those shapes.  Same
// organisation and arithmetic as the specialised kernels (see qkm_dec_down.cu, qkm_dec_down_q6k.cu): a unit is (token, 16 output rows)
// and belongs to a block with a warp per pair; the pairs' sums are added in order.  What is different: the number of warps is
// the launch's, a warp also takes the 32-column block of the shared matrix that has its number, and it encodes the 32 values of the
// shared row for that on its own.
//
// Bound by instruction issue like the specialised ones; before, these shapes took the f32 kernels that dequantise every weight for
// every token.  512 experts, top 10, IQ4_XS, 3 tokens: the whole layer 353 -> 42 us, of which this kernel 12.
#include "qkm_dec_tiles.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"
#include "qkm_tiles.cuh"

namespace qkm {

namespace da {
constexpr uint32_t kMaxWarps = 20;                  // (slot, column block) pairs, and at least the n_ff / 32 shared blocks
constexpr int kShBlock = 544;                       // one Q8_0 block column of a 16-row tile: d, quants
constexpr int kChunk = 4;                           // tiles between two block-wide sums
constexpr uint32_t kTab = 0x10000u, kTabBytes = 0x10000u, kHigh = kTab + kTabBytes;   // IQ4_XS table image, absolute shared-window address
template <bool Q6> struct Cfg {
    static constexpr int kTile = Q6 ? kTileQ6 : kTileIq4, kStage = kTile + kShBlock;
    static constexpr uint32_t kStages = 2, kRing = kStages * kStage;      // 7808, 5440
    static constexpr uint32_t kLow = 10;                                           // IQ4_XS: rings below the table, up against it; the others above
    static constexpr uint32_t kScratch = Q6 ? 1024 + kMaxWarps * kRing : kHigh + (kMaxWarps - kLow) * kRing;   // Q6_K: from the aligned start
    static constexpr uint32_t kEnd = kScratch + kMaxWarps * 1024 + 2 * kMaxWarps * kChunk * 16 * 4;
    static constexpr uint32_t kDyn = Q6 ? kEnd + 128 : kEnd - 1024;                // the first KB of the window is the system's
};
static_assert(Cfg<true>::kDyn <= 231000 && Cfg<false>::kDyn <= 231000, "with the static part at most 227 KB");
}  // namespace da

template <bool Q6>
__global__ void __launch_bounds__(da::kMaxWarps * 32, 1)
decode_down_any_kernel(const __grid_constant__ DownDecodeArgs a) {
    using C = da::Cfg<Q6>;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) unsigned long long s_bar[da::kMaxWarps * C::kStages + 1];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    const qkm_dims d = a.d;
    const uint32_t n_slots = d.n_used + 1, n_warps = blockDim.x >> 5;
    constexpr uint32_t KB = 2;   // n_ff = 512
    const uint32_t RT = d.n_embd / 16, slot = warp / KB, kb = warp - slot * KB;
    const bool has_tile = a.layer[0].w != nullptr && slot < d.n_used, has_sh = a.layer[0].sh != nullptr && warp < d.n_ff / 32;
    const uint32_t win0 = smem_addr(smem_raw), base = Q6 ? (win0 + 127u) & ~127u : 0u;
    if (!Q6) {   // the fixed addresses must lie inside the dynamic area
        uint32_t dyn_size;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_size));
        if (win0 > da::kTab - C::kLow * C::kRing || win0 + dyn_size < C::kEnd) {
            if (tid == 0) atomicExch(a.status, (uint32_t)kStatusBadLayout);
            return;
        }
    }
    const uint32_t ring = Q6 ? base + 1024 + warp * C::kRing : warp < C::kLow ? da::kTab - (warp + 1) * C::kRing : da::kHigh + (warp - C::kLow) * C::kRing;
    const uint32_t my_dig = base + C::kScratch + warp * 1024;
    uint8_t* dig = smem_raw + (my_dig - win0);
    float* red = reinterpret_cast<float*>(smem_raw + (base + C::kScratch + da::kMaxWarps * 1024 - win0));   // [2 buffers][warps][kChunk tiles][16 rows]
    const uint32_t my_bar = smem_addr(&s_bar[warp * C::kStages]), bar_tab = smem_addr(&s_bar[da::kMaxWarps * C::kStages]);
    bool timed_out = false;

    if (lane == 0) {
        for (uint32_t s = 0; s < C::kStages; ++s) mbar_init(my_bar + 8 * s, 1);
        if (warp == 0) mbar_init(bar_tab, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (!Q6 && tid == 0) {
        mbar_expect_tx(bar_tab, da::kTabBytes);
        for (uint32_t i = 0; i < 4; ++i) bulk_g2s(da::kTab + i * 16384u, a.lut + i * 16384u, 16384u, bar_tab);
    }

    const uint64_t tiles_total = (uint64_t)a.n_layers * a.n_tokens * RT;   // units: (layer, token, tile)
    const uint32_t u_lo = (uint32_t)(tiles_total * blockIdx.x / gridDim.x), u_hi = (uint32_t)(tiles_total * (blockIdx.x + 1) / gridDim.x);

    // producer cursor; lane 0 only
    uint32_t p_u = u_lo, p_tok = u_lo / RT, p_rt = u_lo - p_tok * RT;
    bool p_new_tok = true;
    const uint8_t *p_src = nullptr, *p_sh = nullptr;   // next tile of expert ids[slot]; block column `warp` of the next shared tile
    auto issue = [&](uint32_t stage) {
        if (p_u >= u_hi || timed_out || !(has_tile || has_sh)) return;
        if (p_new_tok) {
            p_new_tok = false;
            const uint32_t l = layer_of(a, p_tok);
            if (has_tile) p_src = a.layer[l].w + (((size_t)min(__ldcg(&layer_sel(a, l)[p_tok - l * a.n_tokens].ids[slot]), d.n_expert - 1) * KB + kb) * RT + p_rt) * C::kTile;
            if (has_sh) p_sh = a.layer[l].sh + ((size_t)(warp >> 3) * RT + p_rt) * kTileQ8 + da::kShBlock * (warp & 7u);
        }
        const uint32_t bar = my_bar + 8 * stage, dst = ring + stage * C::kStage;
        mbar_expect_tx(bar, (has_tile ? C::kTile : 0) + (has_sh ? da::kShBlock : 0));
        if (has_tile) { bulk_g2s(dst, p_src, C::kTile, bar); p_src += C::kTile; }
        if (has_sh) { bulk_g2s(dst + C::kTile, p_sh, da::kShBlock, bar); p_sh += kTileQ8; }
        ++p_u;
        if (++p_rt == RT) { p_rt = 0; ++p_tok; p_new_tok = true; }
    };
    if (lane == 0)
        for (uint32_t s = 0; s < C::kStages; ++s) issue(s);
    // The first weight tiles are on their way (they depend on the selection only, which was final
    // before the gate/up kernel released this one); h is that kernel's output.
    pdl_wait();
    pdl_trigger();
    if (!Q6 && !mbar_wait_bounded(bar_tab, 0)) timed_out = true;   // every thread observes the table's arrival itself

    uint32_t cnt = 0, buf = 0;
    float w_s = 0.f, w_sh = 0.f;   // routing weight x plane scale of this warp's slot, and of its shared block
    uint32_t b0[8], b1[8], hb0 = 0, hb1 = 0;   // B operands: the slot's digits, the shared block's
#pragma unroll
    for (int j = 0; j < 8; ++j) { b0[j] = 0; b1[j] = 0; }
    // digit weights of C columns 2t, 2t+1: digits in columns 0..3, with Q6_K's tiles in 0..3 and 4..7 (its even and odd 16-column groups)
    const float dw0 = t == 0 ? 1.f : (t == 1 ? 16384.f : 0.f), dw1 = dw0 * 128.f;
    const float dq0 = Q6 ? ((t & 1u) ? 16384.f : 1.f) : dw0, dq1 = dq0 * 128.f;
    const uint32_t i_off = 64 * g + piece_at(g, t), tab_c = da::kTab + lane * 4;

    uint32_t tok = u_lo / RT, rt = u_lo - tok * RT;
    bool new_tok = true;
    float* y = nullptr;            // the token's output row
    for (uint32_t u = u_lo; u < u_hi;) {
        if (new_tok) {   // block-uniform
            new_tok = false;
            const uint32_t l = layer_of(a, tok), lt = tok - l * a.n_tokens;   // layer, token of the layer
            const float* h = layer_h(a, l) + (size_t)lt * n_slots * d.n_ff;
            const qkm_sel* rec = layer_sel(a, l) + lt;
            y = a.y + l * a.y_stride + (size_t)lt * d.n_embd;
            if (has_tile) {   // 256 values of h[tok][slot] as digits (28-bit fixed point relative to their largest)
                const float* hs = h + slot * d.n_ff + 256 * kb + 8 * lane;
                const float4 v0 = *reinterpret_cast<const float4*>(hs), v1 = *reinterpret_cast<const float4*>(hs + 4);
                const float hv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
                float m = 0.f;
                bool bad = false;
#pragma unroll
                for (int i = 0; i < 8; ++i) { m = fmaxf(m, fabsf(hv[i])); bad |= !(fabsf(hv[i]) <= 3.0e38f); }
                m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));   // non-negative floats order like their bits
                const bool any_bad = __any_sync(0xFFFFFFFFu, bad);
                const int p = any_bad ? 0 : digit_exponent(m);
                const float up = ldexpf(1.0f, p);
                uint32_t dg[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) dg[i] = any_bad ? 0u : digits4(__float2int_rn(hv[i] * up));
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; ++j) {   // plane j of elements 8 lane .. 8 lane + 7; IQ4_XS in iq4_word's order (0, 2, 1, 3), Q6_K as they come
                    const uint32_t sel = 0x4040u + 0x1111u * j;   // byte j of a, byte j of b, twice
                    const uint32_t p0 = prmt_dec(dg[0], dg[Q6 ? 1 : 2], sel), p1 = prmt_dec(dg[Q6 ? 2 : 1], dg[3], sel);
                    const uint32_t p2 = prmt_dec(dg[4], dg[Q6 ? 5 : 6], sel), p3 = prmt_dec(dg[Q6 ? 6 : 5], dg[7], sel);
                    *reinterpret_cast<uint2*>(dig + 256 * j + 8 * lane) = make_uint2(prmt_dec(p0, p1, 0x5410u), prmt_dec(p2, p3, 0x5410u));
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (Q6) {   // lanes g < 4: digit g of the first 16-column group in b0; g >= 4: digit g - 4 of the second in b1
                        const uint32_t v = lds32(my_dig + (g & 3u) * 256 + 32 * j + 16 * (g >> 2) + 4 * t);
                        b0[j] = g < 4 ? v : 0u;
                        b1[j] = g < 4 ? 0u : v;
                    } else {    // lanes g < 4: digit g of elements 8t .. 8t+7
                        const uint2 v = lds64(my_dig + (g & 3u) * 256 + 32 * j + 8 * t);
                        b0[j] = g < 4 ? v.x : 0u;
                        b1[j] = g < 4 ? v.y : 0u;
                    }
                }
                w_s = rec->w[slot] * (any_bad ? __int_as_float(0x7FC00000) : ldexpf(Q6 ? 0.25f : 1.0f, -p));
            }
            if (has_sh) {   // 32 values of the shared row, one a lane; digit g of elements 4t.. and 16 + 4t.. by shuffles
                const float hv = h[d.n_used * d.n_ff + 32 * warp + lane];
                const bool any_bad = __any_sync(0xFFFFFFFFu, !(fabsf(hv) <= 3.0e38f));
                const float m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(fabsf(hv))));
                const int p = any_bad ? 0 : digit_exponent(m);
                const uint32_t dg = any_bad ? 0u : digits4(__float2int_rn(hv * ldexpf(1.0f, p)));
                uint32_t e[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) e[i] = __shfl_sync(0xFFFFFFFFu, dg, (i >> 2) * 16 + 4 * t + (i & 3));
                const uint32_t sel = 0x4040u + 0x1111u * (g & 3u);
                hb0 = g < 4 ? prmt_dec(prmt_dec(e[0], e[1], sel), prmt_dec(e[2], e[3], sel), 0x5410u) : 0u;
                hb1 = g < 4 ? prmt_dec(prmt_dec(e[4], e[5], sel), prmt_dec(e[6], e[7], sel), 0x5410u) : 0u;
                w_sh = rec->w_shared * (any_bad ? __int_as_float(0x7FC00000) : ldexpf(1.0f, -p));
            }
        }
        const uint32_t n_c = min((uint32_t)da::kChunk, min(u_hi - u, RT - rt));   // tiles of this chunk
#pragma unroll 1
        for (uint32_t i = 0; i < n_c; ++i, ++cnt) {
            const uint32_t stage = cnt & 1u, tb = ring + stage * C::kStage, qb = tb + C::kTile;
            static_assert(C::kStages == 2, "");
            float va = 0.f, vb = 0.f;
            if (has_tile || has_sh) {
                if (!mbar_wait_bounded(my_bar + 8 * stage, (cnt >> 1) & 1u)) timed_out = true;
            }
            if (has_tile) {
                int acc[4] = {0, 0, 0, 0};
                float da, db;
                if (Q6) {
                    // the eight scales of this lane's groups (even groups for t < 2, odd for t >= 2), rows g and g+8
                    const uint2 scA = lds64(tb + 16 * g + 8 * (t >> 1)), scB = lds64(tb + 16 * (g + 8) + 8 * (t >> 1));
                    const uint4 hA = lds128(tb + 2304 + i_off), hB = lds128(tb + 2816 + i_off);
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
                            int c[4];
                            mma_s8_first(c, a0[qd], a1[qd], a2[qd], a3[qd], b0[j], b1[j]);
                            const uint32_t sel = 0x8880u + (uint32_t)(j & 3) * 0x1111u;   // byte j & 3, sign-extended
                            const int sa = (int)prmt_dec(hf ? scA.y : scA.x, 0u, sel), sb = (int)prmt_dec(hf ? scB.y : scB.x, 0u, sel);
                            acc[0] += sa * c[0]; acc[1] += sa * c[1]; acc[2] += sb * c[2]; acc[3] += sb * c[3];
                        }
                    }
                    const uint32_t d2 = lds32(tb + 3328 + 2 * (g & ~1u)), d8 = lds32(tb + 3328 + 16 + 2 * (g & ~1u));
                    da = f16_bits_to_f32((d2 >> (16 * (g & 1u))) & 0xFFFFu); db = f16_bits_to_f32((d8 >> (16 * (g & 1u))) & 0xFFFFu);
                } else {
                    const uint4 hd = lds128(tb + 16 * g);   // row g (x: d | scales_h << 16, y: scales_l), row g+8 (z, w)
                    uint32_t ea, oa, eb, ob;
                    iq4_scales(hd.y, hd.x >> 16, ea, oa);
                    iq4_scales(hd.w, hd.z >> 16, eb, ob);
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
                            mma_s8_first(c, a0, a1, a2, a3, b0[sb], b1[sb]);
                            const uint32_t sel = 0x8880u + (uint32_t)(sb >> 1) * 0x1111u;   // byte sb / 2, sign-extended
                            const int la = (int)prmt_dec((sb & 1) ? oa : ea, 0u, sel), lb = (int)prmt_dec((sb & 1) ? ob : eb, 0u, sel);
                            acc[0] += la * c[0]; acc[1] += la * c[1]; acc[2] += lb * c[2]; acc[3] += lb * c[3];
                        }
                    }
                    da = f16_bits_to_f32(hd.x & 0xFFFFu); db = f16_bits_to_f32(hd.z & 0xFFFFu);
                }
                va = w_s * (da * ((float)acc[0] * dq0 + (float)acc[1] * dq1));
                vb = w_s * (db * ((float)acc[2] * dq0 + (float)acc[3] * dq1));
            }
            if (has_sh) {
                const uint2 qa = lds64(qb + 32 + lane * 8), qc = lds64(qb + 32 + 256 + lane * 8);   // rows g, g+8: qs[4t..4t+3], qs[16+4t..16+4t+3]
                int c[4];
                mma_s8_first(c, qa.x, qc.x, qa.y, qc.y, hb0, hb1);
                const uint32_t dw = lds32(qb + 2 * (g & ~1u)), dw8 = lds32(qb + 2 * (8 + (g & ~1u)));
                va += w_sh * (f16_bits_to_f32((dw >> (16 * (g & 1u))) & 0xFFFFu) * ((float)c[0] * dw0 + (float)c[1] * dw1));
                vb += w_sh * (f16_bits_to_f32((dw8 >> (16 * (g & 1u))) & 0xFFFFu) * ((float)c[2] * dw0 + (float)c[3] * dw1));
            }
            va += __shfl_xor_sync(0xFFFFFFFFu, va, 1); vb += __shfl_xor_sync(0xFFFFFFFFu, vb, 1);
            if (Q6) { va += __shfl_xor_sync(0xFFFFFFFFu, va, 2); vb += __shfl_xor_sync(0xFFFFFFFFu, vb, 2); }
            stage_read();
            __syncwarp();
            if (lane == 0) issue(stage);
            if (t == 0) {
                float* r = red + ((buf * da::kMaxWarps + warp) * da::kChunk + i) * 16;
                r[g] = va; r[g + 8] = vb;
            }
        }
        __syncthreads();
        if (tid < 16 * n_c) {
            const uint32_t i = tid >> 4, r = tid & 15u;   // tile i of the chunk
            float sum = 0.f;
            for (uint32_t w = 0; w < n_warps; w += 2)   // slot order; a slot's two column blocks first (half as many roundings in a chain)
                sum += red[((buf * da::kMaxWarps + w) * da::kChunk + i) * 16 + r] + red[((buf * da::kMaxWarps + w + 1) * da::kChunk + i) * 16 + r];
            y[(rt + i) * 16 + r] = sum;
        }
        buf ^= 1u;
        u += n_c;
        rt += n_c;
        if (rt == RT) { rt = 0; ++tok; new_tok = true; }
    }
    if (timed_out && lane == 0) atomicExch(a.status, (uint32_t)kStatusWaitTimeout);
}

// a warp per (slot, column block), at least one per 32 columns of the shared matrix
static uint32_t any_warps(const qkm_dims& d) {
    const uint32_t pairs = d.n_used * (d.n_ff / 256), sh = d.n_ff / 32;
    return pairs > sh ? pairs : sh;
}
bool decode_down_any_ok(const qkm_dims& d) {
    return d.n_ff == 512 && any_warps(d) <= da::kMaxWarps && d.n_embd % 32 == 0;
}
template <bool Q6>
static cudaError_t any_launch(const Launch& L, const DownDecodeArgs& a, uint32_t n_blocks) {
    const size_t smem = da::Cfg<Q6>::kDyn;
    if (const cudaError_t e = allow_dynamic_smem<decode_down_any_kernel<Q6>>((int)smem)) return e;
    const cudaError_t e = launch_kernel(L, decode_down_any_kernel<Q6>, dim3(n_blocks), dim3(any_warps(a.d) * 32), smem, a);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}
cudaError_t launch_decode_down_any(const Launch& L, const DownDecodeArgs& a, uint32_t type, uint32_t n_blocks) {
    if (!decode_down_any_ok(a.d)) return cudaErrorInvalidValue;
    if (a.n_tokens == 0) return cudaSuccess;
    if (type == QKM_TYPE_Q6_K || a.layer[0].w == nullptr) return any_launch<true>(L, a, n_blocks);
    if (type != QKM_TYPE_IQ4_XS || !a.lut) return cudaErrorInvalidValue;
    return any_launch<false>(L, a, n_blocks);
}

}  // namespace qkm
