// Ranking of f64 router logits (one warp per token) and the list of work that the kernels which go by expert walk, for decode-sized
// batches of one or more layers.
//
// The router kernel ranks a group of tokens in the block that finishes the group's logits last.  Of layers that go together, the block
// that ranks a layer's last tokens groups its pairs for the kernels behind.  A layer on its own is grouped by each block of those kernels
// for itself: one block at the router's end, the lists' way through the L2 and their reads there are a chain that nothing hides, 3 to 6 us of
// a layer (a decode step of 256 experts, top 8: 1 token 27.0 -> 23.6 us, 16: 80.9 -> 71.9, 64: 182.4 -> 168.4; of 512, top 10: 3 tokens 42.6 ->
// 39.7, 64: 252.5 -> 242.9; with the kernels' forms for one layer).
//
// Rules (the reference's): top n_used by raw logit, lowest id on ties
// (shaders/moe_select_256.comp:60-61), non-finite logits at the floor -3.4e38
// (shaders/moe_select.comp:28-34), softmax over the selected only
// (shaders/moe_select.comp:71-76); pairs grouped as shaders/moe_group_pairs.comp:19-50 does,
// ascending token inside an expert.
#pragma once

#include "qkm_kernels.h"

namespace qkm {

namespace rk {
constexpr uint32_t kMaxTokens = 64, kMaxExperts = 512;
constexpr uint32_t kMaxGroups = (kMaxTokens * 16 + kMaxExperts) / 2 + kMaxTokens / 2;   // of a layer: 800
constexpr float kFloor = -3.4e38f;
}  // namespace rk

// What a lane of the ranking warp knows of the token's selection: the id in place `lane` (0 past n_used) and its logit's key.
struct Ranked { uint32_t id, hi, lo; };

// Ranks one token, by one warp.  lt: its n_expert f64 logits in global memory (complete and visible to this block).
template <bool WIDE>   // WIDE: more than 256 experts (two sorted lists of eight keys per lane instead of one)
__device__ __forceinline__ Ranked rank_token_impl(const double* __restrict__ lt, const qkm_dims& d) {
    const uint32_t lane = threadIdx.x & 31u;
    // Ranking with integer keys: an f64 maps to a 64-bit unsigned key whose order is the value's
    // (sign bit flipped for positives, all bits for negatives; -0 is turned into +0 first so the
    // two tie).  One warp per token.  A lane sorts its (up to 16) keys once, as two lists of
    // eight, with a sorting network; then each of the n_used rounds compares only list heads:
    // the warp finds the largest head with three hardware reductions (high word, low word among
    // the lanes that hold it, lowest id among those - lowest id wins ties) and the winning lane
    // pops its list.  Integer arithmetic only: a serial chain of f64 compares and selects is latency-
    // bound (f64 adds and multiplies run at half the f32 rate here, f32<->f64 conversions at an eighth).
    const uint32_t per_lane = (d.n_expert + 31) / 32;   // <= 16
    const unsigned long long kFloorBits = (unsigned long long)__double_as_longlong((double)rk::kFloor);
    constexpr int NK = WIDE ? 16 : 8;
    uint32_t khi[NK], klo[NK], kid[NK];
#pragma unroll
    for (int j = 0; j < NK; ++j) {
        const uint32_t e = lane + 32u * j;
        khi[j] = 0; klo[j] = 0; kid[j] = e;   // key 0 is below every real key
        if ((uint32_t)j < per_lane && e < d.n_expert) {
            unsigned long long b = (unsigned long long)__ldcg(reinterpret_cast<const long long*>(lt) + e);
            if (((b >> 52) & 0x7FFull) == 0x7FFull) b = kFloorBits;      // NaN, +-Inf -> the floor
            if (b == 0x8000000000000000ull) b = 0ull;                    // -0 ties with +0
            const unsigned long long k = (b >> 63) ? ~b : (b | 0x8000000000000000ull);
            khi[j] = (uint32_t)(k >> 32); klo[j] = (uint32_t)k;
        }
    }
    // compare-exchange: afterwards position p holds the entry that ranks first (key descending, id ascending)
    auto cex = [&](int p, int q) {
        const bool swap = khi[q] > khi[p] || (khi[q] == khi[p] && (klo[q] > klo[p] || (klo[q] == klo[p] && kid[q] < kid[p])));
        const uint32_t h = swap ? khi[q] : khi[p], l = swap ? klo[q] : klo[p], i_ = swap ? kid[q] : kid[p];
        khi[q] = swap ? khi[p] : khi[q]; klo[q] = swap ? klo[p] : klo[q]; kid[q] = swap ? kid[p] : kid[q];
        khi[p] = h; klo[p] = l; kid[p] = i_;
    };
#pragma unroll
    for (int o = 0; o < NK; o += 8) {   // Batcher's 19-exchange network on each list of eight
        cex(o + 0, o + 1); cex(o + 2, o + 3); cex(o + 4, o + 5); cex(o + 6, o + 7);
        cex(o + 0, o + 2); cex(o + 1, o + 3); cex(o + 4, o + 6); cex(o + 5, o + 7);
        cex(o + 1, o + 2); cex(o + 5, o + 6);
        cex(o + 0, o + 4); cex(o + 1, o + 5); cex(o + 2, o + 6); cex(o + 3, o + 7);
        cex(o + 2, o + 4); cex(o + 3, o + 5);
        cex(o + 1, o + 2); cex(o + 3, o + 4); cex(o + 5, o + 6);
    }
    uint32_t my_id = 0, my_hi = 0, my_lo = 0;
    for (uint32_t i = 0; i < d.n_used; ++i) {
        // this lane's best remaining entry: the better of the two list heads
        bool second = false;
        if (WIDE) second = khi[NK - 8] > khi[0] || (khi[NK - 8] == khi[0] && (klo[NK - 8] > klo[0] || (klo[NK - 8] == klo[0] && kid[NK - 8] < kid[0])));
        const uint32_t bh = second ? khi[NK - 8] : khi[0], bl = second ? klo[NK - 8] : klo[0], bi = second ? kid[NK - 8] : kid[0];
        const uint32_t mh = __reduce_max_sync(0xFFFFFFFFu, bh);
        const uint32_t ml = __reduce_max_sync(0xFFFFFFFFu, bh == mh ? bl : 0u);
        const bool cand = bh == mh && bl == ml && (bh | bl) != 0u;
        const uint32_t id = __reduce_min_sync(0xFFFFFFFFu, cand ? bi : 0xFFFFFFFFu);
        const bool won = cand && id == bi;
        const bool pop0 = won && !second, pop8 = won && second;
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            if (pop0) { khi[j] = khi[j + 1]; klo[j] = klo[j + 1]; kid[j] = kid[j + 1]; }
            if (WIDE && pop8) { khi[NK - 8 + j] = khi[NK - 7 + j]; klo[NK - 8 + j] = klo[NK - 7 + j]; kid[NK - 8 + j] = kid[NK - 7 + j]; }
        }
        if (pop0) { khi[7] = 0; klo[7] = 0; }
        if (WIDE && pop8) { khi[NK - 1] = 0; klo[NK - 1] = 0; }
        if (lane == i) { my_id = id; my_hi = mh; my_lo = ml; }
    }
    return Ranked{lane < d.n_used ? min(my_id, d.n_expert - 1) : 0u, my_hi, my_lo};
}
__device__ __forceinline__ Ranked rank_token(const double* __restrict__ lt, const qkm_dims& d) {
    return d.n_expert > 256 ? rank_token_impl<true>(lt, d) : rank_token_impl<false>(lt, d);
}
// Writes the ids, weights, route_done and padding of the token's record (w_shared is not touched).
__device__ __forceinline__ void rank_store(const Ranked& r, qkm_sel& sel, const qkm_dims& d) {
    const uint32_t lane = threadIdx.x & 31u;
    // Softmax over the selected: the differences to the top logit are formed in f64 (one
    // subtraction), the exponentials and their normalisation in f32 (relative error ~3e-7
    // against the reference's f64 weights).
    const unsigned long long k = ((unsigned long long)r.hi << 32) | r.lo;
    const unsigned long long b = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
    const double my_val = __longlong_as_double((long long)b);
    const double top = __shfl_sync(0xFFFFFFFFu, my_val, 0);
    const float wv = lane < d.n_used ? expf((float)(my_val - top)) : 0.f;
    float sum = wv;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);   // lanes 0..15
    if (lane < 16) {
        sel.ids[lane] = r.id;
        sel.w[lane] = lane < d.n_used ? wv / sum : 0.f;
    } else if (lane == 16) {
        sel.route_done = 0;
    } else if (lane < 23) {
        sel.pad[lane - 17] = 0.f;
    }
}

// ---- the flat list of (layer, group, 16-row tile) that the kernels which go by expert cut over their teams of warps ----
// Where each layer's groups begin in it, in the calling block's shared memory.
struct LayerCuts {
    uint32_t groups[kDecMaxLayers + 1];   // first group of each layer
    uint32_t cost[kDecMaxLayers + 1];     // and what the groups before it cost, in tiles of a routed group times its weight
};
// group `gi` of layer `l`
__device__ __forceinline__ const DecodeGroup* decode_group_at(const DecodeGroups& g, uint32_t n_tokens, uint32_t n_used, uint32_t l, uint32_t gi) {
    return g.group + (size_t)l * n_tokens * (n_used + 1) + gi;
}
// By one warp: a routed group costs `routed`, a shared one `shared` (relative, per tile).
__device__ __forceinline__ void layer_cuts(LayerCuts& c, const DecodeGroups& g, uint32_t n_tokens, uint32_t n_layers, uint32_t routed, uint32_t shared) {
    const uint32_t lane = threadIdx.x & 31u, n_shared = (n_tokens + 1) / 2;
    uint32_t groups = 0, cost = 0;   // of the layers before
    if (lane == 0) { c.groups[0] = 0; c.cost[0] = 0; }
    for (uint32_t l0 = 0; l0 < n_layers; l0 += 32) {
        uint32_t n = 0;
        if (l0 + lane < n_layers) n = __ldcg(g.count + l0 + lane);
        uint32_t k = l0 + lane < n_layers ? (n - n_shared) * routed + n_shared * shared : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up_n = __shfl_up_sync(0xFFFFFFFFu, n, o), up_k = __shfl_up_sync(0xFFFFFFFFu, k, o);
            if (lane >= (uint32_t)o) { n += up_n; k += up_k; }
        }
        if (l0 + lane < n_layers) { c.groups[l0 + lane + 1] = groups + n; c.cost[l0 + lane + 1] = cost + k; }
        groups += __shfl_sync(0xFFFFFFFFu, n, 31);
        cost += __shfl_sync(0xFFFFFFFFu, k, 31);
    }
}
// ---- a layer's (token, slot) pairs grouped by expert ----
// token t chose expert e in place `slot`
__device__ __forceinline__ void choose(unsigned long long* s_mask, uint16_t* s_ids, uint32_t t, uint32_t slot, uint32_t e) {
    s_ids[t * 16 + slot] = (uint16_t)e;
    atomicOr(reinterpret_cast<uint32_t*>(s_mask) + 2 * e + (t >> 5), 1u << (t & 31u));   // bit t of the expert's 64
}
// By a block of THREADS: writes the layer's groups, returns how many.  s_ids[t][16]: the layer's selection; s_mask: the tokens that chose each
// expert; np: pairs in them (T * n_used, or none: the shared expert's groups only); s_first, s_sum: scratch for an entry an
// expert and a warp.  groups: in global or in the block's shared memory.
template <uint32_t THREADS>
__device__ __forceinline__ uint32_t group_pairs(DecodeGroup* groups, uint32_t* s_first, uint32_t* s_sum, const uint16_t* s_ids, const unsigned long long* s_mask,
                                                uint32_t n_used, uint32_t np, uint32_t T, uint32_t layer) {
    constexpr int PER = rk::kMaxExperts / THREADS;
    static_assert(PER * THREADS == rk::kMaxExperts, "whole experts a thread");
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, n_shared = (T + 1) / 2;
    uint32_t c[PER], v = 0;   // tokens of this thread's experts; groups up to the last one
#pragma unroll
    for (int h = 0; h < PER; ++h) { c[h] = (uint32_t)__popcll(s_mask[PER * tid + h]); v += (c[h] + 1) / 2; }
    const uint32_t n = v;
#pragma unroll
    for (int i = 1; i < 32; i <<= 1) {
        const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, v, i);
        if (lane >= (uint32_t)i) v += up;
    }
    if (lane == 31) s_sum[warp] = v;
    __syncthreads();
    uint32_t base = 0, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < THREADS / 32; ++w) { if (w < warp) base += s_sum[w]; total += s_sum[w]; }
    uint32_t first = base + v - n;
#pragma unroll
    for (int h = 0; h < PER; ++h) {
        const uint32_t e = PER * tid + h;
        s_first[e] = first;
        for (uint32_t i = 0; 2 * i < c[h]; ++i, ++first) {
            groups[first].head = DecodeGroup::make_head(e, min(2u, c[h] - 2 * i), 0);
            groups[first].layer = layer;
        }
    }
    // every token is one of the shared expert's pairs
    for (uint32_t i = tid; i < n_shared; i += THREADS)
        groups[total + i] = DecodeGroup{DecodeGroup::make_head(0, min(2u, T - 2 * i), 1), {((2 * i) << 4) | n_used, (min(2 * i + 1, T - 1) << 4) | n_used}, layer};
    __syncthreads();
    // a pair's rank inside its expert is the number of lower tokens that chose the expert
    for (uint32_t p = tid; p < np; p += THREADS) {
        const uint32_t t = p / n_used, s = p - t * n_used, e = s_ids[t * 16 + s];
        const uint32_t r = (uint32_t)__popcll(s_mask[e] & ((1ull << t) - 1ull));
        groups[s_first[e] + r / 2].pair[r & 1u] = (t << 4) | s;
    }
    return total + n_shared;
}
// Working set of own_groups, dead behind it.
struct OwnScratch {
    unsigned long long mask[rk::kMaxExperts];
    uint32_t first[rk::kMaxExperts], sum[rk::kMaxExperts / 32];
    uint16_t ids[rk::kMaxTokens * 16];
};
// A layer on its own: the block's list of its groups, and the list's cuts, from the tokens' records (NULL: the shared expert's
// groups only).  By a block of THREADS with S.mask zero; ends with a barrier.
template <uint32_t THREADS>
__device__ __forceinline__ void own_groups(OwnScratch& S, DecodeGroup* list, LayerCuts& cuts, const qkm_sel* sel, const qkm_dims& d, uint32_t T, uint32_t routed, uint32_t shared) {
    constexpr uint32_t PER = rk::kMaxTokens * 16 / THREADS;
    uint32_t id[PER];
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
        const uint32_t i = threadIdx.x + k * THREADS;
        if (sel && i < T * 16) id[k] = __ldcg(&sel[i >> 4].ids[i & 15u]);
    }
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
        const uint32_t i = threadIdx.x + k * THREADS;
        if (sel && i < T * 16 && (i & 15u) < d.n_used) choose(S.mask, S.ids, i >> 4, i & 15u, min(id[k], d.n_expert - 1));
    }
    __syncthreads();
    const uint32_t n = group_pairs<THREADS>(list, S.first, S.sum, S.ids, S.mask, d.n_used, sel ? T * d.n_used : 0, T, 0), n_shared = (T + 1) / 2;
    if (threadIdx.x == 0) { cuts.groups[0] = 0; cuts.cost[0] = 0; cuts.groups[1] = n; cuts.cost[1] = (n - n_shared) * routed + n_shared * shared; }
    __syncthreads();
}
// A place in the list: layer, group of the layer, tile of the group.  `tiles` tiles a group.
struct ListPlace {
    uint32_t l, gi, rt;
    __device__ __forceinline__ void next_group(const LayerCuts& c) {
        if (++gi == c.groups[l + 1] - c.groups[l]) { gi = 0; ++l; }
    }
};
// Division by a number known before the kernel waits for the one ahead of it: one multiplication and a correction of at most one behind the
// wait (x < 2^32; the factor 2^32 / d is short by less than one, or by one where d divides 2^32).
struct Divisor {
    uint32_t d, m;
    __device__ __forceinline__ explicit Divisor(uint32_t by) : d(by), m(0xFFFFFFFFu / by) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
        const uint32_t q = __umulhi(x, m);
        return q + (x - q * d >= d ? 1u : 0u);
    }
};
// The warp's share of the list when it is cut into by_parts.d equal costs: its first place, and in `n` its tiles.  Even lanes
// look for the share's begin, odd ones for its end.  (A list's cost in tiles fits 32 bits: at most 768 rows.)
__device__ __forceinline__ ListPlace list_share(const LayerCuts& c, uint32_t n_tokens, uint32_t n_layers, const Divisor& by_tiles, uint32_t routed,
                                                const Divisor& by_shared, uint32_t part, const Divisor& by_parts, uint32_t& n) {
    const uint32_t tiles = by_tiles.d, cut = part + (threadIdx.x & 1u), total = c.cost[n_layers] * tiles, q = by_parts(total);
    const uint32_t want = q * cut + by_parts((total - q * by_parts.d) * cut);   // total * cut / parts; in tiles times weight
    uint32_t l = 0, last = n_layers - 1;   // the last layer that does not begin after `want`
    while (l < last) {
        const uint32_t m = (l + last + 1) / 2;
        if (c.cost[m] * tiles <= want) l = m;
        else last = m - 1;
    }
    const uint32_t n_groups = c.groups[l + 1] - c.groups[l], n_routed = n_groups - (n_tokens + 1) / 2, left = want - c.cost[l] * tiles, r = n_routed * tiles * routed;
    const uint32_t t = min(left <= r ? left / routed : n_routed * tiles + by_shared(left - r), n_groups * tiles);
    const uint32_t at = c.groups[l] * tiles + t, gi = by_tiles(t);
    n = __shfl_sync(0xFFFFFFFFu, at, 1) - __shfl_sync(0xFFFFFFFFu, at, 0);
    return ListPlace{__shfl_sync(0xFFFFFFFFu, l, 0), __shfl_sync(0xFFFFFFFFu, gi, 0), __shfl_sync(0xFFFFFFFFu, t - gi * tiles, 0)};
}

}  // namespace qkm
