// Selection of batched routing: top n_used experts of every token from its router logits, a warp per token.
//
// Replaces moe_select.comp / moe_select_256.comp and the selection half of moe_route_select[_hier].comp.  Rules kept: a
// non-finite logit ranks as -3.4e38 (moe_select.comp:28-34); among equal logits the lowest id ranks first
// (moe_select_256.comp:60-61); weights are a softmax over the selected logits only (moe_select.comp:71-76);
// w_shared = sigmoid(gate_inp_shexp . x) (moe_select.comp:36-45).
//
// The ids equal those of a router that accumulates in f64 (the CPU reference, src/main.cpp:1320-1341): f32 logits carry a provable
// error bound, every expert within twice the bound of the k-th largest is a candidate, and the candidates' logits are
// evaluated again in f64, which also gives the weights.  Small batches come with f64 logits, which are ranked as they are.
//
// Bound by the candidates' f64 dot products: a router row of 8 KB (F32) from the L2 and 2 x 2048 f32 -> f64 conversions
// (16 lanes a cycle and SM) or their like per candidate; x is converted once per token and kept in shared memory as f64.
// 4096 tokens, 256 experts, F32 router: 122 us before (a block per token, all of it in eight warps' lockstep, and twice the
// candidates) -> see below at the launch.
#include <math.h>

#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"

namespace qkm {

namespace sl {
constexpr float kFloor = -3.4e38f;
constexpr uint32_t kMaxExperts = 512;
constexpr uint32_t kListBytes = kMaxExperts * 10;   // keys (u64) and ids (u16) of the candidates
constexpr uint32_t kMaxWarps = 4;
}  // namespace sl

struct SelectArgs {
    const uint8_t* router;
    const void* logits;        // f64 [token][expert], or n_parts partial sums of f32 ones
    const float* norm2;        // n_norm values: their largest bounds |router row|^2
    const float* gis;
    const float* x;
    qkm_sel* sel;
    int8_t* xplanes;           // optional: x as digit planes [kb][digit][256], and their scale
    float* xscale;
    uint32_t* counts;          // optional: pairs per resident expert, added to; ranks[t * n_used + s] = a pair's number inside its expert
    uint32_t* ranks;
    size_t part_stride;
    uint32_t n_parts, n_norm, n_tokens, expert_first, expert_count;
    float eps_terms, eps_abs;
    qkm_dims d;
};

__device__ __forceinline__ unsigned long long key_of(double v) {   // order of the value; -0 ties with +0; non-finite: the floor
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if (((b >> 52) & 0x7FFull) == 0x7FFull) b = (unsigned long long)__double_as_longlong((double)sl::kFloor);
    if (b == 0x8000000000000000ull) b = 0ull;
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double value_of(unsigned long long k) {
    return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}
__device__ __forceinline__ uint32_t key32_of(float v) {   // likewise, f32
    v = (isnan(v) || isinf(v)) ? sl::kFloor : v + 0.0f;
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
// four consecutive router weights
template <int TYPE>
__device__ __forceinline__ float4 router4(const uint8_t* row, uint32_t u) {
    if (TYPE == QKM_TYPE_F32) return __ldg(reinterpret_cast<const float4*>(row) + u);
    const uint2 h = __ldg(reinterpret_cast<const uint2*>(row) + u);
    return make_float4(f16_bits_to_f32(h.x & 0xFFFFu), f16_bits_to_f32(h.x >> 16), f16_bits_to_f32(h.y & 0xFFFFu), f16_bits_to_f32(h.y >> 16));
}

template <int TYPE, bool EXACT>
__global__ void __launch_bounds__(sl::kMaxWarps * 32)
select_tokens_kernel(const SelectArgs a) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, t = blockIdx.x * (blockDim.x >> 5) + warp;
    const qkm_dims d = a.d;
    const uint32_t K4 = d.n_embd / 4;   // a multiple of 64
    // per warp: x as f64, elements 4u, 4u+1 of every four in one plane and 4u+2, 4u+3 in the other (no bank conflicts); the candidates
    const size_t per_warp = (EXACT ? 0 : (size_t)d.n_embd * 8) + sl::kListBytes;
    double2* x0 = reinterpret_cast<double2*>(smem_raw + warp * per_warp);
    double2* x1 = x0 + K4;
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem_raw + (warp + 1) * per_warp - sl::kListBytes);
    uint16_t* ids = reinterpret_cast<uint16_t*>(keys + sl::kMaxExperts);
    pdl_trigger();
    pdl_wait();
    if (t >= a.n_tokens) return;   // a warp on its own from here on
    const float4* xt = reinterpret_cast<const float4*>(a.x + (size_t)t * d.n_embd);

    // one pass over the row: f64 copy, |x|^2 and the largest |x|, the shared expert's gate
    float xs = 0.f, xm = 0.f;
    bool bad = false;
    double sg = 0.0;
#pragma unroll 8
    for (uint32_t u = lane; u < K4; u += 32) {
        const float4 v = xt[u], g = __ldg(reinterpret_cast<const float4*>(a.gis) + u);
        const double2 v0 = make_double2(v.x, v.y), v1 = make_double2(v.z, v.w);
        if (!EXACT) { x0[u] = v0; x1[u] = v1; }
        xs += v.x * v.x; xs += v.y * v.y; xs += v.z * v.z; xs += v.w * v.w;
        xm = fmaxf(fmaxf(xm, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        bad |= !(fabsf(v.x) <= 3.0e38f) || !(fabsf(v.y) <= 3.0e38f) || !(fabsf(v.z) <= 3.0e38f) || !(fabsf(v.w) <= 3.0e38f);
        sg += (double)g.x * v0.x; sg += (double)g.y * v0.y; sg += (double)g.z * v1.x; sg += (double)g.w * v1.y;
    }
    xs = warp_sum(xs);
    sg = warp_sum(sg);
    xm = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(xm)));   // non-negative floats order like their bits
    bad = __any_sync(0xFFFFFFFFu, bad);
    if (a.xplanes != nullptr) {
        const int p = digit_exponent(bad ? 0.f : xm);
        const float up = ldexpf(1.0f, p);
        for (uint32_t u = lane; u < K4; u += 32) {
            const float4 v = xt[u];
            const uint32_t e[4] = {bad ? 0u : digits4(__float2int_rn(v.x * up)), bad ? 0u : digits4(__float2int_rn(v.y * up)),
                                   bad ? 0u : digits4(__float2int_rn(v.z * up)), bad ? 0u : digits4(__float2int_rn(v.w * up))};
            uint32_t* q = reinterpret_cast<uint32_t*>(a.xplanes + (size_t)t * 4 * d.n_embd + (size_t)(u >> 6) * 1024 + 4 * (u & 63u));
#pragma unroll
            for (int j = 0; j < 4; ++j) {   // digit j of the four
                const uint32_t s = 0x4040u + 0x1111u * j;
                q[64 * j] = __byte_perm(__byte_perm(e[0], e[1], s), __byte_perm(e[2], e[3], s), 0x5410u);
            }
        }
        if (lane == 0) a.xscale[t] = bad ? __int_as_float(0x7FC00000) : ldexpf(1.0f, -p);
    }

    uint32_t nc = d.n_expert;   // candidates
    if (EXACT) {
        const double* lt = reinterpret_cast<const double*>(a.logits) + (size_t)t * d.n_expert;
        for (uint32_t e = lane; e < d.n_expert; e += 32) { keys[e] = key_of(__ldcg(lt + e)); ids[e] = (uint16_t)e; }
        __syncwarp();
    } else {
        constexpr int NK = sl::kMaxExperts / 32;
        const float* lt = reinterpret_cast<const float*>(a.logits) + (size_t)t * d.n_expert;
        float l[NK];
#pragma unroll
        for (int j = 0; j < NK; ++j) l[j] = 0.f;
#pragma unroll 2
        for (uint32_t p = 0; p < a.n_parts; ++p)   // partial sums over column ranges, added in order
#pragma unroll
            for (int j = 0; j < NK; ++j)
                if (lane + 32u * j < d.n_expert) l[j] += __ldcg(lt + p * a.part_stride + lane + 32 * j);
        float r2 = 0.f;
        for (uint32_t i = lane; i < a.n_norm; i += 32) r2 = fmaxf(r2, a.norm2[i]);
        r2 = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(r2)));
        // k-th largest: n_used rounds of the warp's largest key, each taking one lane's out
        uint32_t k[NK];
#pragma unroll
        for (int j = 0; j < NK; ++j) k[j] = lane + 32u * j < d.n_expert ? key32_of(l[j]) : 0u;
        uint32_t kth = 0;
#pragma unroll 1
        for (uint32_t i = 0; i < d.n_used; ++i) {
            uint32_t m = 0;
#pragma unroll
            for (int j = 0; j < NK; ++j) m = max(m, k[j]);
            kth = __reduce_max_sync(0xFFFFFFFFu, m);
            const uint32_t first = __ffs(__ballot_sync(0xFFFFFFFFu, m == kth)) - 1;
            bool out = lane == first;
#pragma unroll
            for (int j = 0; j < NK; ++j)
                if (out && k[j] == kth) { k[j] = 0; out = false; }
        }
        const float kv = __uint_as_float((kth & 0x80000000u) ? (kth ^ 0x80000000u) : ~kth);
        // |error of one logit| <= eps_terms * 2^-24 * sum|w_k x_k| <= that * |w| * |x|; two logits are compared.  A NaN threshold (NaN in
        // x) admits every expert.
        const float eps = 5.9604645e-8f * (a.eps_terms * sqrtf(r2) + a.eps_abs) * sqrtf(xs);
        const float thresh = kv - 2.1f * eps;
        nc = 0;
#pragma unroll
        for (int j = 0; j < NK; ++j) {
            const uint32_t e = lane + 32u * j;
            const float v = (isnan(l[j]) || isinf(l[j])) ? sl::kFloor : l[j];
            const uint32_t in = __ballot_sync(0xFFFFFFFFu, e < d.n_expert && !(v < thresh));
            if ((in >> lane) & 1u) ids[nc + __popc(in & ((1u << lane) - 1u))] = (uint16_t)e;   // ascending
            nc += __popc(in);
        }
        __syncwarp();
        const size_t rb = row_bytes(TYPE, d.n_embd);
        for (uint32_t c = 0; c < nc; c += 2) {   // two candidates at a time share the reads of x
            const uint8_t* ra = a.router + (size_t)ids[c] * rb;
            const uint8_t* rc = a.router + (size_t)ids[min(c + 1, nc - 1)] * rb;
            double s0 = 0.0, s1 = 0.0, q0 = 0.0, q1 = 0.0;
#pragma unroll 8
            for (uint32_t u = lane; u < K4; u += 32) {
                const float4 wa = router4<TYPE>(ra, u), wc = router4<TYPE>(rc, u);
                const double2 v0 = x0[u], v1 = x1[u];
                s0 += (double)wa.x * v0.x; s1 += (double)wa.y * v0.y; s0 += (double)wa.z * v1.x; s1 += (double)wa.w * v1.y;
                q0 += (double)wc.x * v0.x; q1 += (double)wc.y * v0.y; q0 += (double)wc.z * v1.x; q1 += (double)wc.w * v1.y;
            }
            const double s = warp_sum(s0 + s1), q = warp_sum(q0 + q1);
            if (lane == (c & 31u)) keys[c] = key_of(s);
            if (lane == ((c + 1) & 31u) && c + 1 < nc) keys[c + 1] = key_of(q);
        }
        __syncwarp();
    }
    // rank: every round takes the largest key, the lowest id (place in the list) among equal ones; lane c & 31 owns candidate c
    unsigned long long my_key = 0;
    uint32_t my_c = 0;
#pragma unroll 1
    for (uint32_t i = 0; i < d.n_used; ++i) {
        unsigned long long best = 0;
        uint32_t bc = 0xFFFFFFFFu;
        for (uint32_t c = lane; c < nc; c += 32)
            if (keys[c] > best) { best = keys[c]; bc = c; }
        const uint32_t bh = (uint32_t)(best >> 32), bl = (uint32_t)best;
        const uint32_t mh = __reduce_max_sync(0xFFFFFFFFu, bh);
        const uint32_t ml = __reduce_max_sync(0xFFFFFFFFu, bh == mh ? bl : 0u);
        const uint32_t c = __reduce_min_sync(0xFFFFFFFFu, bh == mh && bl == ml ? bc : 0xFFFFFFFFu);
        if (c == bc && c < nc) keys[c] = 0;   // below every real key
        if (lane == i) { my_key = ((unsigned long long)mh << 32) | ml; my_c = min(c, nc - 1); }
    }
    // lane i < n_used: softmax term of pick i
    const double v = value_of(my_key), top = __shfl_sync(0xFFFFFFFFu, v, 0);
    const double wv = lane < d.n_used ? exp(v - top) : 0.0;
    double sum = wv;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);   // lanes 0..15
    qkm_sel* s = a.sel + t;
    if (lane < 16) {
        const uint32_t id = lane < d.n_used ? min((uint32_t)ids[my_c], d.n_expert - 1) : 0u;
        s->ids[lane] = id;
        s->w[lane] = lane < d.n_used ? (float)(wv / sum) : 0.f;
        const uint32_t e = id - a.expert_first;
        if (a.counts != nullptr && lane < d.n_used) a.ranks[t * d.n_used + lane] = e < a.expert_count ? atomicAdd(a.counts + e, 1u) : 0u;
    } else if (lane == 16) {
        s->w_shared = (float)(1.0 / (1.0 + exp(-sg)));
        s->route_done = 0;
    } else if (lane < 23) {
        s->pad[lane - 17] = 0.f;
    }
}

template <int TYPE, bool EXACT>
static cudaError_t select_launch(const Launch& L, const SelectArgs& a) {
    const size_t per_warp = (EXACT ? 0 : (size_t)a.d.n_embd * 8) + sl::kListBytes;
    if (per_warp > 220 * 1024) return cudaErrorInvalidValue;
    if (const cudaError_t e = allow_dynamic_smem<select_tokens_kernel<TYPE, EXACT>>(220 * 1024)) return e;
    // as many warps a block as two blocks an SM allow, fewer for few tokens (they spread over the SMs)
    uint32_t warps = sl::kMaxWarps;
    while (warps > 1 && (warps * per_warp > 110 * 1024 || (a.n_tokens + warps - 1) / warps < 148u)) warps /= 2;
    const cudaError_t e = launch_kernel(Launch{L.stream, nullptr, true}, select_tokens_kernel<TYPE, EXACT>, dim3((a.n_tokens + warps - 1) / warps), dim3(warps * 32),
                                        warps * per_warp, a);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}
cudaError_t launch_select_tokens(const Launch& L, const qkm_dims& d, uint32_t router_type, const SelectIn& in, qkm_sel* sel, uint32_t n_tokens) {
    SelectArgs a{};
    a.router = (const uint8_t*)in.router; a.logits = in.logits; a.norm2 = in.norm2; a.n_norm = in.n_norm; a.gis = in.gis; a.x = in.x; a.sel = sel;
    a.xplanes = in.xplanes; a.xscale = in.xscale; a.counts = in.counts; a.ranks = in.ranks; a.part_stride = (size_t)n_tokens * d.n_expert; a.n_parts = in.n_parts;
    a.n_tokens = n_tokens; a.expert_first = in.expert_first; a.expert_count = in.expert_count; a.eps_terms = in.eps_terms; a.eps_abs = in.eps_abs; a.d = d;
    if (in.exact) return router_type == QKM_TYPE_F32 ? select_launch<QKM_TYPE_F32, true>(L, a) : select_launch<QKM_TYPE_F16, true>(L, a);
    return router_type == QKM_TYPE_F32 ? select_launch<QKM_TYPE_F32, false>(L, a) : select_launch<QKM_TYPE_F16, false>(L, a);
}

// ---- grouping ----------------------------------------------------------------------------------------------------
// Numbers the (token, slot) pairs of records that came from elsewhere inside their experts, as the selection does for its own.
__global__ void __launch_bounds__(256)
group_rank_kernel(const qkm_sel* __restrict__ sel, uint32_t np, uint32_t n_used, uint32_t n_expert, uint32_t expert_first, uint32_t expert_count,
                  uint32_t* __restrict__ counts, uint32_t* __restrict__ ranks) {
    const uint32_t p = blockIdx.x * 256 + threadIdx.x;
    if (p >= np) return;
    const uint32_t t = p / n_used, s = p - t * n_used, e = local_expert_of(sel[t].ids[s], n_expert, expert_first, expert_count);
    ranks[p] = e < expert_count ? atomicAdd(counts + e, 1u) : 0u;
}
cudaError_t launch_group_rank(const Launch& L, const qkm_dims& d, const qkm_sel* sel, uint32_t n_tokens, uint32_t expert_first, uint32_t expert_count,
                              uint32_t* counts, uint32_t* ranks) {
    const uint32_t np = n_tokens * d.n_used;
    if (np == 0) return cudaSuccess;
    group_rank_kernel<<<(np + 255) / 256, 256, 0, L.stream>>>(sel, np, d.n_used, d.n_expert, expert_first, expert_count, counts, ranks);
    L.count();
    return cudaGetLastError();
}

// From the pairs' numbers to the GEMMs' work lists, in one launch: every block turns the counts into the experts' first positions
// (a scan of at most 512 values), then the blocks share the pairs (pairs[position], pos_of) and the experts (units).  The order of an
// expert's pairs is that of the atomics that numbered them and differs from run to run; a pair's row of the GEMMs does not depend on it.
//
// Units of the two GEMMs: the shared expert's first (they are the longest), then for every expert its pairs in tiles of `tile`, times the
// 128-row tiles of the gate/up matrices (items_gu) and the 256-row units of the down matrix (items_dn).  The shared expert's "pairs" are
// the rows [sh_first, sh_first + sh_count), stored after the routed pairs.  pos_of[t * (n_used+1) + s] = position of pair (t, s), or
// 0xFFFFFFFF when its expert is not here.
// (Counting, scanning, placing and planning took four launches, 25 us at 77 tokens, 34 at 4096.)
__global__ void __launch_bounds__(512)
group_place_kernel(const GroupPlace a) {
    __shared__ uint32_t s_off[512];
    __shared__ unsigned long long s_wsum[16];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    pdl_trigger();
    pdl_wait();
    const uint32_t n = tid < a.expert_count ? __ldcg(a.counts + tid) : 0u, tiles = (n + a.tile - 1) / a.tile;
    const unsigned long long mine = (unsigned long long)n | ((unsigned long long)tiles << 32);
    unsigned long long v = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long up = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= (uint32_t)o) v += up;
    }
    if (lane == 31) s_wsum[warp] = v;
    __syncthreads();
    unsigned long long base = 0, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < 16; ++w) { if (w < warp) base += s_wsum[w]; total += s_wsum[w]; }
    const unsigned long long excl = base + v - mine;
    const uint32_t off = (uint32_t)excl, np_here = (uint32_t)total, sh_tiles = (a.sh_count + a.tile - 1) / a.tile;
    s_off[tid] = off;
    __syncthreads();
    auto put = [&](uint32_t at, MmaItem it) {
        for (uint32_t r = 0; r < a.rt_gu; ++r) { it.rt = (uint16_t)r; a.items_gu[(size_t)at * a.rt_gu + r] = it; }
        for (uint32_t r = 0; r < a.rt_dn; ++r) { it.rt = (uint16_t)r; a.items_dn[(size_t)at * a.rt_dn + r] = it; }
    };
    if (tid % gridDim.x == blockIdx.x) {
        const uint32_t first = sh_tiles + (uint32_t)(excl >> 32);
        for (uint32_t i = 0; i < tiles; ++i) put(first + i, MmaItem{(uint16_t)tid, 0, off + i * a.tile, min(a.tile, n - i * a.tile)});
    }
    for (uint32_t i = blockIdx.x * 512 + tid; i < sh_tiles; i += gridDim.x * 512)
        put(i, MmaItem{(uint16_t)kSharedItem, 0, np_here + i * a.tile, min(a.tile, a.sh_count - i * a.tile)});
    if (blockIdx.x == 0 && tid == 0) {
        const uint32_t all = sh_tiles + (uint32_t)(total >> 32);
        a.n_items[0] = all * a.rt_gu; a.n_items[1] = all * a.rt_dn;
        a.n_items[2] = a.n_items[3] = 0;   // the GEMMs' tickets
    }
    const uint32_t slots = a.n_used + 1;
    for (uint32_t i = blockIdx.x * 512 + tid; i < a.n_tokens * slots; i += gridDim.x * 512) {
        const uint32_t t = i / slots, s = i - t * slots;
        uint32_t pos = 0xFFFFFFFFu;
        if (s < a.n_used) {
            const uint32_t e = a.expert_count ? local_expert_of(__ldcg(&a.sel[t].ids[s]), a.n_expert, a.expert_first, a.expert_count) : 0xFFFFFFFFu;
            if (e < a.expert_count) pos = s_off[e] + __ldcg(a.ranks + t * a.n_used + s);
        } else if (t - a.sh_first < a.sh_count) {   // wraps below the range
            pos = np_here + t - a.sh_first;
        }
        a.pos_of[i] = pos;
        if (pos != 0xFFFFFFFFu) a.pairs[pos] = (t << 4) | s;
    }
}
cudaError_t launch_group_place(const Launch& L, const GroupPlace& a) {
    if (a.expert_count > 512 || a.sh_first > a.n_tokens || a.sh_count > a.n_tokens - a.sh_first) return cudaErrorInvalidValue;
    const uint32_t want = (a.n_tokens * (a.n_used + 1) + 511) / 512, blocks = want < 16 ? 16 : want > 148 ? 148 : want;
    const cudaError_t e = launch_kernel(Launch{L.stream, nullptr, true}, group_place_kernel, dim3(blocks), dim3(512), 0, a);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace qkm
