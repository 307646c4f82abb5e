// Selection of batched routing: top n_used experts of every token from its router logits.
//
// Replaces moe_select.comp / moe_select_256.comp and the selection half of moe_route_select[_hier].comp.  Rules kept: a
// non-finite logit ranks as -3.4e38 (moe_select.comp:28-34); among equal logits the lowest id ranks first
// (moe_select_256.comp:60-61); weights are a softmax over the selected logits only (moe_select.comp:71-76);
// w_shared = sigmoid(gate_inp_shexp . x) (moe_select.comp:36-45).
//
// The ids equal those of a router that accumulates in f64 (the CPU reference, src/main.cpp:1320-1341): f32 logits carry an error
// bound (the f32 sums' proven, the tensor cores' with a measured allowance for their accumulation, see launch_route_select), every
// expert within twice the bound of the k-th largest is a candidate, and the candidates' logits are evaluated again in f64, which
// also gives the weights.  Small batches come with f64 logits, which are ranked as they are.
//
// Bound by the candidates' f64 dot products (a router row of 8 KB from the L2 and 2048 conversions each; the converter takes 16 lanes
// a cycle and SM, so a weight becomes an f64 by shifts instead, see weight) and, for few tokens, by the chain of phases.
// A block per token; four warps where there are tokens enough for every SM to hold many blocks, eight below.
// 4096 tokens, 256 experts, F32 router: 122 us (twice the candidates, converted weights, 12 k instructions to find the k-th) -> 75;
// 600: 29 -> 19.
#include <math.h>

#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"

namespace qkm {

namespace sl {
constexpr float kFloor = -3.4e38f;
constexpr uint32_t kMaxExperts = 512, kMaxWarps = 8;
}  // namespace sl

struct SelectArgs {
    const uint8_t* router;
    const void* logits;        // f64 [token][expert], or n_parts partial sums of f32 ones
    const float* norm2;        // n_norm values: their largest bounds |router row|^2
    const float* gis;
    const float* x;
    qkm_sel* sel;
    int8_t* xplanes;           // optional, with f64 logits: x as digit planes and their negatives [kb][8][256], and their scales [token][kb]
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
// Four consecutive router weights as f64, times 2^-scale_bits: an f32 (f16) whose bits are moved to where an f64 has its exponent and
// mantissa is that number times 2^(127 - 1023) (2^(15 - 1023)), zeros and denormals included.  Finite values only.
template <int TYPE> constexpr int scale_bits() { return TYPE == QKM_TYPE_F32 ? 896 : 1008; }
__device__ __forceinline__ double f32_shifted(uint32_t u) { return __hiloint2double(((int)u >> 3) & (int)0x8FFFFFFF, (int)(u * 0x20000000u)); }
__device__ __forceinline__ double f16_shifted(uint32_t u) { return __hiloint2double(((int)u >> 6) & (int)0x81FFFC00, 0); }   // the upper half of u
template <int TYPE>
__device__ __forceinline__ uint4 raw4(const uint8_t* row, uint32_t u) {
    if (TYPE == QKM_TYPE_F32) return __ldg(reinterpret_cast<const uint4*>(row) + u);
    const uint2 h = __ldg(reinterpret_cast<const uint2*>(row) + u);
    return make_uint4(h.x << 16, h.x, h.y << 16, h.y);   // upper halves
}
template <int TYPE, bool SHIFT>
__device__ __forceinline__ double weight(uint32_t raw) {
    if (SHIFT) return TYPE == QKM_TYPE_F32 ? f32_shifted(raw) : f16_shifted(raw);
    return TYPE == QKM_TYPE_F32 ? (double)__uint_as_float(raw) : (double)f16_bits_to_f32(raw >> 16);
}
// two rows . x by one warp; x as f64 in two planes (elements 4u, 4u+1 and 4u+2, 4u+3 of every four: no bank conflicts)
template <int TYPE, bool SHIFT>
__device__ __forceinline__ void dot2(const uint8_t* ra, const uint8_t* rc, const double2* x0, const double2* x1, uint32_t K4, uint32_t lane, double& a, double& c) {
    double a0 = 0.0, a1 = 0.0, c0 = 0.0, c1 = 0.0;
    for (uint32_t u0 = lane; u0 < K4; u0 += 128) {
        uint4 wa[4], wc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (u0 + 32u * i < K4) { wa[i] = raw4<TYPE>(ra, u0 + 32 * i); wc[i] = raw4<TYPE>(rc, u0 + 32 * i); }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (u0 + 32u * i < K4) {
                const double2 v0 = x0[u0 + 32 * i], v1 = x1[u0 + 32 * i];
                a0 += weight<TYPE, SHIFT>(wa[i].x) * v0.x; a1 += weight<TYPE, SHIFT>(wa[i].y) * v0.y;
                a0 += weight<TYPE, SHIFT>(wa[i].z) * v1.x; a1 += weight<TYPE, SHIFT>(wa[i].w) * v1.y;
                c0 += weight<TYPE, SHIFT>(wc[i].x) * v0.x; c1 += weight<TYPE, SHIFT>(wc[i].y) * v0.y;
                c0 += weight<TYPE, SHIFT>(wc[i].z) * v1.x; c1 += weight<TYPE, SHIFT>(wc[i].w) * v1.y;
            }
    }
    a = warp_sum(a0 + a1);
    c = warp_sum(c0 + c1);
}

template <int TYPE, bool EXACT, int NK>   // 32 NK >= experts
__global__ void __launch_bounds__(sl::kMaxWarps * 32, 4)
select_tokens_kernel(const SelectArgs a) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ unsigned long long keys[sl::kMaxExperts];   // of the candidates
    __shared__ float s_log[EXACT ? 1 : sl::kMaxExperts];
    __shared__ uint16_t ids[sl::kMaxExperts];
    __shared__ double s_sg[sl::kMaxWarps];
    __shared__ float s_xs[sl::kMaxWarps], s_xm[sl::kMaxWarps];
    __shared__ uint32_t s_nc;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, n_threads = blockDim.x, n_warps = n_threads >> 5, t = blockIdx.x;
    const qkm_dims d = a.d;
    const uint32_t K4 = d.n_embd / 4;   // a multiple of 64
    double2* x0 = reinterpret_cast<double2*>(smem_raw);
    double2* x1 = x0 + K4;
    pdl_trigger();
    pdl_wait();
    const float4* xt = reinterpret_cast<const float4*>(a.x + (size_t)t * d.n_embd);

    // the logits
    if (EXACT) {
        const double* lt = reinterpret_cast<const double*>(a.logits) + (size_t)t * d.n_expert;
        for (uint32_t e = tid; e < d.n_expert; e += n_threads) { keys[e] = key_of(__ldcg(lt + e)); ids[e] = (uint16_t)e; }
    } else {
        const float* lt = reinterpret_cast<const float*>(a.logits) + (size_t)t * d.n_expert;
        for (uint32_t e = tid; e < d.n_expert; e += n_threads) {
            float v = 0.f;
#pragma unroll 8
            for (uint32_t p = 0; p < a.n_parts; ++p) v += __ldcg(lt + p * a.part_stride + e);   // partial sums over column ranges, in order
            s_log[e] = v;
        }
    }
    // one pass over the row: f64 copy, |x|^2 and the largest |x|, the shared expert's gate
    const double up = EXACT ? 1.0 : __hiloint2double((1023 + scale_bits<TYPE>()) << 20, 0);   // 2^scale_bits
    float xs = 0.f, xm = 0.f;
    double sg = 0.0;
#pragma unroll 4
    for (uint32_t u = tid; u < K4; u += n_threads) {
        const float4 v = xt[u], g = __ldg(reinterpret_cast<const float4*>(a.gis) + u);
        const double2 v0 = make_double2(v.x, v.y), v1 = make_double2(v.z, v.w);
        if (!EXACT) { x0[u] = make_double2(v0.x * up, v0.y * up); x1[u] = make_double2(v1.x * up, v1.y * up); }
        xs += v.x * v.x; xs += v.y * v.y; xs += v.z * v.z; xs += v.w * v.w;
        const float m = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
        const bool ok = fabsf(v.x) <= 3.0e38f && fabsf(v.y) <= 3.0e38f && fabsf(v.z) <= 3.0e38f && fabsf(v.w) <= 3.0e38f;
        xm = ok ? fmaxf(xm, m) : __int_as_float(0x7F800000);   // a bad value sticks as infinity
        sg += (double)g.x * v0.x; sg += (double)g.y * v0.y; sg += (double)g.z * v1.x; sg += (double)g.w * v1.y;
    }
    xs = warp_sum(xs);
    sg = warp_sum(sg);
    xm = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(xm)));   // non-negative floats order like their bits
    if (lane == 0) { s_xs[warp] = xs; s_sg[warp] = sg; s_xm[warp] = xm; }
    __syncthreads();
    xs = 0.f; xm = 0.f;
    for (uint32_t w = 0; w < n_warps; ++w) { xs += s_xs[w]; xm = fmaxf(xm, s_xm[w]); }
    if (EXACT && a.xplanes != nullptr) {   // a scale per 256 columns, a warp per such block at a time
        for (uint32_t kb = warp; kb < d.n_embd / 256; kb += n_warps) {
            float4 v[2];
            float m = 0.f;
            bool off = false;   // an infinity, a NaN or an element too large
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                v[h] = xt[64 * kb + 32 * h + lane];
                const float b = fmaxf(fmaxf(fabsf(v[h].x), fabsf(v[h].y)), fmaxf(fabsf(v[h].z), fabsf(v[h].w)));
                off |= !(fabsf(v[h].x) <= 3.0e38f && fabsf(v[h].y) <= 3.0e38f && fabsf(v[h].z) <= 3.0e38f && fabsf(v[h].w) <= 3.0e38f);
                m = fmaxf(m, b);
            }
            m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));
            off = __any_sync(0xFFFFFFFFu, off);
            const int p = off ? 0 : digit_exponent(m);
            const float up_f = ldexpf(1.0f, p);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t e[4] = {off ? 0u : digits4(__float2int_rn(v[h].x * up_f)), off ? 0u : digits4(__float2int_rn(v[h].y * up_f)),
                                       off ? 0u : digits4(__float2int_rn(v[h].z * up_f)), off ? 0u : digits4(__float2int_rn(v[h].w * up_f))};
                uint32_t* q = reinterpret_cast<uint32_t*>(a.xplanes + (size_t)t * 8 * d.n_embd + (size_t)kb * 2048 + 4 * (32 * h + lane));
#pragma unroll
                for (int j = 0; j < 4; ++j) {   // digit j of the four
                    const uint32_t s = 0x4040u + 0x1111u * j;
                    q[64 * j] = __byte_perm(__byte_perm(e[0], e[1], s), __byte_perm(e[2], e[3], s), 0x5410u);
                    q[64 * (j + 4)] = __vneg4(q[64 * j]);
                }
            }
            if (lane == 0) a.xscale[t * (d.n_embd / 256) + kb] = off ? __int_as_float(0x7FC00000) : ldexpf(1.0f, -p);
        }
    }

    if (!EXACT) {
        // every warp looks up the largest norm (a NaN's bits lie above all numbers')
        uint32_t r2b = 0;
        for (uint32_t i = lane; i < a.n_norm; i += 32) r2b = max(r2b, __float_as_uint(a.norm2[i]));
        const float r2 = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, r2b));
        if (warp == 0) {
            // k-th largest: n_used rounds of the warp's largest key, each taking one lane's out
            uint32_t k[NK];
#pragma unroll
            for (int j = 0; j < NK; ++j) k[j] = lane + 32u * j < d.n_expert ? key32_of(s_log[lane + 32 * j]) : 0u;
            uint32_t kth = 0;
#pragma unroll 1
            for (uint32_t i = 0; i < d.n_used; ++i) {
                uint32_t m = 0;
#pragma unroll
                for (int j = 0; j < NK; ++j) m = max(m, k[j]);
                kth = __reduce_max_sync(0xFFFFFFFFu, m);
                bool out = lane == __ffs(__ballot_sync(0xFFFFFFFFu, m == kth)) - 1;
#pragma unroll
                for (int j = 0; j < NK; ++j)
                    if (out && k[j] == kth) { k[j] = 0; out = false; }
            }
            const float kv = __uint_as_float((kth & 0x80000000u) ? (kth ^ 0x80000000u) : ~kth);
            // |error of one logit| <= eps_terms * 2^-24 * sum|w_k x_k| <= that * |w| * |x|; two logits are compared.  A NaN threshold
            // (NaN in x or in the router) admits every expert.
            const float eps = 5.9604645e-8f * (a.eps_terms * sqrtf(r2) + a.eps_abs) * sqrtf(xs);
            const float thresh = kv - 2.1f * eps;
            uint32_t nc = 0;
#pragma unroll
            for (int j = 0; j < NK; ++j) {
                const uint32_t e = lane + 32u * j;
                float v = e < d.n_expert ? s_log[e] : 0.f;
                v = (isnan(v) || isinf(v)) ? sl::kFloor : v;
                const uint32_t in = __ballot_sync(0xFFFFFFFFu, e < d.n_expert && !(v < thresh));
                if ((in >> lane) & 1u) ids[nc + __popc(in & ((1u << lane) - 1u))] = (uint16_t)e;   // ascending
                nc += __popc(in);
            }
            if (lane == 0) s_nc = nc;
        }
        __syncthreads();
        const uint32_t nc = s_nc;
        const size_t rb = row_bytes(TYPE, d.n_embd);
        // the shifted form needs finite weights and an x that the scale does not overflow
        const bool shift = r2 <= 3.0e38f && xm <= (TYPE == QKM_TYPE_F32 ? 1.0e37f : 16384.f);
        for (uint32_t c = 2 * warp; c < nc; c += 2 * n_warps) {   // two candidates at a time share the reads of x
            const uint8_t* ra = a.router + (size_t)ids[c] * rb;
            const uint8_t* rc = a.router + (size_t)ids[min(c + 1, nc - 1)] * rb;
            double p, q;
            if (shift) {
                dot2<TYPE, true>(ra, rc, x0, x1, K4, lane, p, q);
            } else {   // rare: x as it is, weights converted
                double a0 = 0.0, c0 = 0.0;
                for (uint32_t u = lane; u < K4; u += 32) {
                    const uint4 wa = raw4<TYPE>(ra, u), wc = raw4<TYPE>(rc, u);
                    const float4 v = xt[u];
                    a0 += weight<TYPE, false>(wa.x) * (double)v.x; a0 += weight<TYPE, false>(wa.y) * (double)v.y;
                    a0 += weight<TYPE, false>(wa.z) * (double)v.z; a0 += weight<TYPE, false>(wa.w) * (double)v.w;
                    c0 += weight<TYPE, false>(wc.x) * (double)v.x; c0 += weight<TYPE, false>(wc.y) * (double)v.y;
                    c0 += weight<TYPE, false>(wc.z) * (double)v.z; c0 += weight<TYPE, false>(wc.w) * (double)v.w;
                }
                p = warp_sum(a0); q = warp_sum(c0);
            }
            if (lane == 0) keys[c] = key_of(p);
            if (lane == 0 && c + 1 < nc) keys[c + 1] = key_of(q);
        }
    }
    __syncthreads();
    if (warp != 0) return;
    const uint32_t nc = EXACT ? d.n_expert : s_nc;
    // rank: every round takes the largest key, the lowest id (place in the list) among equal ones; lane c & 31 owns candidate c
    unsigned long long my_key = 0, mine = lane < nc ? keys[lane] : 0ull;   // up to 32 candidates stay in registers
    uint32_t my_c = 0;
#pragma unroll 1
    for (uint32_t i = 0; i < d.n_used; ++i) {
        unsigned long long best = mine;
        uint32_t bc = lane < nc ? lane : 0xFFFFFFFFu;
        for (uint32_t c = lane + 32; c < nc; c += 32)
            if (keys[c] > best) { best = keys[c]; bc = c; }
        const uint32_t bh = (uint32_t)(best >> 32), bl = (uint32_t)best;
        const uint32_t mh = __reduce_max_sync(0xFFFFFFFFu, bh);
        const uint32_t ml = __reduce_max_sync(0xFFFFFFFFu, bh == mh ? bl : 0u);
        const uint32_t c = __reduce_min_sync(0xFFFFFFFFu, bh == mh && bl == ml ? bc : 0xFFFFFFFFu);
        if (c == bc) { if (c < 32) mine = 0; else if (c < nc) keys[c] = 0; }   // below every real key
        if (lane == i) { my_key = ((unsigned long long)mh << 32) | ml; my_c = min(c, nc - 1); }
    }
    // lane i < n_used: softmax term of pick i
    const double v = value_of(my_key), top = __shfl_sync(0xFFFFFFFFu, v, 0);
    double gate = 0.0;
    for (uint32_t w = 0; w < n_warps; ++w) gate += s_sg[w];
    const double ex = exp(lane < 16 ? v - top : -gate);   // lanes 0..15: picks; the others: the gate
    const double wv = lane < d.n_used ? ex : 0.0;
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
        s->w_shared = (float)(1.0 / (1.0 + ex));
        s->route_done = 0;
    } else if (lane < 23) {
        s->pad[lane - 17] = 0.f;
    }
}

template <int TYPE, bool EXACT, int NK>
static cudaError_t select_launch(const Launch& L, const SelectArgs& a) {
    const size_t smem = EXACT ? 0 : (size_t)a.d.n_embd * 8;
    if (smem > 200 * 1024) return cudaErrorInvalidValue;
    if (const cudaError_t e = allow_dynamic_smem<select_tokens_kernel<TYPE, EXACT, NK>>(200 * 1024)) return e;
    // eight warps share a token's candidates while the blocks of all tokens fit the SMs at once, four beyond (less waits for the one
    // warp that ranks)
    const uint32_t warps = a.n_tokens <= 592 ? 8 : 4;
    const cudaError_t e = launch_kernel(Launch{L.stream, nullptr, true}, select_tokens_kernel<TYPE, EXACT, NK>, dim3(a.n_tokens), dim3(warps * 32), smem, a);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}
cudaError_t launch_select_tokens(const Launch& L, const qkm_dims& d, uint32_t router_type, const SelectIn& in, qkm_sel* sel, uint32_t n_tokens) {
    if (in.xplanes && (!in.exact || d.n_embd % 256)) return cudaErrorInvalidValue;
    SelectArgs a{};
    a.router = (const uint8_t*)in.router; a.logits = in.logits; a.norm2 = in.norm2; a.n_norm = in.n_norm; a.gis = in.gis; a.x = in.x; a.sel = sel;
    a.xplanes = in.xplanes; a.xscale = in.xscale; a.counts = in.counts; a.ranks = in.ranks; a.part_stride = (size_t)n_tokens * d.n_expert; a.n_parts = in.n_parts;
    a.n_tokens = n_tokens; a.expert_first = in.expert_first; a.expert_count = in.expert_count; a.eps_terms = in.eps_terms; a.eps_abs = in.eps_abs; a.d = d;
    if (in.exact) return router_type == QKM_TYPE_F32 ? select_launch<QKM_TYPE_F32, true, 1>(L, a) : select_launch<QKM_TYPE_F16, true, 1>(L, a);
    if (d.n_expert <= 256) return router_type == QKM_TYPE_F32 ? select_launch<QKM_TYPE_F32, false, 8>(L, a) : select_launch<QKM_TYPE_F16, false, 8>(L, a);
    return router_type == QKM_TYPE_F32 ? select_launch<QKM_TYPE_F32, false, 16>(L, a) : select_launch<QKM_TYPE_F16, false, 16>(L, a);
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
