// Hidden rows of batched prefill between the two expert GEMMs (qkm_wgemm.cu): rows whose scale served them badly are made again.
//
// The gate/up epilogue scales a row before any of its values is known, from the bound |h| <= |gate row| |x| |up row| |x|, to at
// most 2^15.  As a rule the row's largest value lies 2^7 to 2^13 below the bound and the row keeps f16's full precision.  But nothing
// limits the distance: x that is large where the weights are small, or gates that are all strongly negative, leave a row among f16's
// subnormals or flush it to zero (an element of 1e5 in columns without weights: layer output 4.6e-2 from 64 bits instead of 6e-4),
// and a bound that passes f32 leaves it infinite.  So every row's largest magnitude is looked at here: from 2^-3 on an element's error
// is at most 2^-11 of itself or 2^-22 of the row's largest, and the row stays; else the row's gate/up products are taken again in f32
// from the same operands and scaled by what they turn out to be.
//
// A warp looks at a row or at four (one read of them, from the L2: 38 MB at 4096 tokens); a block makes a row again, its warps share
// the weight rows.  Bound by that read and the launch: 3.0 us of a layer's 177 at 77 tokens, none measurable of 238 at 600, 7.7 of 534
// at 4096 (rows found by token and slot, a position looked up first and a row a warp: 3.8, 3.4 and 13.6).
#include <cuda_fp16.h>

#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"

namespace qkm {

namespace hr {
constexpr uint32_t kWarps = 8, kMaxFf = 4096;
constexpr uint32_t kFewRows = 9472;   // below: a row a warp (8 blocks of 8 warps an SM hold them at once), above: four rows' loads under way together
constexpr uint32_t kLow = 0x3000u, kInf = 0x7C00u;   // f16 bits of 2^-3 and of infinity
}  // namespace hr

// silu(gate . x) * (up . x) of the weight rows this warp owns -> s_h.  xh: the row as the GEMM's operand, elements (0, 2, 1, 3)
template <int TYPE>
__device__ __forceinline__ void hidden_again(const uint8_t* gate, const uint8_t* up, const __half* xh, float x_inv, uint32_t n_ff, uint32_t K, float* s_h) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const size_t rb = row_bytes(TYPE, K);
#pragma unroll 1
    for (uint32_t r = warp; r < n_ff; r += hr::kWarps) {
        float g = 0.f, u = 0.f;
#pragma unroll 1
        for (uint32_t k = 8 * lane; k < K; k += 256) {
            const uint4 q = *reinterpret_cast<const uint4*>(xh + k);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
            float x[8], wg[8], wu[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {   // word i: elements 4 (i / 2) + (i & 1) and two on
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                x[4 * (i >> 1) + (i & 1)] = f.x;
                x[4 * (i >> 1) + (i & 1) + 2] = f.y;
            }
            dequant8<TYPE>(gate + r * rb, k, wg);
            dequant8<TYPE>(up + r * rb, k, wu);
#pragma unroll
            for (int i = 0; i < 8; ++i) { g += wg[i] * x[i]; u += wu[i] * x[i]; }
        }
        g = warp_sum(g) * x_inv;
        u = warp_sum(u) * x_inv;
        if (lane == 0) s_h[r] = g / (1.0f + expf(-g)) * u;
    }
}

// ROWS consecutive rows a warp
template <int TYPE, int ROWS>
__global__ void __launch_bounds__(hr::kWarps * 32)
hidden_rows_check_kernel(const HiddenRows a) {
    constexpr uint32_t kRows = hr::kWarps * ROWS;
    __shared__ float s_h[hr::kMaxFf];
    __shared__ float s_max[hr::kWarps];
    __shared__ uint32_t s_bad[kRows];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, slots = a.n_used + 1, rows = a.n_tokens * slots;
    pdl_trigger();
    pdl_wait();
    auto expert_of = [&](uint32_t t, uint32_t s) { return s < a.n_used ? local_expert_of(a.sel[t].ids[s], a.n_expert, a.expert_first, a.expert_count) : a.expert_count; };
    const uint32_t base = blockIdx.x * kRows;
    uint32_t m[ROWS];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) m[j] = 0;
    for (uint32_t k = lane; k < a.n_ff / 8; k += 32) {
        uint4 v[ROWS];   // under way together
#pragma unroll
        for (int j = 0; j < ROWS; ++j) v[j] = reinterpret_cast<const uint4*>(a.h + (size_t)min(base + warp * ROWS + j, rows - 1) * a.n_ff)[k];
#pragma unroll
        for (int j = 0; j < ROWS; ++j)
            m[j] = __vmaxu2(__vmaxu2(m[j], __vmaxu2(v[j].x & 0x7FFF7FFFu, v[j].y & 0x7FFF7FFFu)), __vmaxu2(v[j].z & 0x7FFF7FFFu, v[j].w & 0x7FFF7FFFu));
    }
    bool any = false;
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, max(m[j] & 0xFFFFu, m[j] >> 16)), p = base + warp * ROWS + j;
        bool bad = false;
        if (p < rows && (most < hr::kLow || most >= hr::kInf)) {
            // a shard has fewer rows than positions: a row counts if its pair (left by an earlier call, or never written) says it lies here
            const uint32_t pair = a.pairs[p], t = pair >> 4, s = pair & 15u;
            if (t < a.n_tokens && s <= a.n_used && a.pos_of[t * slots + s] == p) {
                const uint32_t e = expert_of(t, s);
                const float xn = a.x_norm[t];
                bad = a.w_norm[e] * xn * (a.w_norm[a.expert_count + 1 + e] * xn) > 0.f;   // not for rows of zeros, nor for NaN in x
            }
        }
        if (lane == 0) s_bad[warp * ROWS + j] = bad ? 1u : 0u;
        any |= bad;
    }
    if (!__syncthreads_or(any ? 1 : 0)) return;
#pragma unroll 1
    for (uint32_t w = 0; w < kRows; ++w) {
        if (!s_bad[w]) continue;
        const uint32_t pos = base + w, t = a.pairs[pos] >> 4, s = a.pairs[pos] & 15u;
        const __half* xh = a.xrows + (size_t)t * a.n_embd;
        if (s < a.n_used) {
            const size_t at = (size_t)expert_of(t, s) * a.n_ff * row_bytes(TYPE, a.n_embd);
            hidden_again<TYPE>(a.w[0] + at, a.w[1] + at, xh, a.x_inv_scale[t], a.n_ff, a.n_embd, s_h);
        } else {
            hidden_again<QKM_TYPE_Q8_0>(a.sh[0], a.sh[1], xh, a.x_inv_scale[t], a.n_ff, a.n_embd, s_h);
        }
        __syncthreads();
        float m = 0.f;
        for (uint32_t r = threadIdx.x; r < a.n_ff; r += hr::kWarps * 32) {
            const float v = fabsf(s_h[r]);
            if (v <= 3.402823466e38f) m = fmaxf(m, v);
        }
        m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));   // non-negative floats order like their bits
        if (lane == 0) s_max[warp] = m;
        __syncthreads();
        m = 0.f;
#pragma unroll
        for (uint32_t v = 0; v < hr::kWarps; ++v) m = fmaxf(m, s_max[v]);
        int q = 0;
        if (m > 0.f) { int e; frexpf(m, &e); q = min(14 - e, 126); }   // m * 2^q in [2^13, 2^14)
        const float up = ldexpf(1.0f, q);
        for (uint32_t r = threadIdx.x; r < a.n_ff; r += hr::kWarps * 32)
            a.h[(size_t)pos * a.n_ff + (r & ~3u) + ((r & 1u) << 1) + ((r >> 1) & 1u)] = __float2half_rn(s_h[r] * up);
        if (threadIdx.x == 0) a.h_inv_scale[pos] = ldexpf(1.0f, -q);
        __syncthreads();
    }
}

template <int TYPE, int ROWS>
static cudaError_t check_launch(const Launch& L, const HiddenRows& a) {
    const uint32_t rows = a.n_tokens * (a.n_used + 1);
    const cudaError_t e = launch_kernel(Launch{L.stream, nullptr, true}, hidden_rows_check_kernel<TYPE, ROWS>, dim3((rows + hr::kWarps * ROWS - 1) / (hr::kWarps * ROWS)),
                                        dim3(hr::kWarps * 32), 0, a);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}
cudaError_t launch_hidden_rows_check(const Launch& L, uint32_t type, const HiddenRows& a) {
    const uint64_t rows = (uint64_t)a.n_tokens * (a.n_used + 1);
    if (rows == 0) return cudaSuccess;
    if (a.n_ff > hr::kMaxFf || a.n_ff % 8 || a.n_embd % 256 || rows > 0xFFFFFFFFull) return cudaErrorInvalidValue;
    if (type == QKM_TYPE_IQ3_XXS) return rows <= hr::kFewRows ? check_launch<QKM_TYPE_IQ3_XXS, 1>(L, a) : check_launch<QKM_TYPE_IQ3_XXS, 4>(L, a);
    if (type == QKM_TYPE_IQ4_XS) return rows <= hr::kFewRows ? check_launch<QKM_TYPE_IQ4_XS, 1>(L, a) : check_launch<QKM_TYPE_IQ4_XS, 4>(L, a);
    return cudaErrorInvalidValue;
}

}  // namespace qkm
