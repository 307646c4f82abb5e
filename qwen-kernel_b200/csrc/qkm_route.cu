// Router: logits, top-k selection, and token-expert pair grouping.
//
// Replaces moe_logits.comp / moe_logits_gemm.comp (logits), moe_select.comp /
// moe_select_256.comp (selection from f32 logits), moe_route_select[_hier].comp
// (both in one call) and moe_group_pairs.comp.
//
// Selection rules kept from the reference: a non-finite logit ranks as -3.4e38
// (moe_select.comp:28-34); among equal logits the lowest expert id ranks first
// (moe_select_256.comp:60-61); weights are a softmax over the selected logits
// only (moe_select.comp:71-76); w_shared = sigmoid(gate_inp_shexp . x)
// (moe_select.comp:36-45).
//
// The fused path additionally guarantees that ids equal those of a router that
// accumulates in f64 (the CPU reference, src/main.cpp:1320-1341): f32 logits
// carry an error bound eps, every expert whose f32 logit lies within
// 2*eps of the k-th largest is a candidate, candidates are re-evaluated in f64
// and the final ranking uses those values.
#include <math.h>

#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"

namespace qkm {

static constexpr float kFloor = -3.4e38f;

// ---- logits: two expert rows per block, four warps (column quarters) per row ----------------
// Every lane owns at most kMaxUnits 8-element units of its quarter, loads them and the
// matching x values of kTokPerBlock tokens up front (one memory round trip), adds its
// products in a fixed order, then the lanes meet in a 5-level tree and the four quarters
// in shared memory: fewer sequential additions than the error bound of the refined
// selection assumes.  Also writes |router row|^2 when row_norm2 != NULL.
static constexpr int kTokPerBlock = 4;
static constexpr int kMaxUnits = 2;  // K <= 2048 in one pass; longer rows loop

// With ACC = double the logits are those of an f64-accumulating router outright (the f64
// pipe does the 2 * K * n_expert flops of a decode batch in well under a microsecond), and
// the selection needs no error bound or re-evaluation.
template <int TYPE, typename ACC>
__global__ void __launch_bounds__(256)
logits_kernel(const uint8_t* __restrict__ router, const float* __restrict__ x, ACC* __restrict__ logits,
              float* __restrict__ row_norm2, uint32_t n_expert, uint32_t K, uint32_t n_tokens) {
    __shared__ ACC s_part[8][kTokPerBlock + 1];
    pdl_trigger();
    pdl_wait();   // the logits buffer is reused from layer to layer
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t e = blockIdx.x * 2u + (warp >> 2), quarter = warp & 3u;
    const uint32_t t0 = blockIdx.y * kTokPerBlock;
    const uint32_t units_q = K / 32;  // units per quarter
    ACC acc[kTokPerBlock], nrm = 0;
#pragma unroll
    for (int j = 0; j < kTokPerBlock; ++j) acc[j] = 0;
    if (e < n_expert) {
        const uint8_t* row = router + (size_t)e * row_bytes(TYPE, K);
        for (uint32_t u0 = lane; u0 < units_q; u0 += 32 * kMaxUnits) {
            float w[kMaxUnits][8];
            float4 xa[kMaxUnits][kTokPerBlock], xb[kMaxUnits][kTokPerBlock];
#pragma unroll
            for (int i = 0; i < kMaxUnits; ++i) {
                const uint32_t u = u0 + 32 * i;
                if (u < units_q) {
                    const uint32_t k = (quarter * units_q + u) * 8;
                    dequant8<TYPE>(row, k, w[i]);
#pragma unroll
                    for (int j = 0; j < kTokPerBlock; ++j) {
                        const uint32_t tt = min(t0 + j, n_tokens - 1);
                        const float* xt = x + (size_t)tt * K + k;
                        xa[i][j] = *reinterpret_cast<const float4*>(xt);
                        xb[i][j] = *reinterpret_cast<const float4*>(xt + 4);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < kMaxUnits; ++i) {
                if (u0 + 32 * i < units_q) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) nrm += (ACC)(w[i][q] * w[i][q]);
#pragma unroll
                    for (int j = 0; j < kTokPerBlock; ++j) {
                        ACC s = acc[j];
                        s += (ACC)w[i][0] * (ACC)xa[i][j].x; s += (ACC)w[i][1] * (ACC)xa[i][j].y;
                        s += (ACC)w[i][2] * (ACC)xa[i][j].z; s += (ACC)w[i][3] * (ACC)xa[i][j].w;
                        s += (ACC)w[i][4] * (ACC)xb[i][j].x; s += (ACC)w[i][5] * (ACC)xb[i][j].y;
                        s += (ACC)w[i][6] * (ACC)xb[i][j].z; s += (ACC)w[i][7] * (ACC)xb[i][j].w;
                        acc[j] = s;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kTokPerBlock; ++j) {
        const ACC v = warp_sum(acc[j]);
        if (lane == 0) s_part[warp][j] = v;
    }
    nrm = warp_sum(nrm);
    if (lane == 0) s_part[warp][kTokPerBlock] = nrm;
    __syncthreads();
    if (quarter == 0 && e < n_expert && lane <= kTokPerBlock) {
        const ACC v = ((s_part[warp][lane] + s_part[warp + 1][lane]) + s_part[warp + 2][lane]) + s_part[warp + 3][lane];
        if (lane < kTokPerBlock) {
            if (t0 + lane < n_tokens) logits[(size_t)(t0 + lane) * n_expert + e] = v;
        } else if (row_norm2 != nullptr && blockIdx.y == 0) {
            row_norm2[e] = (float)v;
        }
    }
}

cudaError_t launch_logits(const Launch& L, const qkm_dims& d, uint32_t router_type, const void* router,
                          const float* x, float* logits, float* row_norm2, uint32_t n_tokens) {
    if (n_tokens == 0) return cudaSuccess;
    const dim3 grid((d.n_expert + 1) / 2, (n_tokens + kTokPerBlock - 1) / kTokPerBlock);
    const uint8_t* r = (const uint8_t*)router;
    if (router_type == QKM_TYPE_F32)
        logits_kernel<QKM_TYPE_F32, float><<<grid, 256, 0, L.stream>>>(r, x, logits, row_norm2, d.n_expert, d.n_embd, n_tokens);
    else if (router_type == QKM_TYPE_F16)
        logits_kernel<QKM_TYPE_F16, float><<<grid, 256, 0, L.stream>>>(r, x, logits, row_norm2, d.n_expert, d.n_embd, n_tokens);
    else
        return cudaErrorInvalidValue;
    L.count();
    return cudaGetLastError();
}

static cudaError_t launch_logits64(const Launch& L, const qkm_dims& d, uint32_t router_type, const void* router,
                                   const float* x, double* logits, uint32_t n_tokens) {
    const dim3 grid((d.n_expert + 1) / 2, (n_tokens + kTokPerBlock - 1) / kTokPerBlock);
    const uint8_t* r = (const uint8_t*)router;
    cudaError_t e;
    if (router_type == QKM_TYPE_F32)
        e = launch_kernel(L, logits_kernel<QKM_TYPE_F32, double>, grid, dim3(256), 0, r, x, logits, (float*)nullptr, d.n_expert, d.n_embd, n_tokens);
    else
        e = launch_kernel(L, logits_kernel<QKM_TYPE_F16, double>, grid, dim3(256), 0, r, x, logits, (float*)nullptr, d.n_expert, d.n_embd, n_tokens);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}

// ---- logits for many tokens: 64 x 64 output tiles, f32 FMA -------------------------------------
// logits[t][e] = sum_k x[t][k] * w[e][k], k ascending in one chain per output (the refined
// selection is told the chain length).  Operands are staged through shared memory 16
// columns at a time; each thread owns a 4 x 4 block of outputs.
template <int TYPE>
__global__ void __launch_bounds__(256)
logits_gemm_kernel(const uint8_t* __restrict__ router, const float* __restrict__ x, float* __restrict__ logits,
                   uint32_t n_expert, uint32_t K, uint32_t n_tokens) {
    __shared__ __align__(16) float s_xt[16][64 + 4];   // [k][token]
    __shared__ __align__(16) float s_wt[16][64 + 4];   // [k][expert]
    const uint32_t tid = threadIdx.x, tx = tid & 15u, ty = tid >> 4;
    const uint32_t e0 = blockIdx.x * 64, t0 = blockIdx.y * 64;
    const size_t rb = row_bytes(TYPE, K);
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    // loader role: thread -> (row = tid / 4, 4 columns at (tid % 4) * 4) of both operand tiles
    const uint32_t lr = tid >> 2, lc = (tid & 3u) * 4;
    auto fetch = [&](uint32_t k0, float4& xv, float4& wv) {
        xv = make_float4(0.f, 0.f, 0.f, 0.f); wv = xv;
        if (t0 + lr < n_tokens) xv = *reinterpret_cast<const float4*>(x + (size_t)(t0 + lr) * K + k0 + lc);
        if (e0 + lr < n_expert) {
            const uint8_t* row = router + (size_t)(e0 + lr) * rb;
            if (TYPE == QKM_TYPE_F32) {
                wv = *reinterpret_cast<const float4*>(row + (size_t)(k0 + lc) * 4);
            } else {
                const uint2 hv = *reinterpret_cast<const uint2*>(row + (size_t)(k0 + lc) * 2);
                wv = make_float4(f16_bits_to_f32(hv.x & 0xFFFFu), f16_bits_to_f32(hv.x >> 16),
                                 f16_bits_to_f32(hv.y & 0xFFFFu), f16_bits_to_f32(hv.y >> 16));
            }
        }
    };
    float4 xv, wv;
    fetch(0, xv, wv);
    for (uint32_t k0 = 0; k0 < K; k0 += 16) {
        __syncthreads();
        s_xt[lc + 0][lr] = xv.x; s_xt[lc + 1][lr] = xv.y; s_xt[lc + 2][lr] = xv.z; s_xt[lc + 3][lr] = xv.w;
        s_wt[lc + 0][lr] = wv.x; s_wt[lc + 1][lr] = wv.y; s_wt[lc + 2][lr] = wv.z; s_wt[lc + 3][lr] = wv.w;
        __syncthreads();
        if (k0 + 16 < K) fetch(k0 + 16, xv, wv);   // next tile's loads fly during this tile's math
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float4 a = *reinterpret_cast<const float4*>(&s_xt[k][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&s_wt[k][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += av[i] * bv[j];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t t = t0 + ty * 4 + i;
        if (t < n_tokens) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t e = e0 + tx * 4 + j;
                if (e < n_expert) logits[(size_t)t * n_expert + e] = acc[i][j];
            }
        }
    }
}

// |router row|^2, one warp per row
template <int TYPE>
__global__ void __launch_bounds__(256)
row_norm2_kernel(const uint8_t* __restrict__ router, float* __restrict__ row_norm2, uint32_t* __restrict__ max_bits, uint32_t n_expert, uint32_t K) {
    const uint32_t e = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (e >= n_expert) return;
    const uint8_t* row = router + (size_t)e * row_bytes(TYPE, K);
    float nrm = 0.f;
    for (uint32_t u = lane; u < K / 8; u += 32) {
        float w[8];
        dequant8<TYPE>(row, u * 8, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) nrm += w[i] * w[i];
    }
    nrm = warp_sum(nrm);
    if (lane == 0 && row_norm2) row_norm2[e] = nrm;
    if (lane == 0 && max_bits) atomicMax(max_bits, __float_as_uint(nrm));   // non-negative floats order like their bits, a NaN above them
}

cudaError_t launch_row_norm2(const Launch& L, const qkm_dims& d, uint32_t router_type, const void* router, float* norm2, float* largest) {
    const uint8_t* r = (const uint8_t*)router;
    if (router_type == QKM_TYPE_F32) row_norm2_kernel<QKM_TYPE_F32><<<(d.n_expert + 7) / 8, 256, 0, L.stream>>>(r, norm2, (uint32_t*)largest, d.n_expert, d.n_embd);
    else if (router_type == QKM_TYPE_F16) row_norm2_kernel<QKM_TYPE_F16><<<(d.n_expert + 7) / 8, 256, 0, L.stream>>>(r, norm2, (uint32_t*)largest, d.n_expert, d.n_embd);
    else return cudaErrorInvalidValue;
    L.count();
    return cudaGetLastError();
}

// ---- helpers for block-wide (value, lowest id) argmax --------------------------------------
// Key orders by value first; among equal values the smaller id gives the larger key.
__device__ __forceinline__ unsigned long long rank_key(float v, uint32_t id) {
    v = v + 0.0f;  // -0 -> +0 so the two zeros tie
    uint32_t b = __float_as_uint(v);
    b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    return ((unsigned long long)b << 32) | (unsigned long long)(0xFFFFFFFFu - id);
}
__device__ __forceinline__ float sane(float v) { return (isnan(v) || isinf(v)) ? kFloor : v; }

__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xFFFFFFFFu, k, o);
        k = other > k ? other : k;
    }
    return k;
}

// Block-wide argmax over the (up to) 2 logits every one of 256 threads holds.
// Returns the winning key to every thread.
__device__ __forceinline__ unsigned long long block_argmax(float v0, uint32_t id0, float v1, uint32_t id1,
                                                           unsigned long long* s_warp /* [8] */) {
    const unsigned long long k0 = rank_key(v0, id0), k1 = rank_key(v1, id1);
    unsigned long long k = warp_max_u64(k0 > k1 ? k0 : k1);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    __syncthreads();  // s_warp reuse across rounds
    if (lane == 0) s_warp[warp] = k;
    __syncthreads();
    k = s_warp[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) k = s_warp[w] > k ? s_warp[w] : k;
    return k;
}

// f64 dot of gate_inp_shexp with x over 256 threads; result valid in thread 0.
__device__ __forceinline__ double block_dot_f64(const float* __restrict__ a, const float* __restrict__ b,
                                                uint32_t K, double* s_red /* [8] */) {
    double acc = 0.0;
    for (uint32_t k = threadIdx.x; k < K; k += 256) acc += (double)a[k] * (double)b[k];
    acc = warp_sum(acc);
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) s_red[threadIdx.x >> 5] = acc;
    __syncthreads();
    double tot = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < 8; ++w) tot += s_red[w];
    return tot;
}

// ---- selection from given f32 logits: one block per token --------------------------------
__global__ void __launch_bounds__(256)
select_kernel(const float* __restrict__ logits, const float* __restrict__ gis, const float* __restrict__ x,
              qkm_sel* __restrict__ sel, qkm_dims d) {
    __shared__ unsigned long long s_warp[8];
    __shared__ double s_red[8];
    __shared__ float s_pick[16];
    const uint32_t t = blockIdx.x, tid = threadIdx.x;
    const float* lt = logits + (size_t)t * d.n_expert;
    const uint32_t id0 = tid, id1 = tid + 256u;
    float v0 = id0 < d.n_expert ? sane(lt[id0]) : kFloor;
    float v1 = id1 < d.n_expert ? sane(lt[id1]) : kFloor;
    // padding lanes must never beat a real expert on a tie: give them the largest ids
    const uint32_t pid0 = id0 < d.n_expert ? id0 : 0xFFFFFFFEu;
    const uint32_t pid1 = id1 < d.n_expert ? id1 : 0xFFFFFFFEu;

    const double sg = block_dot_f64(gis, x + (size_t)t * d.n_embd, d.n_embd, s_red);
    if (tid == 0) {
        sel[t].w_shared = (float)(1.0 / (1.0 + exp(-sg)));
        sel[t].route_done = 0;
#pragma unroll
        for (int i = 0; i < 6; ++i) sel[t].pad[i] = 0.f;
    }
    for (uint32_t i = 0; i < 16; ++i) {
        if (i >= d.n_used) {
            if (tid == 0) { sel[t].ids[i] = 0; sel[t].w[i] = 0.f; }
            continue;
        }
        const unsigned long long k = block_argmax(v0, pid0, v1, pid1, s_warp);
        uint32_t id = 0xFFFFFFFFu - (uint32_t)(k & 0xFFFFFFFFull);
        if (id >= d.n_expert) id = d.n_expert - 1;  // clamp (moe_select.comp:61-63)
        if (tid == 0) {
            uint32_t b = (uint32_t)(k >> 32);
            b = (b & 0x80000000u) ? (b & 0x7FFFFFFFu) : ~b;
            sel[t].ids[i] = id;
            s_pick[i] = __uint_as_float(b);
        }
        if (id == id0) v0 = kFloor;
        if (id == id1) v1 = kFloor;
    }
    __syncthreads();
    if (tid == 0) {
        double w[16], sum = 0.0;
        for (uint32_t i = 0; i < d.n_used; ++i) { w[i] = exp((double)s_pick[i] - (double)s_pick[0]); sum += w[i]; }
        for (uint32_t i = 0; i < d.n_used; ++i) sel[t].w[i] = (float)(w[i] / sum);
    }
}

cudaError_t launch_select(const Launch& L, const qkm_dims& d, const float* logits, const float* gis,
                          const float* x, qkm_sel* sel, uint32_t n_tokens) {
    if (n_tokens == 0) return cudaSuccess;
    select_kernel<<<n_tokens, 256, 0, L.stream>>>(logits, gis, x, sel, d);
    L.count();
    return cudaGetLastError();
}

static constexpr uint32_t kExactMaxTokens = 64;   // decode-sized batches rank f64 logits directly

size_t route_scratch_bytes(uint32_t n_tokens, uint32_t n_expert) {
    // f32 logits (partial sums over up to 16 column ranges while the batch is small: about 20,000 rows of them at most) + row norms
    const size_t rows = n_tokens > kExactMaxTokens ? (16u * (size_t)n_tokens < 20000 ? 16u * (size_t)n_tokens : n_tokens > 20000 ? n_tokens : 20000) : n_tokens;
    const size_t f32_path = (rows * n_expert + n_expert) * sizeof(float);
    const size_t f64_path = (size_t)(n_tokens < kExactMaxTokens ? n_tokens : kExactMaxTokens) * n_expert * sizeof(double);
    return f32_path > f64_path ? f32_path : f64_path;
}

cudaError_t launch_route_select(const Launch& L, const qkm_dims& d, uint32_t router_type, const void* router, const float* gis, const float* x, qkm_sel* sel,
                                uint32_t n_tokens, void* scratch, size_t scratch_bytes, const RouteExtra& ex) {
    if (n_tokens == 0) return cudaSuccess;
    if (router_type != QKM_TYPE_F32 && router_type != QKM_TYPE_F16) return cudaErrorInvalidValue;
    SelectIn in{};
    in.router = router; in.gis = gis; in.x = x; in.xplanes = ex.xplanes; in.xscale = ex.xscale; in.counts = ex.counts; in.ranks = ex.ranks;
    in.expert_first = ex.expert_first; in.expert_count = ex.expert_count; in.n_parts = 1; in.logits = scratch;
    if (n_tokens <= kExactMaxTokens && (size_t)n_tokens * d.n_expert * sizeof(double) <= scratch_bytes) {
        // small batch: f64 logits, ranked as they are
        in.exact = true;
        if (const cudaError_t e = launch_logits64(L, d, router_type, router, x, (double*)scratch, n_tokens)) return e;
        return launch_select_tokens(L, d, router_type, in, sel, n_tokens);
    }
    if (((size_t)n_tokens * d.n_expert + d.n_expert) * sizeof(float) > scratch_bytes) return cudaErrorInvalidValue;
    float* logits = (float*)scratch;
    float* norm2 = logits + (size_t)n_tokens * d.n_expert;
    const uint8_t* r = (const uint8_t*)router;
    in.norm2 = norm2; in.n_norm = d.n_expert;
    if (ex.x_f16 && ex.router_f16 && ex.router_norm2 && d.n_expert % 128 == 0 && d.n_embd <= 4096) {
        // tensor cores, f16 operands: |error| <= (2^-11 [x] + 2^-11 [router] + columns of a partial sum * 2^-22) |w| |x|, plus the flush of
        // tiny router values.  2^-22 a column for the accumulation is an allowance: nothing documents what the tensor cores keep.  Measured
        // on the B200: addends of an MMA are cut off at 2^-25 of the largest, no column loses more than that (a test holds it to 2^-24).  Few output tiles: the columns are split over more blocks, partial logits side by side (summed by the
        // selection kernel).
        const uint32_t tiles = ((n_tokens + 127) / 128) * (d.n_expert / 128);
        uint32_t splits = 1;
        while (splits < 16 && tiles * splits * 2 <= 148u && (d.n_embd / 64) % (splits * 2) == 0 &&
               (size_t)n_tokens * d.n_expert * (splits * 2) * sizeof(float) <= scratch_bytes) splits *= 2;
        if (const cudaError_t e = launch_logits_mma(L, d, ex.router_f16, ex.x_f16, ex.x_f16_inv, logits, n_tokens, ex.status, splits)) return e;
        in.norm2 = ex.router_norm2; in.n_norm = 1; in.n_parts = splits;
        in.eps_terms = 16384.f + 4.f * (float)(d.n_embd / splits) + (float)splits;   // in units of 2^-24, with the additions of the partial sums
        in.eps_abs = 2.f * sqrtf((float)d.n_embd);                                   // 2^-25 per router element that f16 flushes
    } else if (n_tokens >= 1024) {   // many tokens: tiled GEMM, one chain of n_embd additions per logit
        const dim3 grid((d.n_expert + 63) / 64, (n_tokens + 63) / 64);
        if (const cudaError_t e = launch_row_norm2(L, d, router_type, router, norm2, nullptr)) return e;
        if (router_type == QKM_TYPE_F32) logits_gemm_kernel<QKM_TYPE_F32><<<grid, 256, 0, L.stream>>>(r, x, logits, d.n_expert, d.n_embd, n_tokens);
        else logits_gemm_kernel<QKM_TYPE_F16><<<grid, 256, 0, L.stream>>>(r, x, logits, d.n_expert, d.n_embd, n_tokens);
        L.count();
        if (const cudaError_t e = cudaGetLastError()) return e;
        in.eps_terms = 2.f * ((float)d.n_embd + 8.f);
    } else {
        if (const cudaError_t e = launch_logits(L, d, router_type, router, x, logits, norm2, n_tokens)) return e;
        in.eps_terms = 2.f * (float)(d.n_embd / 32 + 8);
    }
    return launch_select_tokens(L, d, router_type, in, sel, n_tokens);
}

// ---- token-expert pair grouping: deterministic counting sort in one block --------------------
// offsets[e] .. offsets[e+1] delimit expert e's pairs; within a range pairs are in
// ascending (token, slot) order (the reference leaves the order unspecified,
// moe_group_pairs.comp:3-5).  With an expert-parallel view only resident experts
// get ranges, indexed from 0.
__global__ void __launch_bounds__(512)
group_pairs_kernel(const qkm_sel* __restrict__ sel, uint32_t n_tokens, uint32_t n_expert, uint32_t n_used,
                   uint32_t expert_first, uint32_t expert_count, uint32_t n_chunks, uint32_t stage_ids,
                   uint32_t* __restrict__ offsets, uint32_t* __restrict__ pairs) {
    extern __shared__ uint32_t s_dyn[];  // warp totals [16], counters [n_chunks][expert_count], totals
    uint32_t* s_scan = s_dyn;
    uint32_t* s_cnt = s_dyn + 16;
    uint32_t* s_tot = s_cnt + (size_t)n_chunks * expert_count;
    const uint32_t tid = threadIdx.x;
    const uint32_t np = n_tokens * n_used;
    const uint32_t chunk = (np + n_chunks - 1) / n_chunks;
    for (uint32_t i = tid; i < n_chunks * expert_count; i += 512) s_cnt[i] = 0;
    // small inputs: fetch every id once, all loads in flight together, and walk them from
    // shared memory afterwards
    uint32_t* s_ids = s_tot + expert_count;
    if (stage_ids)
        for (uint32_t p = tid; p < np; p += 512) {
            const uint32_t t = p / n_used, s = p - t * n_used;
            s_ids[p] = local_expert_of(sel[t].ids[s], n_expert, expert_first, expert_count);
        }
    __syncthreads();
    auto local_expert = [&](uint32_t p) -> uint32_t {
        if (stage_ids) return s_ids[p];
        const uint32_t t = p / n_used, s = p - t * n_used;
        return local_expert_of(sel[t].ids[s], n_expert, expert_first, expert_count);
    };
    const uint32_t p0 = tid * chunk, p1 = min(np, p0 + chunk);
    if (tid < n_chunks) {
        for (uint32_t p = p0; p < p1; ++p) {
            const uint32_t e = local_expert(p);
            if (e < expert_count) s_cnt[(size_t)tid * expert_count + e]++;
        }
    }
    __syncthreads();
    for (uint32_t e = tid; e < expert_count; e += 512) {
        uint32_t run = 0;
        for (uint32_t c = 0; c < n_chunks; ++c) {
            const uint32_t v = s_cnt[(size_t)c * expert_count + e];
            s_cnt[(size_t)c * expert_count + e] = run;
            run += v;
        }
        s_tot[e] = run;
    }
    __syncthreads();
    // exclusive scan of the per-expert totals (expert_count <= 512: one element per thread)
    const uint32_t mine = tid < expert_count ? s_tot[tid] : 0u;
    {
        // inclusive scan over 512 threads: shuffles inside each warp, then the 16 warp totals
        uint32_t v = mine;
        const uint32_t lane = tid & 31u, wrp = tid >> 5;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, v, o);
            if (lane >= (uint32_t)o) v += up;
        }
        if (lane == 31) s_scan[wrp] = v;
        __syncthreads();
        for (uint32_t w = 0; w < wrp; ++w) v += s_scan[w];
        if (tid < expert_count) { offsets[tid] = v - mine; s_tot[tid] = v - mine; }
        if (tid == 511) offsets[expert_count] = v;
    }
    __syncthreads();
    if (tid < n_chunks) {
        for (uint32_t p = p0; p < p1; ++p) {
            const uint32_t t = p / n_used, s = p - t * n_used;
            const uint32_t e = local_expert(p);
            if (e < expert_count) {
                const uint32_t dst = s_tot[e] + s_cnt[(size_t)tid * expert_count + e]++;
                pairs[dst] = (t << 4) | s;
            }
        }
    }
}

cudaError_t launch_group_pairs(const Launch& L, const qkm_dims& d, const qkm_sel* sel, uint32_t n_tokens,
                               uint32_t* offsets, uint32_t* pairs, uint32_t expert_first, uint32_t expert_count) {
    if (expert_count == 0) { expert_first = 0; expert_count = d.n_expert; }
    if (expert_count > 512) return cudaErrorInvalidValue;
    // one chunk of pairs per thread: enough chunks to spread the pairs, no more counters
    // than 32768 words of shared memory hold
    const uint32_t np = n_tokens * d.n_used;
    uint32_t n_chunks = 32768u / expert_count;
    if (n_chunks > 512) n_chunks = 512;
    const uint32_t want = (np + 7) / 8;
    if (n_chunks > want) n_chunks = want ? want : 1;
    const uint32_t stage_ids = np <= 8192 ? 1u : 0u;
    const size_t smem = ((size_t)n_chunks * expert_count + expert_count + 16 + (stage_ids ? np : 0)) * sizeof(uint32_t);
    cudaError_t e = cudaFuncSetAttribute(group_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)((32768 + 512 + 16 + 8192) * sizeof(uint32_t)));
    if (e != cudaSuccess) return e;
    group_pairs_kernel<<<1, 512, smem, L.stream>>>(sel, n_tokens, d.n_expert, d.n_used, expert_first,
                                                   expert_count, n_chunks, stage_ids, offsets, pairs);
    L.count();
    return cudaGetLastError();
}

}  // namespace qkm
