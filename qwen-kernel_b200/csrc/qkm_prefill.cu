// Batched prefill around the expert GEMMs (qkm_wgemm.cu): the router logits on the tensor cores and the slot-order fold
// of add_rms3_grouped.comp:22-27.
#include <cuda_fp16.h>

#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"
#include "qkm_tiles.cuh"
#include "qkm_umma.cuh"

namespace qkm {

namespace pf {
constexpr int kThreads = 256;                  // copying threads of the logits kernel; one more warp issues the MMAs
constexpr int kBlock = kThreads + 32;
constexpr int kTileBytes = 128 * 128;          // 128 rows x 64 f16
}  // namespace pf

// ---- router logits on the tensor cores -----------------------------------------------------------------
// logits[t][e] = router[e] . x[t] with f16 operands (router rows as written by router_f16_kernel, x rows by
// f16_rows_kernel: the same element order) and f32 accumulation in tensor
// memory.  These logits only pre-select: the selection kernel re-evaluates every expert within
// its error bound of the k-th in f64, so the bound has to hold, not the last bits.
// Error per logit <= (2^-11 [x rounding] + 2^-11 [router rounding] + K * 2^-22 [accumulation, measured 2^-25])
// * |w| * |x|, below 2^-9 * |w| * |x| for K <= 4096.
// Block = 128 experts (M) x up to 128 tokens (N); 256 producer threads copy both operand tiles
// into the swizzled layout, the ninth warp issues the MMAs.
constexpr int kLgStages = 4;   // stages of the logits kernel (one block per SM: it is a small grid)
constexpr int kLgDepth = 3;    // k-steps of asynchronous copies in flight

__device__ __forceinline__ void cp_async16(uint32_t smem_dst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

__global__ void __launch_bounds__(pf::kBlock, 1)
logits_mma_kernel(const uint8_t* __restrict__ router, const __half* __restrict__ xh, const float* __restrict__ x_inv_scale,
                  float* __restrict__ logits_all, uint32_t n_expert, uint32_t K_all, uint32_t n_tokens, uint32_t* __restrict__ status) {
    // blockIdx.z: the column range [z, z+1) * K_all / gridDim.z; its partial logits go to part z of the output
    const uint32_t K = K_all / gridDim.z;
    float* __restrict__ logits = logits_all + (size_t)blockIdx.z * n_tokens * n_expert;
    router += (size_t)blockIdx.z * K * 2;
    xh += (size_t)blockIdx.z * K;
    extern __shared__ __align__(1024) uint8_t smem_dyn[];
    __shared__ __align__(8) unsigned long long s_bar[2 * kLgStages + 1];  // empty[stage], full[stage], done
    __shared__ uint32_t s_tmem;
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t t0 = blockIdx.x * 128u, e0 = blockIdx.y * 128u;
    const uint32_t n = min(128u, n_tokens - t0), n_mma = (n + 15u) & ~15u, KS = K / 64;
    if (tid == 0) {
        for (int s = 0; s < kLgStages; ++s) {
            mbar_init(smem_addr(&s_bar[s]), 1);
            mbar_init(smem_addr(&s_bar[kLgStages + s]), pf::kThreads);
        }
        mbar_init(smem_addr(&s_bar[2 * kLgStages]), 1);
        mbar_fence_init();
    }
    if (warp == 0) { umma::tmem_alloc(smem_addr(&s_tmem), 128); umma::tmem_relinquish(); }
    umma::fence_before_sync();
    pdl_trigger();
    pdl_wait();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = s_tmem;
    const uint32_t idesc = umma::instr_desc_f16(n_mma);
    bool timed_out = false;
    if (tid >= pf::kThreads) {
        if (lane == 0) {
            for (uint32_t ks = 0; ks < KS; ++ks) {
                const uint32_t stage = ks % kLgStages;
                if (!mbar_wait_bounded(smem_addr(&s_bar[kLgStages + stage]), (ks / kLgStages) & 1u)) timed_out = true;
                umma::fence_after_sync();
                const uint32_t a = smem_addr(smem + stage * 2 * pf::kTileBytes), b = a + pf::kTileBytes;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    umma::mma_f16_ss(tmem, umma::smem_desc(a + 32 * j), umma::smem_desc(b + 32 * j), idesc, (ks | (uint32_t)j) != 0);
                umma::commit(smem_addr(&s_bar[stage]));
                if (ks + 1 == KS) umma::commit(smem_addr(&s_bar[2 * kLgStages]));
            }
        }
    } else {
        {
            // Both operands are plain copies: 16-byte asynchronous copies straight into the
            // swizzled tiles, kLgDepth k-steps in flight, so the global-load latency of a
            // block that has the SM almost to itself (small batches) is hidden.
            auto issue = [&](uint32_t ks) {
                const uint32_t stage = ks % kLgStages;
                if (ks >= (uint32_t)kLgStages)
                    if (!mbar_wait_bounded(smem_addr(&s_bar[stage]), ((ks / kLgStages) - 1) & 1u)) timed_out = true;
                const uint32_t st = smem_addr(smem + stage * 2 * pf::kTileBytes), k0 = ks * 64;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t qd = tid + i * pf::kThreads, row = qd >> 3, c = qd & 7u;
                    cp_async16(st + umma::sw128_chunk(row, c), router + ((size_t)(e0 + row) * K_all + k0 + 8 * c) * 2);
                    if (qd < n_mma * 8) {
                        const uint32_t src_row = row < n ? row : 0u;   // rows past n feed accumulator columns nobody reads
                        cp_async16(st + pf::kTileBytes + umma::sw128_chunk(row, c), xh + (size_t)(t0 + src_row) * K_all + k0 + 8 * c);
                    }
                }
                cp_async_commit();
            };
            for (uint32_t ks = 0; ks < (uint32_t)kLgDepth; ++ks)
                if (ks < KS) issue(ks); else cp_async_commit();
            for (uint32_t ks = 0; ks < KS; ++ks) {
                if (ks + kLgDepth < KS) issue(ks + kLgDepth); else cp_async_commit();   // keep the group count in step
                cp_async_wait<kLgDepth>();          // the copies of step ks have landed
                umma::fence_smem_to_async();
                mbar_arrive(smem_addr(&s_bar[kLgStages + ks % kLgStages]));
            }
        }
        if (!mbar_wait_bounded(smem_addr(&s_bar[2 * kLgStages]), 0)) timed_out = true;
        umma::fence_after_sync();
        const uint32_t lg = warp & 3u, e = e0 + 32 * lg + lane;
        for (uint32_t cb = warp >> 2; cb < n_mma / 16; cb += 2) {
            uint32_t v[16];
            umma::tmem_ld16(tmem + ((32 * lg) << 16) + cb * 16, v);
            umma::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const uint32_t col = cb * 16 + i;
                if (col < n) logits[(size_t)(t0 + col) * n_expert + e] = __uint_as_float(v[i]) * x_inv_scale[t0 + col];
            }
        }
    }
    umma::fence_before_sync();
    // any thread's wait that ran out counts (the MMA issuer's too, not only thread 0's)
    const int any_timed_out = __syncthreads_or(timed_out ? 1 : 0);
    if (warp == 0) umma::tmem_dealloc(tmem, 128);
    if (any_timed_out && tid == 0) atomicExch(status, (uint32_t)kStatusWaitTimeout);
}

cudaError_t launch_logits_mma(const Launch& L, const qkm_dims& d, const void* router_f16,
                              const void* x_f16, const float* x_inv_scale, float* logits, uint32_t n_tokens,
                              uint32_t* status, uint32_t splits) {
    if (n_tokens == 0) return cudaSuccess;
    if (d.n_expert % 128 || d.n_embd % 64 || d.n_embd > 4096 || splits == 0 || (d.n_embd / 64) % splits) return cudaErrorInvalidValue;
    const size_t smem = (size_t)kLgStages * 2 * pf::kTileBytes + 1024;
    const dim3 grid((n_tokens + 127) / 128, d.n_expert / 128, splits);
    if (const cudaError_t e = allow_dynamic_smem<logits_mma_kernel>((int)smem)) return e;
    const cudaError_t e = launch_kernel(Launch{L.stream, nullptr, true}, logits_mma_kernel, grid, dim3(pf::kBlock), smem, (const uint8_t*)router_f16, (const __half*)x_f16,
                                        x_inv_scale, logits, d.n_expert, d.n_embd, n_tokens, status);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}

// router rows as f16 in the element order of the f16 activation rows (0, 2, 1, 3 in every group of four)
template <int TYPE>
__global__ void router_f16_kernel(const uint8_t* __restrict__ router, __half* __restrict__ out, uint64_t n8) {
    const uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n8) return;
    float w[8];
    dequant8<TYPE>(router + u * 8 * (TYPE == QKM_TYPE_F32 ? 4 : 2), 0, w);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[u * 8 + (i & 4) + ((i & 1) << 1) + ((i >> 1) & 1)] = __float2half_rn(w[i]);
}
cudaError_t launch_router_f16(const Launch& L, uint32_t router_type, const void* router, void* out, uint64_t n_elems) {
    const uint64_t n8 = n_elems / 8;
    if (router_type == QKM_TYPE_F32) router_f16_kernel<QKM_TYPE_F32><<<(unsigned)((n8 + 255) / 256), 256, 0, L.stream>>>((const uint8_t*)router, (__half*)out, n8);
    else if (router_type == QKM_TYPE_F16) router_f16_kernel<QKM_TYPE_F16><<<(unsigned)((n8 + 255) / 256), 256, 0, L.stream>>>((const uint8_t*)router, (__half*)out, n8);
    else return cudaErrorInvalidValue;
    L.count();
    return cudaGetLastError();
}

// ---- fold: y[t] = sum over slots (in order) of contrib[pos(t,s)], then the shared expert -----------------
__global__ void fold_pairs_kernel(const float* contrib, const uint32_t* pos_of,
                                  float* __restrict__ y, uint32_t n_used, uint32_t n_embd) {
    pdl_trigger();
    pdl_wait();
    const uint32_t t = blockIdx.y;
    const uint32_t o = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (o >= n_embd) return;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t s = 0; s <= n_used; ++s) {
        const uint32_t p = pos_of[t * (n_used + 1) + s];
        if (p == 0xFFFFFFFFu) continue;
        const float4 c = *reinterpret_cast<const float4*>(contrib + (size_t)p * n_embd + o);
        v.x += c.x; v.y += c.y; v.z += c.z; v.w += c.w;
    }
    *reinterpret_cast<float4*>(y + (size_t)t * n_embd + o) = v;
}

// The same sum for an expert-parallel shard whose rows are slots (source rank s, token i): the
// row goes straight into rank s's return buffer, at (this rank, i), over the peer mapping; a
// slot none of whose pairs ran here is not written (its owner does not read it).
__global__ void fold_pairs_peer_kernel(const float* __restrict__ contrib, const uint32_t* __restrict__ pos_of,
                                       EpPeerTable peers, uint32_t slot_rows, uint32_t rank, uint32_t n_used,
                                       uint32_t n_embd) {
    const uint32_t t = blockIdx.y;
    const uint32_t o = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (o >= n_embd) return;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    bool any = false;
    for (uint32_t s = 0; s <= n_used; ++s) {
        const uint32_t p = pos_of[t * (n_used + 1) + s];
        if (p == 0xFFFFFFFFu) continue;
        any = true;
        const float4 c = *reinterpret_cast<const float4*>(contrib + (size_t)p * n_embd + o);
        v.x += c.x; v.y += c.y; v.z += c.z; v.w += c.w;
    }
    if (!any) return;
    const uint32_t src = t / slot_rows, i = t - src * slot_rows;
    *reinterpret_cast<float4*>(peers.back[src] + ((size_t)rank * slot_rows + i) * n_embd + o) = v;
}

// ---- launchers ---------------------------------------------------------------------------------------------
cudaError_t launch_fold_pairs(const Launch& L, const qkm_dims& d, const float* contrib, const uint32_t* pos_of,
                              float* y, uint32_t n_tokens) {
    if (n_tokens == 0) return cudaSuccess;
    const dim3 grid((d.n_embd / 4 + 255) / 256, n_tokens);
    const cudaError_t e = launch_kernel(Launch{L.stream, nullptr, true}, fold_pairs_kernel, grid, dim3(256), 0, contrib, pos_of, y, d.n_used, d.n_embd);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_fold_pairs_peer(const Launch& L, const qkm_dims& d, const float* contrib, const uint32_t* pos_of,
                                   const EpPeerTable& peers, uint32_t slot_rows, uint32_t rank, uint32_t n_ranks) {
    if (slot_rows == 0 || n_ranks == 0 || n_ranks > kMaxPeerRanks || rank >= n_ranks) return cudaErrorInvalidValue;
    const dim3 grid((d.n_embd / 4 + 255) / 256, n_ranks * slot_rows);
    fold_pairs_peer_kernel<<<grid, 256, 0, L.stream>>>(contrib, pos_of, peers, slot_rows, rank, d.n_used, d.n_embd);
    L.count();
    return cudaGetLastError();
}

}  // namespace qkm
