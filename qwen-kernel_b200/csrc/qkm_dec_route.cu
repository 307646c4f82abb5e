// Decode-sized batches (<= 64 tokens) of one or more layers: router logits, top-k selection, the pairs grouped by
// expert and the activation rows as int8 digit planes, in one launch.
//
// Replaces, for the fused decode sequence, moe_logits.comp + moe_select_256.comp, i.e. their
// fused form moe_route_select.comp.  Two kinds of blocks share the grid:
//   * logits blocks: pairs of router rows and up to eight tokens each, f64 accumulation - the logits are
//     those of the CPU reference's f64 router (src/main.cpp:1320-1324) up to the order of the
//     f64 additions, so they are ranked as they are, without an error bound; the block that
//     finishes a group of tokens last ranks them, one warp per token, and, of several layers, the one that ranks
//     a layer's last group groups the layer's pairs;
//   * one block per token encodes x as digit planes (and their negatives, which the IQ3_XXS
//     kernel multiplies with its sign masks) and evaluates the shared expert's gate
//     sigmoid(gis . x) in f64 (moe_select.comp's wShared).
#include "qkm_common.cuh"
#include "qkm_dec_rank.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"

namespace qkm {

namespace rd {
constexpr int kThreads = 256;
}  // namespace rd

// digit planes of one row, layout [kb][8][256]: planes 0..3 the digits, 4..7 their negatives
__device__ __forceinline__ void store_planes8(int8_t* __restrict__ pl, uint32_t k, uint32_t dgt) {
    int8_t* q = pl + (size_t)(k >> 8) * 2048 + (k & 255u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int dj = (int)(int8_t)((dgt >> (8 * j)) & 255u);
        q[256 * j] = (int8_t)dj;
        q[256 * (j + 4)] = (int8_t)(-dj);
    }
}

// The ticket's number.  Release and acquire for the device: what the block wrote before the barrier ahead of it is seen by the block
// that draws the last number, behind the barrier that follows.  (One such add for two fences by every thread: 0.3 us less.)
__device__ __forceinline__ uint32_t ticket(uint32_t* counter) {
    uint32_t n;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(n) : "l"(counter) : "memory");
    return n;
}
// TOK: tokens of a group; a.pairs_per_block: router row pairs that a logits block takes one after the other; KEEP: the tokens' x stays in
// registers as doubles for all of them
template <int TYPE, int TOK, bool KEEP>
__global__ void __launch_bounds__(rd::kThreads, 2)
route_decode_kernel(const __grid_constant__ RouteDecodeArgs a) {
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, layer = blockIdx.y;
    const qkm_dims d = a.d;
    const uint32_t T = a.n_tokens;
    const float* x = a.x + layer * a.x_stride;
    qkm_sel* sel = layer + 1 == a.n_layers ? a.sel_last : a.sel + (size_t)layer * T;
    double* logits = a.logits + (size_t)layer * T * d.n_expert;
    const uint32_t n_pairs = (d.n_expert + 1) / 2, n_pair_blocks = (n_pairs + a.pairs_per_block - 1) / a.pairs_per_block;   // blocks along the experts
    const uint32_t n_groups = (T + TOK - 1) / TOK, n_logit_blocks = n_pair_blocks * n_groups;                              // times the token groups

    __shared__ unsigned long long s_mask[rk::kMaxExperts];
    for (uint32_t e = tid; e < rk::kMaxExperts; e += rd::kThreads) s_mask[e] = 0ull;

    // x is the output of the kernel before; the selection, planes and logits written here are still
    // read by the previous layer's kernels until that kernel has ended
    pdl_wait();
    pdl_trigger();

    if (blockIdx.x >= n_logit_blocks) {
        // ---- one token: digit planes + shared gate ----------------------------------------------
        __shared__ uint32_t s_xm[16][8];
        __shared__ float s_up[16];
        __shared__ double s_sg[8];
        const uint32_t t = blockIdx.x - n_logit_blocks, KB = d.n_embd / 256;
        const float *xt = x + (size_t)t * d.n_embd, *gis = a.layer[layer].gis;
        float v[8];   // n_embd <= 2048: element tid of every 256 columns
        double dsg = 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t k = tid + 256 * i;
            v[i] = k < d.n_embd ? xt[k] : 0.f;
            if (k < d.n_embd) dsg += (double)gis[k] * (double)v[i];
        }
        // a scale per 256 columns: a large element costs the others of its own block bits, not the whole row
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (256u * i < d.n_embd) {
                const float ax = fabsf(v[i]);
                const uint32_t m = __reduce_max_sync(0xFFFFFFFFu, ax <= 3.0e38f ? __float_as_uint(ax) : 0x7F800000u);   // non-negative floats order like their bits
                if (lane == 0) s_xm[i][warp] = m;
            }
        dsg = warp_sum(dsg);
        if (lane == 0) s_sg[warp] = dsg;
        __syncthreads();
        if (tid < KB) {
            uint32_t m = 0;
#pragma unroll
            for (int w = 0; w < 8; ++w) m = max(m, s_xm[tid][w]);
            const bool bad = m >= 0x7F800000u;
            const int p = min(digit_exponent(__uint_as_float(m)), 126);
            s_up[tid] = bad ? 0.f : ldexpf(1.0f, p);   // (then NaN or zero times zero: digits of zero)
            a.xscale[(layer * T + t) * KB + tid] = bad ? __int_as_float(0x7FC00000) : ldexpf(1.0f, -p);
        } else if (tid == 32) {
            double sg = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) sg += s_sg[w];
            sel[t].w_shared = (float)(1.0 / (1.0 + exp(-sg)));
        }
        __syncthreads();
        int8_t* pl = a.planes + (size_t)(layer * T + t) * 8 * d.n_embd;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t k = tid + 256 * i;
            if (k < d.n_embd) store_planes8(pl, k, digits4(__float2int_rn(v[i] * s_up[i])));
        }
        return;
    }

    // ---- logits of pairs of experts for TOK tokens --------------------------------------------------
    // warp w owns the w-th eighth of the columns; a lane loads one 8-element unit of both router
    // rows and the matching x values of the block's tokens in one go; the next pair's rows are on their way meanwhile
    constexpr int NV = 2 * TOK, kLanes = 32 / NV;   // sums of a pair; lanes that end with the same one
    __shared__ double s_part[2][8][NV];
    const uint32_t p0 = blockIdx.x % n_pair_blocks * a.pairs_per_block, p1 = min(p0 + a.pairs_per_block, n_pairs), t0 = (blockIdx.x / n_pair_blocks) * TOK;
    const size_t rb = row_bytes(TYPE, d.n_embd);
    const uint8_t* router = a.layer[layer].w;
    const uint32_t units_w = d.n_embd / 64, k = (warp * units_w + lane) * 8;   // 8-element units of a warp: at most one a lane; its first column
    float w0[8], w1[8];
    auto rows = [&](uint32_t pair) {
        const uint8_t* row0 = router + (size_t)(2 * pair) * rb;
        dequant8<TYPE>(row0, k, w0);
        dequant8<TYPE>(2 * pair + 1 < d.n_expert ? row0 + rb : row0, k, w1);
    };
    if (lane < units_w) rows(p0);
    constexpr int kKept = KEEP ? TOK : 1;
    double xd[kKept][8];
    if (KEEP && lane < units_w) {
        float4 xa[kKept], xb[kKept];
#pragma unroll
        for (int j = 0; j < kKept; ++j) {
            const float* xt = x + (size_t)min(t0 + j, T - 1) * d.n_embd + k;
            xa[j] = *reinterpret_cast<const float4*>(xt);
            xb[j] = *reinterpret_cast<const float4*>(xt + 4);
        }
#pragma unroll
        for (int j = 0; j < kKept; ++j) {
            xd[j][0] = xa[j].x; xd[j][1] = xa[j].y; xd[j][2] = xa[j].z; xd[j][3] = xa[j].w;
            xd[j][4] = xb[j].x; xd[j][5] = xb[j].y; xd[j][6] = xb[j].z; xd[j][7] = xb[j].w;
        }
    }
    for (uint32_t pair = p0; pair < p1; ++pair) {
        double acc[NV];   // [expert 0: tokens][expert 1: tokens]
#pragma unroll
        for (int j = 0; j < NV; ++j) acc[j] = 0.0;
        if (KEEP) {
            if (lane < units_w) {
                float c0[8], c1[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) { c0[i] = w0[i]; c1[i] = w1[i]; }
                if (pair + 1 < p1) rows(pair + 1);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const double v0 = c0[i], v1 = c1[i];
#pragma unroll
                    for (int j = 0; j < kKept; ++j) { acc[j] += v0 * xd[j][i]; acc[TOK + j] += v1 * xd[j][i]; }
                }
            }
        } else
        if (lane < units_w) {
            constexpr int kHalf = TOK < 4 ? TOK : 4;   // four tokens' values at a time: more do not fit the registers
            float4 xa[kHalf], xb[kHalf];
            auto tokens = [&](int j0) {
#pragma unroll
                for (int j = 0; j < kHalf; ++j) {
                    const float* xt = x + (size_t)min(t0 + j0 + j, T - 1) * d.n_embd + k;
                    xa[j] = *reinterpret_cast<const float4*>(xt);
                    xb[j] = *reinterpret_cast<const float4*>(xt + 4);
                }
            };
            tokens(0);   // (on its way together with the rows: the conversions below wait for those)
            double v0[8], v1[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) { v0[i] = w0[i]; v1[i] = w1[i]; }
            if (pair + 1 < p1) rows(pair + 1);
#pragma unroll
            for (int j0 = 0; j0 < TOK; j0 += kHalf) {
                if (j0 > 0) tokens(j0);
#pragma unroll
                for (int j = 0; j < kHalf; ++j) {
                    const double xv[8] = {xa[j].x, xa[j].y, xa[j].z, xa[j].w, xb[j].x, xb[j].y, xb[j].z, xb[j].w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) { acc[j0 + j] += v0[i] * xv[i]; acc[TOK + j0 + j] += v1[i] * xv[i]; }
                }
            }
        }
        // reduce-scatter over the warp: after the step with distance o a lane keeps the half of its values selected by (lane & o); once one is
        // left, plain sums
        int n = NV;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            if (n > 1) {
                n >>= 1;
                const bool up = (lane & o) != 0;
#pragma unroll
                for (int j = 0; j < NV / 2; ++j)
                    if (j < n) {
                        const double send = up ? acc[j] : acc[j + n], keep = up ? acc[j + n] : acc[j];
                        acc[j] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
                    }
            } else {
                acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], o);
            }
        }
        double (&part)[8][NV] = s_part[pair & 1u];   // two: a pair's sums are read while the next one's are written
        if (lane % kLanes == 0) part[warp][lane / kLanes] = acc[0];
        __syncthreads();
        if (tid < NV) {
            const uint32_t r = tid / TOK, j = tid % TOK;
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) v += part[w][tid];
            if (t0 + j < T && 2 * pair + r < d.n_expert) logits[(size_t)(t0 + j) * d.n_expert + 2 * pair + r] = v;
        }
    }

    // ---- the block that finishes a token group's logits last ranks the group's tokens ---------------
    // (a ticket counter per group, taken by one thread between two barriers: the block's writes come before it, the
    // reads after it - the device-scope release/acquire the reference's fused router relies on, moe_route_select.comp:56-67)
    __shared__ uint32_t s_last;
    uint32_t* counter = a.counter + layer * kDecCounters + blockIdx.x / n_pair_blocks;
    __syncthreads();
    if (tid == 0) s_last = ticket(counter) == n_pair_blocks - 1 ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    if (tid == 0) *counter = 0;   // ready for the next launch
    __shared__ uint16_t s_ids[rk::kMaxTokens * 16];
    static_assert(TOK <= rd::kThreads / 32, "a warp ranks one token");
    const bool ranks = warp < min((uint32_t)TOK, T - t0), lists = a.groups.group != nullptr;
    const uint32_t my_t = t0 + warp;
    Ranked mine{};
    if (ranks) {
        mine = rank_token(logits + (size_t)my_t * d.n_expert, d);
        if (n_groups > 1 || !lists) rank_store(mine, sel[my_t], d);
        else if (lane < d.n_used) choose(s_mask, s_ids, my_t, lane, mine.id);
    }
    if (!lists) return;

    // ---- and the block that ranks a layer's last token group groups the layer's pairs --------------
    if (n_groups > 1) {   // (the only group's ids are in shared memory)
        __syncthreads();
        uint32_t* groups_done = a.counter + layer * kDecCounters + kDecCounters - 1;
        if (tid == 0) s_last = ticket(groups_done) == n_groups - 1 ? 1u : 0u;
        __syncthreads();
        if (!s_last) return;
        if (tid == 0) *groups_done = 0;
        for (uint32_t i = tid; i < T * 16; i += rd::kThreads)
            if ((i & 15u) < d.n_used) choose(s_mask, s_ids, i >> 4, i & 15u, min(__ldcg(&sel[i >> 4].ids[i & 15u]), d.n_expert - 1));
    }
    __syncthreads();
    __shared__ uint32_t s_sum[rd::kThreads / 32], s_first[rk::kMaxExperts];
    const uint32_t n = group_pairs<rd::kThreads>(a.groups.group + (size_t)layer * T * (d.n_used + 1), s_first, s_sum, s_ids, s_mask, d.n_used, T * d.n_used, T, layer);
    if (tid == 0) a.groups.count[layer] = n;
    if (n_groups == 1 && ranks) rank_store(mine, sel[my_t], d);   // (after the lists: the next kernel waits for those)
}

bool route_decode_ok(const qkm_dims& d) { return d.n_expert <= rk::kMaxExperts && d.n_embd <= 2048; }

// Tokens of a group: as few as the batch has (a group of eight costs one token as much as eight).  Pairs a block: one for a layer on its own and while
// the blocks find room on the SMs at once (a chain of latencies: start-up, loads, ticket), more when layers go together, so that a block's share of
// that chain is small: 40 layers of 16 tokens 159 us with one pair a block, 119 so.  About kBlocks blocks: with half as many 24 layers of one token
// 117 -> 119 us for the whole call, 12 of one 71 -> 74, 6 of 12 243 -> 250; with twice as many 24 of one 117 -> 120, 24 of 5 413 -> 422, 6 of 16
// 301 -> 308 (but 4 of 3, 512 experts, 85 -> 82).  At most 8, 16 or 32 pairs a block: the same.
// Blocks of several pairs keep the x of up to four tokens as doubles (the converter takes 16 lanes a cycle and SM, the f64 units 64): 24 layers of
// one token 124 -> 119 us, and so groups of four go ahead of groups of eight where they find several pairs a block: 12 layers of 64 tokens
// 1,712 -> 1,669, 4 of 12 173 -> 170, 2 of 9 (512 experts) 114 -> 111.  With one pair a block there is nothing to keep it for, and groups of four are
// more blocks than one of eight is worth (2 layers of 16 tokens 121 -> 124, a step of 3 tokens with it kept 341 -> 348).
template <int TYPE, int TOK, bool KEEP>
static cudaError_t route_launch(const Launch& L, const RouteDecodeArgs& a, uint32_t groups) {
    const uint32_t pairs = (a.d.n_expert + 1) / 2;
    const dim3 grid((pairs + a.pairs_per_block - 1) / a.pairs_per_block * groups + a.n_tokens, a.n_layers);
    return launch_kernel(L, route_decode_kernel<TYPE, TOK, KEEP>, grid, dim3(rd::kThreads), 0, a);
}
template <int TYPE>
static cudaError_t route_launch(const Launch& L, RouteDecodeArgs a) {
    constexpr uint32_t kBlocks = 600, kMostPairs = 16;
    const uint32_t T = a.n_tokens, pairs = (a.d.n_expert + 1) / 2;
    const bool four = a.n_layers > 1 && T > 8 && pairs * ((T + 3) / 4) * a.n_layers >= 2 * kBlocks;
    const uint32_t tok = T <= 1 ? 1 : T <= 2 ? 2 : T <= 4 || four ? 4 : 8, groups = (T + tok - 1) / tok, per = a.n_layers == 1 ? 1 : pairs * groups * a.n_layers / kBlocks;
    a.pairs_per_block = per < 1 ? 1 : per < kMostPairs ? per : kMostPairs;
    const bool keep = a.pairs_per_block > 1;
    switch (tok) {
        case 1: return keep ? route_launch<TYPE, 1, true>(L, a, groups) : route_launch<TYPE, 1, false>(L, a, groups);
        case 2: return keep ? route_launch<TYPE, 2, true>(L, a, groups) : route_launch<TYPE, 2, false>(L, a, groups);
        case 4: return keep ? route_launch<TYPE, 4, true>(L, a, groups) : route_launch<TYPE, 4, false>(L, a, groups);
        default: return route_launch<TYPE, 8, false>(L, a, groups);
    }
}
cudaError_t launch_route_decode(const Launch& L, uint32_t router_type, const RouteDecodeArgs& a) {
    if (router_type != QKM_TYPE_F32 && router_type != QKM_TYPE_F16) return cudaErrorInvalidValue;
    if (a.n_tokens == 0 || a.n_tokens > rk::kMaxTokens || !route_decode_ok(a.d) || a.n_layers == 0 || a.n_layers > kDecMaxLayers) return cudaErrorInvalidValue;
    const cudaError_t e = router_type == QKM_TYPE_F32 ? route_launch<QKM_TYPE_F32>(L, a) : route_launch<QKM_TYPE_F16>(L, a);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace qkm
