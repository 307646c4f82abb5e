// Inner steps the decode down kernels share: IQ4_XS and Q6_K quants as int8 MMA operands.
#pragma once

#include "qkm_stream.cuh"

namespace qkm {

__device__ __forceinline__ uint32_t prmt_dec(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// The eight sub-block scales ls - 32 of one row as int8: even sub-blocks 0,2,4,6 in ev, odd 1,3,5,7 in od.
// sl: scales_l (eight 4-bit fields), sh: scales_h (eight 2-bit fields)  (src/quants.h:107-113, :139-146)
__device__ __forceinline__ void iq4_scales(uint32_t sl, uint32_t sh, uint32_t& ev, uint32_t& od) {
    const uint32_t r = prmt_dec(sh, 0u, 0x1100u);                       // bytes (B0, B0, B1, B1) of scales_h
    const uint32_t he = ((r << 4) & 0x00300030u) | (r & 0x30003000u);  // top two bits of sub-blocks 0,2,4,6 at bits 4..5
    const uint32_t ho = ((r << 2) & 0x00300030u) | ((r >> 2) & 0x30003000u);
    const uint32_t te = ((sl & 0x0F0F0F0Fu) | he) ^ 0x20202020u;       // ls ^ 32 per byte
    const uint32_t to = (((sl >> 4) & 0x0F0F0F0Fu) | ho) ^ 0x20202020u;
    // ls - 32 as int8: bit 5 of (ls ^ 32) extended into bits 6..7 (no carry leaves a byte)
    ev = (te & 0x20202020u) * 6u + te;
    od = (to & 0x20202020u) * 6u + to;
}

// Eight IQ4_XS weights of one quant word (elements e0 .. e7 = 8t .. 8t+7 of a sub-block; a byte's nibbles are two
// elements apart, see qkm_tiles.cuh) as two int8 MMA A-operand registers: lo = (e0, e2, e1, e3), hi = (e4, e6, e5, e7).
// tab_c: bytes (lane * 4, -, 0x01, 0x00): with a quant byte in byte 1 it is that byte's table entry for this lane.
__device__ __forceinline__ void iq4_word(uint32_t w, uint32_t tab_c, uint32_t& lo, uint32_t& hi) {
    const uint32_t e0 = lds32(prmt_dec(w, tab_c, 0x7604u)), e1 = lds32(prmt_dec(w, tab_c, 0x7614u));
    const uint32_t e2 = lds32(prmt_dec(w, tab_c, 0x7624u)), e3 = lds32(prmt_dec(w, tab_c, 0x7634u));
    lo = prmt_dec(e0, e1, 0x5410u);
    hi = prmt_dec(e2, e3, 0x5410u);
}

// Sixteen Q6_K weights as four int8 MMA A-operand registers, each 4 * (q - 32): w1 / w2 are the ql
// words of elements l..l+3 in the first / second 32-byte run of a half, hq the qh word of the same
// l; r[qd] holds elements l + 32 * qd .. + 3  (src/quants.h:148-163).
__device__ __forceinline__ void q6k_words(uint32_t w1, uint32_t w2, uint32_t hq, uint32_t (&r)[4]) {
    const uint32_t hx = hq ^ 0xAAAAAAAAu;          // top bit of every pair flipped: the sign of q - 32
    const uint32_t lo1 = w1 & 0x0F0F0F0Fu, hi1 = w1 & 0xF0F0F0F0u;
    const uint32_t lo2 = w2 & 0x0F0F0F0Fu, hi2 = w2 & 0xF0F0F0F0u;
    r[0] = ((hx << 6) & 0xC0C0C0C0u) | (lo1 << 2);
    r[1] = ((hx << 4) & 0xC0C0C0C0u) | (lo2 << 2);
    r[2] = ((hx << 2) & 0xC0C0C0C0u) | (hi1 >> 2);
    r[3] = (hx & 0xC0C0C0C0u) | (hi2 >> 2);
}

}  // namespace qkm
