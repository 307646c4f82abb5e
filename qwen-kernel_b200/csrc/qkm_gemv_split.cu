// Dense dequant-GEMV for 1 to 16 activation rows, K split over a cluster of blocks.
//
// Contract of the other GEMV kernels: y[n][M] = W[M][K] . x[n][K] on raw ggml rows, z-batched over n
// (shaders/gemv_q8_0.comp:31-32 and its siblings).
//
// Every weight is unpacked once for all n rows: the unpacked weights of 16 rows are the A operand of
// mma.sync MMAs, the activations the B operand - for the quantised formats x as four int8 digit
// planes (27-bit fixed point relative to the largest of 256 columns, qkm_stream.cuh), for F16 weights x as
// three f16 pieces (33 significant bits) - so a row of x takes four of the eight MMA columns and an
// unpacked fragment is multiplied with NT column tiles (2 NT rows of x).  Integer sums are exact; one f32
// rounding per 256 columns and row.
//
// Split.  A block owns a slice of the columns (KB / KS blocks of 256) and walks 16-row tiles, one per warp
// at a time; the KS blocks of a cluster own the slices of the same rows and add their partial sums through
// distributed shared memory.  What sets the time of a small matrix is latency, not bytes (4096 x 2048 is
// 0.5 to 2.6 us of HBM time): with K split over blocks every SM has work for all its warps at 4096 rows, and
// a block encodes only its own slice of x, which for 16 rows would otherwise cost more than the weights.
// (4096 x 2048, 16 rows: 10.3 to 13.1 us by format, where re-reading and re-decoding the matrix for every row took
// about 160; one row 6.3 to 6.9 us.)  For 16 rows of a large matrix issue slots are the bound (55 % busy, 32768 x 2048 Q8_0
// 40 us): four of the instructions of every 32-column step repeat for each column tile.
// A tile's bytes come in with 16-byte cp.async (the 16-byte units that cover a row's slice; ggml rows are
// only 2-byte aligned), one tile ahead, into a buffer of the warp's own; F16 rows are loaded to registers.
#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_stream.cuh"

namespace qkm {

namespace gs {
constexpr int kMaxWarps = 16;

template <int TYPE> struct Geo;   // bytes per 256 columns, staged bytes per row (stride: conflict-free over the 8 row groups), 16-byte units
template <> struct Geo<QKM_TYPE_Q8_0>    { static constexpr int kBytes = 272, kStride = 272, kUnits = 17; };
template <> struct Geo<QKM_TYPE_Q6_K>    { static constexpr int kBytes = 210, kStride = 240, kUnits = 15; };
template <> struct Geo<QKM_TYPE_IQ4_XS>  { static constexpr int kBytes = 136, kStride = 144, kUnits = 9; };
template <> struct Geo<QKM_TYPE_IQ3_XXS> { static constexpr int kBytes = 98,  kStride = 144, kUnits = 8; };
template <> struct Geo<QKM_TYPE_F16>     { static constexpr int kBytes = 512, kStride = 0,   kUnits = 0; };

// bytes of B fragments per 256 columns and column tile: eight 32-column steps of 32 lanes x 8 bytes (int8), twice that for f16
template <int TYPE> constexpr uint32_t frag_bytes() { return TYPE == QKM_TYPE_F16 ? 4096u : 2048u; }
}  // namespace gs

__device__ __forceinline__ uint32_t prmt_gs(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sts8(uint32_t addr, uint32_t v) { asm volatile("st.shared.b8 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
// a 32-bit word at a 2-byte aligned shared address
__device__ __forceinline__ uint32_t lds32_u2(uint32_t addr) {
    const uint32_t a = addr & ~3u;
    return __funnelshift_r(lds32(a), lds32(a + 4), (addr & 2u) * 8u);
}
// D(16x8, s32) = A(16x16, s8, row) * B(16x8, s8, col)
__device__ __forceinline__ void mma_s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
// D(16x8, f32) = A(16x16, f16, row) * B(16x8, f16, col)
__device__ __forceinline__ void mma_f16_k16_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// (a0, a1) += (b0, b1), one instruction
__device__ __forceinline__ void add_f32x2(float& a0, float& a1, float b0, float b1) {
    asm("{\n.reg .b64 x, y;\nmov.b64 x, {%0,%1};\nmov.b64 y, {%2,%3};\nadd.rn.f32x2 x, x, y;\nmov.b64 {%0,%1}, x;\n}\n" : "+f"(a0), "+f"(a1) : "f"(b0), "f"(b1));
}

// Eight consecutive columns (8 * lane ..) of one activation row into the B fragments of one 256-column block.
// frag: this block's and this row's column tile; cg: the row's first column (0 or 4) in the tile.
template <int TYPE>
__device__ __forceinline__ void encode_fragments(const float (&v)[8], uint32_t lane, uint32_t frag, uint32_t cg, float up) {
    const uint32_t sb = lane >> 2, e = (lane & 3u) * 8u;   // 32-column step, first column inside it
    if (TYPE == QKM_TYPE_F16) {
        // lane t of a step owns columns 8t .. 8t+7 (one 16-byte load of the weight row): MMA 2s takes 8t..8t+3, MMA 2s+1 the rest
        const uint32_t at = frag + sb * 512u + (cg * 4u + (lane & 3u)) * 16u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // column pairs
            float r0 = v[2 * j] * up, r1 = v[2 * j + 1] * up;
#pragma unroll
            for (int p = 0; p < 4; ++p) {   // pieces: hi, mid * 2^11, lo * 2^22, nothing
                uint32_t w = 0;
                if (p < 3) {
                    const __half2 h = __floats2half2_rn(r0, r1);
                    w = *reinterpret_cast<const uint32_t*>(&h);
                    r0 = (r0 - __low2float(h)) * 2048.f; r1 = (r1 - __high2float(h)) * 2048.f;
                }
                sts32(at + p * 64u + j * 4u, w);
            }
        }
        return;
    }
    uint32_t d[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) d[i] = digits4(__float2int_rn(v[i] * up));
#pragma unroll
    for (int h = 0; h < 2; ++h) {       // columns e + 4h .. e + 4h + 3
        // transpose four packed digit words: word j = digit j of the four columns
        const uint32_t x0 = prmt_gs(d[4 * h], d[4 * h + 1], 0x5140u), x1 = prmt_gs(d[4 * h + 2], d[4 * h + 3], 0x5140u);
        const uint32_t y0 = prmt_gs(d[4 * h], d[4 * h + 1], 0x7362u), y1 = prmt_gs(d[4 * h + 2], d[4 * h + 3], 0x7362u);
        const uint32_t w[4] = {prmt_gs(x0, x1, 0x5410u), prmt_gs(x0, x1, 0x7632u), prmt_gs(y0, y1, 0x5410u), prmt_gs(y0, y1, 0x7632u)};
        const uint32_t c = e + 4 * h;   // 0, 4, .., 28
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t row = frag + sb * 256u + (cg + j) * 32u;
            if (TYPE == QKM_TYPE_IQ3_XXS) {            // lane t owns columns 8t .. 8t+7
                sts32(row + (c >> 3) * 8u + (c & 4u), w[j]);
            } else if (TYPE == QKM_TYPE_IQ4_XS) {      // order (4t, 16+4t, 4t+1, 17+4t | 4t+2, 18+4t, 4t+3, 19+4t), see iq4_pairs
                const uint32_t at = row + ((c & 15u) >> 2) * 8u + (c >> 4);
                sts8(at, w[j]); sts8(at + 2, w[j] >> 8); sts8(at + 4, w[j] >> 16); sts8(at + 6, w[j] >> 24);
            } else {                                   // Q8_0, Q6_K: b0 = columns 4t.., b1 = 16 + 4t..
                sts32(row + ((c & 15u) >> 2) * 8u + (c >> 4) * 4u, w[j]);
            }
        }
    }
}

// Sums of one 16-row x 256-column tile: f[nt][0] += row g, f[nt][1] += row g + 8, this lane's digit pair (or piece pair)
// of x row 2 nt + t / 2.  r0 / r1: the shared address of the block of rows g / g + 8.  bf: fragments of the 256 columns, + 8 * lane.
template <int TYPE, int NT>
__device__ __forceinline__ void tile_sums(uint32_t r0, uint32_t r1, uint32_t bf, uint32_t t, uint32_t lut, const float (&sc)[NT], float dw0,
                                          float dw1, float (&f)[NT][2]) {
    constexpr uint32_t kNt = gs::frag_bytes<TYPE>();   // from one column tile to the next
    if constexpr (TYPE == QKM_TYPE_Q8_0) {
        float q[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) q[nt][0] = q[nt][1] = 0.f;
#pragma unroll
        for (int sb = 0; sb < 8; ++sb) {
            const uint32_t p0 = r0 + 34u * sb, p1 = r1 + 34u * sb;
            uint32_t a0, a1, a2, a3, h0, h1;
            if ((sb & 1) == 0) {   // rows are 16-byte aligned: even blocks start on a word, their quants two bytes into it
                h0 = lds32(p0) & 0xFFFFu; h1 = lds32(p1) & 0xFFFFu;
                a0 = __funnelshift_r(lds32(p0 + 4 * t), lds32(p0 + 4 * t + 4), 16); a1 = __funnelshift_r(lds32(p1 + 4 * t), lds32(p1 + 4 * t + 4), 16);
                a2 = __funnelshift_r(lds32(p0 + 16 + 4 * t), lds32(p0 + 20 + 4 * t), 16); a3 = __funnelshift_r(lds32(p1 + 16 + 4 * t), lds32(p1 + 20 + 4 * t), 16);
            } else {
                h0 = lds32(p0 - 2) >> 16; h1 = lds32(p1 - 2) >> 16;
                a0 = lds32(p0 + 2 + 4 * t); a1 = lds32(p1 + 2 + 4 * t);
                a2 = lds32(p0 + 18 + 4 * t); a3 = lds32(p1 + 18 + 4 * t);
            }
            const float d0 = f16_bits_to_f32(h0), d1 = f16_bits_to_f32(h1);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint2 b = lds64(bf + nt * kNt + sb * 256u);
                int c[4];
                mma_s8_first(c, a0, a1, a2, a3, b.x, b.y);
                q[nt][0] += d0 * (float)(c[0] + (c[1] << 7));   // this lane's two digits, exact
                q[nt][1] += d1 * (float)(c[2] + (c[3] << 7));
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) { f[nt][0] += q[nt][0] * (sc[nt] * dw0); f[nt][1] += q[nt][1] * (sc[nt] * dw0); }
        return;
    }
    int acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0;
    float d0, d1;
    if constexpr (TYPE == QKM_TYPE_Q6_K) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const uint32_t q0 = r0 + 64 * hf + 4 * t, h0 = r0 + 128 + 32 * hf + 4 * t, q1 = r1 + 64 * hf + 4 * t, h1 = r1 + 128 + 32 * hf + 4 * t;
            uint32_t wl[2][2][2], wh[2][2], s[2][2];   // [row][run][16-column half], [row][half]; scales of the half's eight groups
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const uint32_t q = v ? q1 : q0, h = v ? h1 : h0, b = v ? r1 : r0;
                wl[v][0][0] = lds32_u2(q); wl[v][0][1] = lds32_u2(q + 16); wl[v][1][0] = lds32_u2(q + 32); wl[v][1][1] = lds32_u2(q + 48);
                wh[v][0] = lds32_u2(h); wh[v][1] = lds32_u2(h + 16);
                s[v][0] = lds32_u2(b + 192 + 8 * hf); s[v][1] = lds32_u2(b + 196 + 8 * hf);
            }
#pragma unroll
            for (int qd = 0; qd < 4; ++qd) {
#pragma unroll
                for (int m = 0; m < 2; ++m) {   // columns 128 hf + 32 qd + 16 m ..: 6-bit values in the top bits of a byte, top bit flipped = 4 (q - 32)
                    uint32_t a[2];
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const uint32_t w = wl[v][qd & 1][m], hx = wh[v][m] ^ 0xAAAAAAAAu;
                        const uint32_t top = (qd == 0 ? hx << 6 : qd == 1 ? hx << 4 : qd == 2 ? hx << 2 : hx) & 0xC0C0C0C0u;
                        a[v] = top | (qd < 2 ? (w & 0x0F0F0F0Fu) << 2 : (w & 0xF0F0F0F0u) >> 2);
                    }
                    const uint32_t sel = 0x8880u + (uint32_t)(2 * (qd & 1) + m) * 0x1111u;   // byte 2 qd + m of the eight, sign-extended
                    const int s0 = (int)prmt_gs(s[0][qd >> 1], 0u, sel), s1 = (int)prmt_gs(s[1][qd >> 1], 0u, sel);
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const uint32_t b = lds32(bf + nt * kNt + (4 * hf + qd) * 256u + 4 * m);
                        int c[4];
                        mma_s8_k16(c, a[0], a[1], b);
                        acc[nt][0] += s0 * c[0]; acc[nt][1] += s0 * c[1]; acc[nt][2] += s1 * c[2]; acc[nt][3] += s1 * c[3];
                    }
                }
            }
        }
        d0 = f16_bits_to_f32(lds_u16(r0 + 208)) * 0.25f; d1 = f16_bits_to_f32(lds_u16(r1 + 208)) * 0.25f;
    } else if constexpr (TYPE == QKM_TYPE_IQ4_XS) {
        const uint32_t T0 = 0xBFAD9881u, T1 = 0xF6EADDCFu, T2 = 0x26190D01u, T3 = 0x71594535u;   // kvalues_iq4nl as int8
        const uint32_t h0 = lds32(r0), h1 = lds32(r1), l0 = lds32(r0 + 4), l1 = lds32(r1 + 4);   // d | scales_h << 16, scales_l
#pragma unroll
        for (int sb = 0; sb < 8; ++sb) {
            uint32_t a[2][2];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const uint32_t w = lds32((v ? r1 : r0) + 8 + 16 * sb + 4 * t);
                const uint32_t s = w & 0x77777777u, s2 = s >> 16, w4 = w << 4;
                const uint32_t m_lo = prmt_gs(w4, w, 0xD9C8u), m_hi = prmt_gs(w4, w, 0xFBEAu);   // 0xFF where a nibble's top bit is set
                a[v][0] = (prmt_gs(T0, T1, s) & ~m_lo) | (prmt_gs(T2, T3, s) & m_lo);
                a[v][1] = (prmt_gs(T0, T1, s2) & ~m_hi) | (prmt_gs(T2, T3, s2) & m_hi);
            }
            const int s0 = (int)(((l0 >> (4 * sb)) & 15u) | (((h0 >> (16 + 2 * sb)) & 3u) << 4)) - 32;
            const int s1 = (int)(((l1 >> (4 * sb)) & 15u) | (((h1 >> (16 + 2 * sb)) & 3u) << 4)) - 32;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint2 b = lds64(bf + nt * kNt + sb * 256u);
                int c[4];
                mma_s8_first(c, a[0][0], a[1][0], a[0][1], a[1][1], b.x, b.y);
                acc[nt][0] += s0 * c[0]; acc[nt][1] += s0 * c[1]; acc[nt][2] += s1 * c[2]; acc[nt][3] += s1 * c[3];
            }
        }
        d0 = f16_bits_to_f32(h0 & 0xFFFFu); d1 = f16_bits_to_f32(h1 & 0xFFFFu);
    } else {   // IQ3_XXS
#pragma unroll
        for (int sb = 0; sb < 8; ++sb) {
            uint32_t a[2][2];
            int q[2];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const uint32_t b = v ? r1 : r0;
                const uint32_t idx = lds_u16(b + 2 + 8 * sb + 2 * t), aux = lds32_u2(b + 66 + 4 * sb);
                const uint32_t g0 = lds32(lut + (idx & 255u) * 4u), g1 = lds32(lut + (idx >> 8) * 4u);
                const uint32_t sg = signs8((aux >> (7 * t)) & 127u);
                // one 0 / 1 byte per sign bit; -m = ~m + 1 byte by byte (magnitudes are 4 .. 62: no carry leaves a byte)
                const uint32_t n0 = ((sg & 15u) * 0x00204081u) & 0x01010101u, n1 = ((sg >> 4) * 0x00204081u) & 0x01010101u;
                a[v][0] = (g0 ^ (n0 * 255u)) + n0;
                a[v][1] = (g1 ^ (n1 * 255u)) + n1;
                q[v] = (int)(2u * (aux >> 28) + 1u);
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint2 b = lds64(bf + nt * kNt + sb * 256u);
                int c[4];
                mma_s8_first(c, a[0][0], a[1][0], a[0][1], a[1][1], b.x, b.y);
                acc[nt][0] += q[0] * c[0]; acc[nt][1] += q[0] * c[1]; acc[nt][2] += q[1] * c[2]; acc[nt][3] += q[1] * c[3];
            }
        }
        d0 = f16_bits_to_f32(lds_u16(r0)) * 0.25f; d1 = f16_bits_to_f32(lds_u16(r1)) * 0.25f;   // d (s + 0.5) / 2 = d (2 s + 1) / 4
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        f[nt][0] += d0 * (((float)acc[nt][0] * dw0 + (float)acc[nt][1] * dw1) * sc[nt]);
        f[nt][1] += d1 * (((float)acc[nt][2] * dw0 + (float)acc[nt][3] * dw1) * sc[nt]);
    }
}

// F16 weights: rows straight from global memory, eight 16-byte loads per row and 256 columns.
// An f16 MMA adds its products (and the D it is given) by truncation, so a chain of sixteen of them drifts towards zero: 3.5e-7
// from 64 bits (norm, K 512 to 4096), where f32 FMAs of rounded additions are at 0.9e-7 to 2.1e-7.  Every MMA therefore starts from
// zero and eight partial sums at a time are added in f32 as a tree: 0.8e-7 to 1.1e-7; one after the other 0.9e-7 to 1.1e-7 (above
// the FMAs at K = 512).  It costs up to 16 % (4096 x 2048: 16 rows 11.1 -> 12.3 us, 2 rows 6.1 -> 6.1; 12.9 with scalar additions).
template <int NT>
__device__ __forceinline__ void tile_sums_f16(const uint8_t* __restrict__ p0, const uint8_t* __restrict__ p1, uint32_t bf, const float (&sc)[NT],
                                              float dw0, float dw1, float (&f)[NT][2]) {
    uint4 a[8], b[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) { a[s] = __ldg(reinterpret_cast<const uint4*>(p0 + 64 * s)); b[s] = __ldg(reinterpret_cast<const uint4*>(p1 + 64 * s)); }
    float c[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) c[nt][0] = c[nt][1] = c[nt][2] = c[nt][3] = 0.f;
#pragma unroll
    for (int s0 = 0; s0 < 8; s0 += 4) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float p[2 * 4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {   // 32 columns, two MMAs, each
                const int s = s0 + i;
                const uint4 x = lds128(bf + nt * gs::frag_bytes<QKM_TYPE_F16>() + s * 512u);
                mma_f16_k16_first(p[2 * i], a[s].x, b[s].x, a[s].y, b[s].y, x.x, x.y);
                mma_f16_k16_first(p[2 * i + 1], a[s].z, b[s].z, a[s].w, b[s].w, x.z, x.w);
            }
#pragma unroll
            for (int w = 4; w > 0; w >>= 1)
#pragma unroll
                for (int i = 0; i < w; ++i)
#pragma unroll
                    for (int j = 0; j < 4; j += 2) add_f32x2(p[i][j], p[i][j + 1], p[i + w][j], p[i + w][j + 1]);
#pragma unroll
            for (int j = 0; j < 4; j += 2) add_f32x2(c[nt][j], c[nt][j + 1], p[0][j], p[0][j + 1]);
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        f[nt][0] += (c[nt][0] * dw0 + c[nt][1] * dw1) * sc[nt];
        f[nt][1] += (c[nt][2] * dw0 + c[nt][3] * dw1) * sc[nt];
    }
}

// One output as the f32 sum that the formula gives.  Rows of x with an infinity, a NaN or an element above 3.0e38 have no digit
// planes: their sums come out as NaN; and sums of large elements can pass f32 before the weight scale is applied.  What is not
// finite is taken again here, a thread an output: rare, and only then slow.
template <int TYPE>
__device__ __noinline__ float plain_dot(const uint8_t* __restrict__ w, const float* x, uint32_t K) {
    float s = 0.f;
#pragma unroll 1
    for (uint32_t k = 0; k < K; k += 8) {
        float v[8];
        dequant8<TYPE>(w, k, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) s += v[i] * x[k + i];
    }
    return s;
}

struct GemvSplitArgs {
    const uint8_t* W;
    const float* x;      // [n][K]
    float* y;            // [n][M]
    uint32_t M, K, n;    // n <= 2 NT
    uint32_t slices;     // blocks per cluster
    uint32_t kb_slice;   // 256-column blocks per slice (the last slice may have fewer)
};

template <int TYPE, int NT>
__global__ void __launch_bounds__(gs::kMaxWarps * 32, 1)
gemv_split_kernel(GemvSplitArgs a) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    using G = gs::Geo<TYPE>;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t n_warps = blockDim.x >> 5;
    const uint32_t KB = a.K / 256;
    uint32_t rank = 0, n_ctas = 1;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(n_ctas));
    const uint32_t cluster = blockIdx.x / n_ctas, n_clusters = gridDim.x / n_ctas;
    const uint32_t kb0 = rank * a.kb_slice, kb_n = kb0 < KB ? min(a.kb_slice, KB - kb0) : 0u;
    const uint32_t n_tiles = (a.M + 15) / 16;

    // layout: B fragments [kb][NT] | scales [kb][2 NT] | IQ3_XXS grid | partial sums [2][warps][n][16] | tile buffers [warps][2][16 rows]
    const uint32_t s_frag = smem_addr(smem_raw);
    const uint32_t s_scale = s_frag + a.kb_slice * NT * gs::frag_bytes<TYPE>();
    const uint32_t s_lut = s_scale + a.kb_slice * 2 * NT * 4;
    const uint32_t s_part = (s_lut + (TYPE == QKM_TYPE_IQ3_XXS ? 1024u : 0u) + 15u) & ~15u;
    const uint32_t part_bytes = n_warps * a.n * 64u;
    const uint32_t s_buf = (s_part + 2 * part_bytes + 127u) & ~127u;
    constexpr uint32_t kBuf = 16u * G::kStride;
    const uint32_t my_buf = s_buf + warp * 2 * kBuf;
    const size_t rb = (size_t)KB * G::kBytes;

    // work of a warp: (tile, kb) steps, tile = cluster + n_clusters * (warp + n_warps * round); each step's bytes one step ahead
    const uint32_t per_round = n_warps * n_clusters;
    const uint32_t rounds = (n_tiles + per_round - 1) / per_round;
    auto fetch = [&](uint32_t tile, uint32_t kb, uint32_t buf) {   // rows past the end of the matrix: its last row
        if constexpr (TYPE != QKM_TYPE_F16) {
            const uint32_t dst0 = my_buf + buf * kBuf;
            for (uint32_t i = lane; i < 16u * G::kUnits; i += 32) {
                const uint32_t r = i / G::kUnits, u = i - r * G::kUnits;
                const uintptr_t src = (uintptr_t)a.W + (size_t)min(tile * 16u + r, a.M - 1) * rb + (size_t)(kb0 + kb) * G::kBytes;
                const uint32_t off = (uint32_t)(src & 15u);
                if (u * 16u < off + G::kBytes)   // a unit is read only if it holds a byte of the slice
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst0 + r * G::kStride + u * 16u), "l"(src - off + u * 16u) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto tile_of = [&](uint32_t round) { return cluster + n_clusters * (warp + n_warps * round); };
    uint32_t p_round = 0, p_kb = 0, p_buf = 0;   // next step to fetch
    auto fetch_next = [&]() -> bool {
        if (p_round >= rounds || !kb_n) return false;
        const uint32_t tile = tile_of(p_round);
        if (tile >= n_tiles) return false;   // a warp's later tiles lie past the end too
        fetch(tile, p_kb, p_buf);
        p_buf ^= 1u;
        if (++p_kb == kb_n) { p_kb = 0; ++p_round; }
        return true;
    };
    // Nothing that other kernels write is read or written before the wait, but the table can be filled and the first step's
    // weights asked into the L2 while the kernel before this one ends.
    pdl_trigger();
    if (TYPE == QKM_TYPE_IQ3_XXS)
        for (uint32_t i = tid; i < 256; i += blockDim.x) sts32(s_lut + i * 4, c_iq3_grid[i]);
    if (kb_n && tile_of(0) < n_tiles)
        for (uint32_t o = (lane >> 4) * 128u; o < (uint32_t)G::kBytes; o += 256u)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a.W + (size_t)min(tile_of(0) * 16u + (lane & 15u), a.M - 1) * rb + (size_t)kb0 * G::kBytes + o));
    pdl_wait();
    fetch_next();

    // x of this block's slice as B fragments, a warp per (row, 256 columns)
    constexpr int kAhead = NT >= 4 ? 4 : NT;   // rows whose loads are in flight together (one at a time would cost a memory latency each)
    for (uint32_t i0 = warp; i0 < kb_n * 2 * NT; i0 += n_warps * kAhead) {
        float v[kAhead][8];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const uint32_t i = i0 + u * n_warps, kb = i / (2 * NT), row = i - kb * 2 * NT;
#pragma unroll
            for (int j = 0; j < 8; ++j) v[u][j] = 0.f;
            if (i < kb_n * 2 * NT && row < a.n) {
                const float4* p = reinterpret_cast<const float4*>(a.x + (size_t)row * a.K + (size_t)(kb0 + kb) * 256 + 8 * lane);
                const float4 lo = p[0], hi = p[1];
                v[u][0] = lo.x; v[u][1] = lo.y; v[u][2] = lo.z; v[u][3] = lo.w; v[u][4] = hi.x; v[u][5] = hi.y; v[u][6] = hi.z; v[u][7] = hi.w;
            }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const uint32_t i = i0 + u * n_warps, kb = i / (2 * NT), row = i - kb * 2 * NT;
            if (i >= kb_n * 2 * NT) break;
            float m = 0.f;
            bool bad = false;
#pragma unroll
            for (int j = 0; j < 8; ++j) { m = fmaxf(m, fabsf(v[u][j])); bad |= !(fabsf(v[u][j]) <= 3.0e38f); }
            m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));   // non-negative floats order like their bits
            bad = __any_sync(0xFFFFFFFFu, bad);
            int p = min(digit_exponent(m), 126);
            if (TYPE == QKM_TYPE_F16) p = m > 0.f ? p - 12 : 0;   // the largest value in [2^13, 2^14): f16 pieces
            const float up = bad ? 1.f : ldexpf(1.0f, p);
            if (bad) {
#pragma unroll
                for (int j = 0; j < 8; ++j) v[u][j] = 0.f;
            }
            encode_fragments<TYPE>(v[u], lane, s_frag + (kb * NT + (row >> 1)) * gs::frag_bytes<TYPE>(), (row & 1u) * 4u, up);
            if (lane == 0) sts32(s_scale + i * 4, __float_as_uint(bad ? __int_as_float(0x7FC00000) : ldexpf(1.0f, -p)));   // its outputs: plain_dot
        }
    }
    __syncthreads();

    // weights of MMA columns 2t, 2t+1: digits 128^j, or pieces 2^-11j (the fourth piece is empty)
    const float dw0 = TYPE == QKM_TYPE_F16 ? ((t & 1u) ? 2.384185791015625e-07f : 1.f) : ((t & 1u) ? 16384.f : 1.f);
    const float dw1 = TYPE == QKM_TYPE_F16 ? ((t & 1u) ? 0.f : 4.8828125e-04f) : dw0 * 128.f;
    uint32_t c_buf = 0;
    for (uint32_t round = 0; round < rounds; ++round) {
        const uint32_t tile = tile_of(round);
        float f[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) f[nt][0] = f[nt][1] = 0.f;
        if (tile < n_tiles) {
            for (uint32_t kb = 0; kb < kb_n; ++kb) {
                const bool more = fetch_next();   // one step ahead: the other buffer was read before the last __syncwarp
                float sc[NT];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) sc[nt] = __uint_as_float(lds32(s_scale + (kb * 2 * NT + 2 * nt + (t >> 1)) * 4));
                const uint32_t bf = s_frag + kb * NT * gs::frag_bytes<TYPE>() + lane * (TYPE == QKM_TYPE_F16 ? 16u : 8u);
                if (TYPE == QKM_TYPE_F16) {
                    const uint8_t* p0 = a.W + (size_t)min(tile * 16u + g, a.M - 1) * rb + (size_t)(kb0 + kb) * 512 + 16 * t;
                    const uint8_t* p1 = a.W + (size_t)min(tile * 16u + g + 8, a.M - 1) * rb + (size_t)(kb0 + kb) * 512 + 16 * t;
                    tile_sums_f16<NT>(p0, p1, bf, sc, dw0, dw1, f);
                } else {
                    if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
                    else asm volatile("cp.async.wait_group 0;" ::: "memory");
                    __syncwarp();
                    const uintptr_t s0 = (uintptr_t)a.W + (size_t)min(tile * 16u + g, a.M - 1) * rb + (size_t)(kb0 + kb) * G::kBytes;
                    const uintptr_t s1 = (uintptr_t)a.W + (size_t)min(tile * 16u + g + 8, a.M - 1) * rb + (size_t)(kb0 + kb) * G::kBytes;
                    const uint32_t b = my_buf + c_buf * kBuf;
                    tile_sums<TYPE, NT>(b + g * G::kStride + (uint32_t)(s0 & 15u), b + (g + 8) * G::kStride + (uint32_t)(s1 & 15u), bf, t, s_lut, sc, dw0, dw1, f);
                    c_buf ^= 1u;
                    __syncwarp();
                }
            }
        }
        // the other two digits (pieces) of a row of x sit in lane t ^ 1; then the slices' sums over the cluster
        const uint32_t part = s_part + (round & 1u) * part_bytes;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const float v0 = f[nt][0] + __shfl_xor_sync(0xFFFFFFFFu, f[nt][0], 1), v1 = f[nt][1] + __shfl_xor_sync(0xFFFFFFFFu, f[nt][1], 1);
            const uint32_t row = 2 * nt + (t >> 1);
            if ((t & 1u) == 0 && row < a.n) {
                const uint32_t at = part + ((warp * a.n + row) * 16u + g) * 4u;
                sts32(at, __float_as_uint(v0)); sts32(at + 32, __float_as_uint(v1));
            }
        }
        // (two buffers: a block writes one again only after the barrier of the round between, which follows every read of it)
        if (n_ctas > 1) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        else __syncthreads();
        const uint32_t outs = n_warps * a.n * 16u, share = (outs + n_ctas - 1) / n_ctas;
        for (uint32_t o = rank * share + tid; o < min(outs, (rank + 1) * share); o += blockDim.x) {
            const uint32_t w = o / (a.n * 16u), row = (o >> 4) - w * a.n, r = o & 15u;
            const uint32_t m = (cluster + n_clusters * (w + n_warps * round)) * 16u + r;
            if (m < a.M) {
                float p[8], v = 0.f;   // at most eight slices; all reads under way before the first is used
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                    if (q < n_ctas) {
                        uint32_t remote;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(part + o * 4u), "r"(q));
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(p[q]) : "r"(remote) : "memory");
                    }
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)   // slice order
                    if (q < n_ctas) v += p[q];
                if (!(fabsf(v) <= 3.402823466e38f)) v = plain_dot<TYPE>(a.W + (size_t)m * rb, a.x + (size_t)row * a.K, a.K);
                a.y[(size_t)row * a.M + m] = v;
            }
        }
    }
    if (n_ctas > 1)   // no block leaves while another still reads its partial sums
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int TYPE, int NT>
static cudaError_t gemv_split_launch_nt(const Launch& L, GemvSplitArgs a, uint32_t n_sms, bool* taken) {
    using G = gs::Geo<TYPE>;
    const uint32_t KB = a.K / 256, n_tiles = (a.M + 15) / 16;
    // Eight slices while one round of tiles covers the matrix (33 such clusters are resident), four beyond: more
    // slices share the work of few tiles between more warps, fewer waste less on the cluster's barriers and sums.
    // (More than eight rows of F16 x above 2048 columns: eight always, a quarter's fragments would leave room for one block an SM.)
    uint32_t slices = KB >= 8 && (n_tiles <= 33u * 8u || (TYPE == QKM_TYPE_F16 && NT > 4 && KB > 8)) ? 8u : KB >= 4 ? 4u : KB >= 2 ? 2u : 1u;
    a.kb_slice = (KB + slices - 1) / slices;
    slices = (KB + a.kb_slice - 1) / a.kb_slice;   // no empty slice
    a.slices = slices;
    if (const cudaError_t e = allow_dynamic_smem<gemv_split_kernel<TYPE, NT>>(220 * 1024)) return e;
    const size_t fixed = (size_t)a.kb_slice * NT * gs::frag_bytes<TYPE>() + (size_t)a.kb_slice * 2 * NT * 4 + 1024 + 256;
    auto need = [&](uint32_t w) { return fixed + 2 * (size_t)w * a.n * 64 + (size_t)w * 2 * 16 * G::kStride; };
    // Two blocks of up to eight warps per SM.  How many clusters are resident at once is less than the SMs would
    // hold (a GPC's SMs are not a multiple of the cluster), and one cluster more takes the time of a second wave.
    uint32_t warps = 8;
    while (warps > 4 && need(warps) > 110u * 1024u) --warps;
    const size_t most = need(warps);
    *taken = most <= 220u * 1024u;
    if (!*taken) return cudaSuccess;
    const bool two = most <= 110u * 1024u;
    uint32_t clusters_max = (two ? 2u : 1u) * n_sms / slices;
    if (slices > 4) clusters_max = clusters_max * (two ? 33u : 30u) / 37u;
    else if (slices > 2) clusters_max = clusters_max * (two ? 71u : 66u) / 74u;
    // one tile per warp and round; fewer warps where there are not tiles enough for every cluster
    const uint32_t per_cluster = (n_tiles + clusters_max - 1) / clusters_max;
    if (per_cluster < warps) warps = per_cluster < 4 ? 4 : per_cluster;
    const size_t smem = need(warps);
    const uint32_t want = (n_tiles + warps - 1) / warps;
    const uint32_t clusters = want < clusters_max ? want : clusters_max;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * slices); cfg.blockDim = dim3(warps * 32); cfg.dynamicSmemBytes = smem; cfg.stream = L.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = slices; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemv_split_kernel<TYPE, NT>, a);
    L.count();
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int TYPE>
static cudaError_t gemv_split_launch(const Launch& L, const uint8_t* W, const float* x, float* y, uint32_t M, uint32_t K, uint32_t n,
                                     uint32_t n_sms, uint32_t* rows_done) {
    *rows_done = 0;
    while (n) {   // sixteen rows of x a pass (eight where the fragments of sixteen would not leave room for the tiles)
        const uint32_t most = TYPE == QKM_TYPE_F16 && K > 4096 ? 8u : 16u;
        GemvSplitArgs a{};
        a.W = W; a.x = x + (size_t)*rows_done * K; a.y = y + (size_t)*rows_done * M; a.M = M; a.K = K;
        a.n = n < most ? n : most;
        bool taken = false;
        cudaError_t e;
        if (a.n <= 2) e = gemv_split_launch_nt<TYPE, 1>(L, a, n_sms, &taken);
        else if (a.n <= 4) e = gemv_split_launch_nt<TYPE, 2>(L, a, n_sms, &taken);
        else if (a.n <= 6) e = gemv_split_launch_nt<TYPE, 3>(L, a, n_sms, &taken);
        else if (a.n <= 8) e = gemv_split_launch_nt<TYPE, 4>(L, a, n_sms, &taken);
        else if (a.n <= 12) e = gemv_split_launch_nt<TYPE, 6>(L, a, n_sms, &taken);
        else e = gemv_split_launch_nt<TYPE, 8>(L, a, n_sms, &taken);
        if (e != cudaSuccess || !taken) return e;
        *rows_done += a.n;
        n -= a.n;
    }
    return cudaSuccess;
}

// x rows [0, *rows_done) are done; shapes this form does not take leave it at 0
cudaError_t launch_gemv_split(const Launch& L, uint32_t type, const void* W, const float* x, float* y, uint32_t M, uint32_t K, uint32_t n,
                              uint32_t n_sms, uint32_t* rows_done) {
    *rows_done = 0;
    if (M == 0 || n == 0 || K % 256 || K > 8192 || ((uintptr_t)x & 15u) || ((uintptr_t)W & (type == QKM_TYPE_IQ4_XS ? 7u : type == QKM_TYPE_Q6_K || type == QKM_TYPE_IQ3_XXS ? 1u : 15u)))
        return cudaSuccess;
    const uint8_t* w = (const uint8_t*)W;
    switch (type) {
        case QKM_TYPE_F16: return gemv_split_launch<QKM_TYPE_F16>(L, w, x, y, M, K, n, n_sms, rows_done);
        case QKM_TYPE_Q8_0: return gemv_split_launch<QKM_TYPE_Q8_0>(L, w, x, y, M, K, n, n_sms, rows_done);
        case QKM_TYPE_Q6_K: return gemv_split_launch<QKM_TYPE_Q6_K>(L, w, x, y, M, K, n, n_sms, rows_done);
        case QKM_TYPE_IQ4_XS: return gemv_split_launch<QKM_TYPE_IQ4_XS>(L, w, x, y, M, K, n, n_sms, rows_done);
        case QKM_TYPE_IQ3_XXS: return gemv_split_launch<QKM_TYPE_IQ3_XXS>(L, w, x, y, M, K, n, n_sms, rows_done);
        default: return cudaSuccess;
    }
}

}  // namespace qkm
