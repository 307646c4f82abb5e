// Device-resident weight layout of the streaming kernels ("tiles") and the
// activation encoding they consume ("digit planes").
//
// TILES.  qkm_upload_layer keeps the raw ggml tensors and additionally stores a
// re-ordered copy, grouped so that one bulk copy fetches everything a warp (decode) or a
// 128-row unit (prefill) needs and both read it back from shared memory with aligned,
// conflict-free 128-bit loads: a decode lane reads its 16 bytes of two rows, a prefill
// thread all bytes of one row.  Values are unchanged; bytes per 16 x 256 tile: IQ3_XXS 1696
// (1568 in the file: the 7-bit sign codes are stored as 8 sign bits, the 4-bit scales as bytes 2 s + 1 -
// two instructions less per eight weights for 8 % more bytes in kernels bound by instruction issue),
// IQ4_XS 2176, Q6_K 3360, Q8_0 4352 as in the file.
// Tiles of one matrix [rows][K] are ordered [kb = K/256][rt = rows/16]: a warp that
// owns column block kb walks consecutive memory as it moves down the rows, and the eight tiles of 128 rows are
// one run.
//
// Inside a tile, "lane" is the MMA lane 4*g + t (g = 0..7 row group, t = 0..3):
// lane (g,t) works on rows g and g+8 of the tile, on columns 8t .. 8t+7 of every 32-column sub-block
// (IQ3_XXS, IQ4_XS).  A row's four 16-byte pieces t of a 64-byte run lie at piece position t ^ ((row >> 1) & 3):
// eight consecutive rows that each read piece t, and one row group's lanes that read pieces 0..3, both hit
// all 32 banks once.
//
//   IQ3_XXS (block: d f16 | qs[64] grid indices | 8 aux words, src/quants.h:115-119)
//     [   0,1024)  grid indices: row r at 64 r, piece t: 2 bytes for each of the eight sub-blocks
//                  (raw qs[8*ib + 2*t], qs[8*ib + 2*t + 1])
//     [1024,1536)  signs: row r at 1024 + 32 r, lane t's 8 bytes at 16 ((t >> 1) ^ ((r >> 2) & 1)) + 8 (t & 1): two words,
//                  word q for sub-blocks 4q .. 4q+3; bit 7 - (2 (s & 3) + h) of byte b = element 8t + 4h + b of sub-block s
//                  is negative (shifted left by 2 (s & 3) + h, the four sign bits of an MMA operand register are the
//                  top bits of its bytes, and of two f16 pairs)
//     [1536,1664)  scales: row r at 1536 + 8 r, byte s = 2 * scale + 1 of sub-block s
//     [1664,1696)  d[16] f16
//   IQ4_XS (block: d f16 | scales_h u16 | scales_l[4] | qs[128], src/quants.h:107-113)
//     [   0, 128)  headers: for g: 8 B of row g then 8 B of row g+8, each the raw first
//                  8 bytes of the block (d, scales_h, scales_l)
//     [ 128,2176)  quants: column half q (sub-blocks 4q .. 4q+3), row r at 128 + 1024 q + 64 r, piece t: one word
//                  per sub-block with the codes of elements 8t .. 8t+7: byte 0 = (e0 low, e2 high nibble), byte 1 = (e1, e3),
//                  byte 2 = (e4, e6), byte 3 = (e5, e7)
//   Q6_K (block: ql[128] | qh[64] | scales[16] int8 | d f16, src/quants.h:98-103).  A 128-column
//   half hf of a block packs element l + 32*qd (l < 32, qd < 4) as nibble (qd >> 1) of
//   ql[64*hf + 32*(qd & 1) + l] and bit pair qd of qh[32*hf + l]; its scale is scales[8*hf + 2*qd + l/16].
//   Word m (0..7) of a 32-byte run holds l = 4m..4m+3.  Lane (g,t) multiplies, for every (hf, qd),
//   the elements l = 4t..4t+3 (16-column group 2*(4*hf+qd)) and l = 16+4t..16+4t+3 (the group after it):
//     [   0, 256)  scales: row r at 16*r, the eight even groups 0,2,..,14 then the eight odd ones
//     [ 256,3328)  quants: k (0..2), row r at 256 + 1024 k + 64 r, piece t:
//                  k = 0, 1: half hf = k: ql words t and 4+t of the first 32-byte run, then of the second
//                  k = 2:    qh words t and 4+t of half 0, then of half 1
//     [3328,3360)  d[16] f16
//   Q8_0 (block: d f16 | qs[32], src/quants.h:53-57), 8 blocks per row per tile; block b of
//   the 16 rows is one 544-byte piece at 544*b (so a run of blocks is one bulk copy):
//     [  0, 32)  d: row r at 2*r
//     [ 32,544)  quants: half h (row g + 8h), lane -> 8 B at 32 + (h*32 + lane)*8
//                = raw qs[4t..4t+3] then qs[16+4t..16+4t+3]
//
// DIGIT PLANES.  An activation row x[K] (or a hidden row) is encoded as four int8 planes with one
// power-of-two scale per 256 columns:
//   v = rint(x * 2^p),  |v| <= 2^26,  v = d0 + 128*d1 + 128^2*d2 + 128^3*d3,  d_j in [-64, 63]
// so x = 2^-p * sum_j 128^j d_j up to a rounding error of 2^-(p+1) <= 2^-26 * max|x| over the block
// (max|x| * 2^p lies in [2^25, 2^26)): finer than f32 for the largest elements, coarser below, and exact integer
// arithmetic from there on (int8 x int8 -> int32 tensor-core MMAs).
#pragma once

#include <stdint.h>

namespace qkm {

static constexpr int kTileIq3 = 1696;
static constexpr int kTileIq4 = 2176;
static constexpr int kTileQ6 = 3360;
static constexpr int kTileQ8 = 4352;

__host__ __device__ inline int tile_bytes(uint32_t type) {
    switch (type) {
        case QKM_TYPE_IQ3_XXS: return kTileIq3;
        case QKM_TYPE_IQ4_XS: return kTileIq4;
        case QKM_TYPE_Q6_K: return kTileQ6;
        case QKM_TYPE_Q8_0: return kTileQ8;
        default: return 0;
    }
}

// bytes of n_mats matrices [rows][K] in tile order
__host__ __device__ inline size_t tiled_bytes(uint32_t type, size_t n_mats, uint32_t rows, uint32_t K) {
    return n_mats * (rows / 16) * (K / 256) * (size_t)tile_bytes(type);
}
// position of piece t of row r inside the row's 64-byte run
__host__ __device__ inline uint32_t piece_at(uint32_t r, uint32_t t) { return (t ^ ((r >> 1) & 3u)) * 16u; }

}  // namespace qkm
