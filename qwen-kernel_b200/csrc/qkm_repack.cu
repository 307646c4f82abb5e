// Upload-time re-ordering of raw ggml tensors into the tile layout the streaming
// kernels read (see qkm_tiles.cuh).  The weights' values are unchanged: Q6_K and Q8_0 bytes are moved, IQ4_XS
// nibbles are paired anew (as many bytes), IQ3_XXS sign codes become sign bits and its 4-bit scales bytes
// 2 s + 1 (1696 bytes a tile for 1568 of the file).
#include "qkm_common.cuh"
#include "qkm_kernels.h"
#include "qkm_tiles.cuh"

namespace qkm {

// A block per tile: its 16 x 256 columns of raw bytes go to shared memory, every thread then puts output words together.
// n_mats matrices of [rows][K] follow each other in both layouts (experts of a stacked tensor); rows % 16 == 0 and K % 256 == 0.
constexpr int kRepackThreads = 128;
template <int TYPE>
__global__ void __launch_bounds__(kRepackThreads)
repack_kernel(const uint8_t* __restrict__ raw, uint8_t* __restrict__ out, uint32_t rows, uint32_t K) {
    constexpr uint32_t kTile = TYPE == QKM_TYPE_IQ3_XXS ? kTileIq3 : TYPE == QKM_TYPE_IQ4_XS ? kTileIq4 : TYPE == QKM_TYPE_Q6_K ? kTileQ6 : kTileQ8;
    constexpr uint32_t kSpan = TYPE == QKM_TYPE_Q8_0 ? 8 * 34 : Fmt<TYPE>::kBytes;   // bytes of one row's 256 columns, even
    __shared__ __align__(4) uint8_t s_raw[16 * kSpan];
    const uint32_t KB = K / 256, RT = rows / 16;
    const uint32_t rt = blockIdx.x % RT, kb = blockIdx.x / RT % KB, mat = blockIdx.x / RT / KB;
    const size_t rb = row_bytes(TYPE, K);
    const uint8_t* m = raw + ((size_t)mat * rows + rt * 16) * rb + (size_t)kb * kSpan;
    for (uint32_t i = threadIdx.x; i < 16 * kSpan / 2; i += kRepackThreads) {
        const uint32_t r = i / (kSpan / 2), c = i - r * (kSpan / 2);
        *reinterpret_cast<uint16_t*>(s_raw + r * kSpan + 2 * c) = *reinterpret_cast<const uint16_t*>(m + r * rb + 2 * c);
    }
    __syncthreads();
    auto src = [&](uint32_t row, uint32_t byte) -> uint32_t { return s_raw[row * kSpan + byte]; };
    auto word16 = [&](uint32_t row, uint32_t byte) -> uint32_t { return *reinterpret_cast<const uint16_t*>(s_raw + row * kSpan + byte); };
    auto out_byte = [&](uint32_t o) -> uint32_t {
    if (TYPE == QKM_TYPE_IQ3_XXS) {
        auto aux = [&](uint32_t row, uint32_t sb) -> uint32_t { return word16(row, 66 + 4 * sb) | (word16(row, 68 + 4 * sb) << 16); };
        uint32_t v = 0;
        if (o < 1024) {
            const uint32_t row = o >> 6, t = ((o >> 4) & 3u) ^ ((row >> 1) & 3u), b = o & 15u;
            v = src(row, 2 + 8 * (b >> 1) + 2 * t + (b & 1u));
        } else if (o < 1536) {
            const uint32_t q = o - 1024, row = q >> 5, t = ((((q >> 4) & 1u) ^ ((row >> 2) & 1u)) << 1) | ((q >> 3) & 1u), b = q & 3u;
            for (uint32_t j = 0; j < 8; ++j) {
                const uint32_t sg = signs8((aux(row, 4 * ((q >> 2) & 1u) + (j >> 1)) >> (7 * t)) & 127u);
                v |= ((sg >> (4 * (j & 1u) + b)) & 1u) << (7 - j);
            }
        } else if (o < 1664) {
            v = 2 * (aux((o - 1536) >> 3, (o - 1536) & 7u) >> 28) + 1;
        } else {
            v = src((o - 1664) >> 1, (o - 1664) & 1u);
        }
        return v;
    } else if (TYPE == QKM_TYPE_IQ4_XS) {
        if (o < 128) {
            return src((o >> 4) + 8 * ((o >> 3) & 1u), o & 7u);
        } else {
            const uint32_t q = o - 128, row = (q >> 6) & 15u, t = ((q >> 4) & 3u) ^ ((row >> 1) & 3u), sb = 4 * (q >> 10) + ((q >> 2) & 3u), b = q & 3u;
            auto code = [&](uint32_t e) -> uint32_t { return (src(row, 8 + 16 * sb + (e & 15u)) >> (e >= 16 ? 4 : 0)) & 15u; };
            const uint32_t e = 8 * t + 4 * (b >> 1) + (b & 1u);
            return code(e) | (code(e + 2) << 4);
        }
    } else if (TYPE == QKM_TYPE_Q6_K) {
        uint32_t row_in_tile, off;
        if (o < 256) {
            const uint32_t b = o & 15u;
            row_in_tile = o >> 4;
            off = 192 + (b < 8 ? 2 * b : 2 * (b - 8) + 1);
        } else if (o < 3328) {
            const uint32_t q = o - 256, k = q >> 10, b = q & 15u, w = b >> 2;
            row_in_tile = (q >> 6) & 15u;
            const uint32_t t = ((q >> 4) & 3u) ^ ((row_in_tile >> 1) & 3u), wm = (w & 1u) ? 4 + t : t;
            off = k < 2 ? 64 * k + 32 * (w >> 1) + 4 * wm + (b & 3u) : 128 + 32 * (w >> 1) + 4 * wm + (b & 3u);
        } else {
            row_in_tile = (o - 3328) >> 1;
            off = 208 + (o & 1u);
        }
        return src(row_in_tile, off);
    } else {  // Q8_0: per 32-column block, the 16 rows' d (32 B) then their quants (512 B)
        const uint32_t blk = o / 544u, q = o - blk * 544u;
        uint32_t row_in_tile, off;
        if (q < 32) {
            row_in_tile = q >> 1;
            off = q & 1u;
        } else {
            const uint32_t v = q - 32, h = (v >> 8) & 1u, lane = (v >> 3) & 31u, b = v & 7u;
            const uint32_t g = lane >> 2, t = lane & 3u;
            row_in_tile = g + 8 * h;
            off = 2 + (b < 4 ? 4 * t + b : 16 + 4 * t + (b - 4));
        }
        return src(row_in_tile, blk * 34 + off);
    }
    };
    uint32_t* dst = reinterpret_cast<uint32_t*>(out + (size_t)blockIdx.x * kTile);
    for (uint32_t w = threadIdx.x; w < kTile / 4; w += kRepackThreads)
        dst[w] = out_byte(4 * w) | (out_byte(4 * w + 1) << 8) | (out_byte(4 * w + 2) << 16) | (out_byte(4 * w + 3) << 24);
}

cudaError_t launch_repack(const Launch& L, uint32_t type, const void* raw, void* out, uint32_t n_mats,
                          uint32_t rows, uint32_t K) {
    if (rows % 16 || K % 256) return cudaErrorInvalidValue;
    const uint64_t tiles = (uint64_t)n_mats * (rows / 16) * (K / 256);
    if (tiles == 0) return cudaSuccess;
    if (tiles > 0x7FFFFFFFu) return cudaErrorInvalidValue;
    const uint8_t* r = (const uint8_t*)raw;
    uint8_t* o = (uint8_t*)out;
    switch (type) {
        case QKM_TYPE_IQ3_XXS: repack_kernel<QKM_TYPE_IQ3_XXS><<<(unsigned)tiles, kRepackThreads, 0, L.stream>>>(r, o, rows, K); break;
        case QKM_TYPE_IQ4_XS: repack_kernel<QKM_TYPE_IQ4_XS><<<(unsigned)tiles, kRepackThreads, 0, L.stream>>>(r, o, rows, K); break;
        case QKM_TYPE_Q6_K: repack_kernel<QKM_TYPE_Q6_K><<<(unsigned)tiles, kRepackThreads, 0, L.stream>>>(r, o, rows, K); break;
        case QKM_TYPE_Q8_0: repack_kernel<QKM_TYPE_Q8_0><<<(unsigned)tiles, kRepackThreads, 0, L.stream>>>(r, o, rows, K); break;
        default: return cudaErrorInvalidValue;
    }
    L.count();
    return cudaGetLastError();
}

// Largest finite |d| of a matrix's blocks, as f16 bits in *out (zero before): a thread a block.
__global__ void __launch_bounds__(256)
scale_max_kernel(const uint8_t* __restrict__ raw, uint32_t* __restrict__ out, uint64_t n_blocks, uint32_t block_bytes) {
    const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    uint32_t d = i < n_blocks ? *reinterpret_cast<const uint16_t*>(raw + i * block_bytes) & 0x7FFFu : 0u;
    if (d >= 0x7C00u) d = 0;
    d = __reduce_max_sync(0xFFFFFFFFu, d);
    if ((threadIdx.x & 31u) == 0 && d) atomicMax(out, d);
}
cudaError_t launch_scale_max(const Launch& L, uint32_t type, const void* raw, uint32_t* out, uint32_t rows, uint32_t K) {
    if (type != QKM_TYPE_Q8_0 && type != QKM_TYPE_IQ4_XS) return cudaErrorInvalidValue;   // d comes first in a block
    const uint32_t elems = type == QKM_TYPE_Q8_0 ? 32 : 256;
    const uint64_t n = (uint64_t)rows * (K / elems);
    if (n == 0) return cudaSuccess;
    scale_max_kernel<<<(unsigned)((n + 255) / 256), 256, 0, L.stream>>>((const uint8_t*)raw, out, n, (uint32_t)row_bytes(type, elems));
    L.count();
    return cudaGetLastError();
}

}  // namespace qkm
