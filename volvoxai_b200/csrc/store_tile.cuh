// How a GEMM epilogue warp gets its 32 rows x 32 columns of finished outputs to global memory when no tensor
// map can: TMEM hands every lane one row, so a store straight from the registers touches 32 rows per
// instruction.  The warp therefore passes the values through a 2 KB shared-memory tile of its own (16-byte
// pieces XORed with the row so that neither the row-wise writes nor the reads meet in a bank) and stores
// along the rows.  All lanes of the warp call these functions together.
#pragma once

#include "common.cuh"

namespace vxb {

// ---- bytes: a [32 rows x 64 B] tile, two 32-column chunks wide ---------------------------------

// This lane's 32 bytes of its row: chunk 0 or 1 of the tile.
__device__ __forceinline__ void stage_bytes(uint8_t* tile, uint32_t lane, uint32_t chunk, const uint32_t (&packed)[8]) {
    uint8_t* row = tile + lane * 64u;
    const uint32_t sw = (lane >> 1) & 3u;
    *reinterpret_cast<uint4*>(row + (((2u * chunk) ^ sw) << 4)) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    *reinterpret_cast<uint4*>(row + (((2u * chunk + 1u) ^ sw) << 4)) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
}

// Rows [0, rows) of the tile to out (row pitch ld bytes, any alignment), `width` <= 64 bytes of each, in the largest
// unit that base, pitch and width allow: words (two rows of 16 lanes per instruction), half words (a row per
// instruction) or bytes (a row in two).  Every store instruction covers consecutive bytes of one or two rows; nothing
// diverges but the row's end.  The GEMM of 777 x 1283 -> 2050 took 37.8 us with a store per byte from the registers, 32
// rows per instruction, and takes 10.7 this way (8.6 for 2048 aligned columns).  Not inlined: a ragged edge is rare, and its registers would be taken from the
// epilogue that every tile runs.
static __device__ __noinline__ void flush_bytes(const uint8_t* tile, uint32_t lane, int8_t* out, uint32_t ld, uint32_t rows, uint32_t width) {
    const uint32_t unit = ((uint32_t)(uintptr_t)out | ld | width) & 3u;
    auto at = [&](uint32_t r, uint32_t byte) { return tile + r * 64u + (((byte >> 4) ^ ((r >> 1) & 3u)) << 4) + (byte & 15u); };
    if (unit == 0) {
        const uint32_t byte = (lane & 15u) * 4u;
        if (byte < width) {
            int8_t* dst = out + (size_t)(lane >> 4) * ld + byte;
#pragma unroll 8
            for (uint32_t r = lane >> 4; r < 32u; r += 2u, dst += 2u * (size_t)ld)
                if (r < rows) *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(at(r, byte));
        }
    } else if (unit == 2) {
        const uint32_t byte = lane * 2u;
        if (byte < width) {
            int8_t* dst = out + byte;
#pragma unroll 8
            for (uint32_t r = 0; r < 32u; r++, dst += ld)
                if (r < rows) *reinterpret_cast<uint16_t*>(dst) = *reinterpret_cast<const uint16_t*>(at(r, byte));
        }
    } else {
        int8_t* dst = out + lane;
        const bool left = lane < width, right = lane + 32u < width;
#pragma unroll 8
        for (uint32_t r = 0; r < 32u; r++, dst += ld) {
            if (r >= rows) break;
            const uint8_t v0 = *at(r, lane), v1 = *at(r, lane + 32u);
            if (left) dst[0] = (int8_t)v0;
            if (right) dst[32] = (int8_t)v1;
        }
    }
}

// ---- 32-bit words: a [16 rows x 128 B] tile ------------------------------------------------------

// 16 rows of the tile to out (row pitch ld words, rows [0, rows), columns [0, columns)) in pairs of words (two rows per
// instruction) where base, pitch and width allow, else in words (a row per instruction).  All reads go ahead of the
// stores: 4096 x 576 -> 2050, quantizer included, takes 19.3 us; read and stored one after the other, with a test of the
// row between, it took 28.8, and in 16-byte pieces of four rows, split where not aligned, 20.8.  Not inlined, like flush_bytes.
static __device__ __noinline__ void flush_words(const uint8_t* tile, uint32_t lane, uint32_t* out, uint32_t ld, uint32_t rows, uint32_t columns) {
    if (((((uint32_t)(uintptr_t)out >> 2) | ld | columns) & 1u) == 0) {
        const uint32_t l = lane & 15u, odd = lane >> 4;
        const bool live = 2u * l < columns;
        uint32_t* dst = out + (size_t)odd * ld + 2u * l;
        uint2 v[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
            const uint32_t r = 2u * i + odd;
            v[i] = *reinterpret_cast<const uint2*>(tile + r * 128u + (((l >> 1) ^ (r & 7u)) << 4) + (l & 1u) * 8u);
        }
#pragma unroll
        for (uint32_t i = 0; i < 8; i++, dst += 2u * (size_t)ld)
            if (live && 2u * i + odd < rows) *reinterpret_cast<uint2*>(dst) = v[i];
    } else {
        const bool live = lane < columns;
        uint32_t* dst = out + lane;
        uint32_t v[16];
#pragma unroll
        for (uint32_t i = 0; i < 16; i++) v[i] = *reinterpret_cast<const uint32_t*>(tile + i * 128u + (((lane >> 2) ^ (i & 7u)) << 4) + (lane & 3u) * 4u);
#pragma unroll
        for (uint32_t i = 0; i < 16; i++, dst += ld)
            if (live && i < rows) *dst = v[i];
    }
}

// One 32 x 32 chunk, this lane's row in o, to out (row pitch ld words, rows [0, rows), columns [0, columns)).
// `aligned` (uniform): all 32 columns exist and every row segment is 16-byte aligned - four rows of 128 bytes per
// instruction; otherwise flush_words.
__device__ __forceinline__ void store_words(uint8_t* tile, uint32_t lane, const uint32_t (&o)[32], uint32_t* out, uint32_t ld,
                                            uint32_t rows, uint32_t columns, bool aligned) {
#pragma unroll
    for (uint32_t half = 0; half < 2; half++) {
        __syncwarp();
        if ((lane >> 4) == half) {
            uint8_t* mine = tile + (lane & 15u) * 128u;
#pragma unroll
            for (uint32_t j = 0; j < 8; j++)
                *reinterpret_cast<uint4*>(mine + ((j ^ (lane & 7u)) << 4)) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        }
        __syncwarp();
        if (aligned) {
            const uint32_t piece = lane & 7u;
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
                const uint32_t r = 4u * i + (lane >> 3);
                const uint4 v = *reinterpret_cast<const uint4*>(tile + r * 128u + ((piece ^ (r & 7u)) << 4));
                if (half * 16u + r < rows) *reinterpret_cast<uint4*>(out + (size_t)(half * 16u + r) * ld + 4u * piece) = v;
            }
        } else {
            const uint32_t r0 = half * 16u;
            flush_words(tile, lane, out + (size_t)r0 * ld, ld, rows > r0 ? rows - r0 : 0u, columns);
        }
    }
}

// ---- 32-bit words, half as many columns: a [32 rows x 64 B] tile ----------------------------------

// The same for a tile of half rows, all 32 of them: four rows per instruction in pairs of words, two in words.
static __device__ __noinline__ void flush_half_words(const uint8_t* tile, uint32_t lane, float* out, uint32_t ld, uint32_t rows, uint32_t columns) {
    if (((((uint32_t)(uintptr_t)out >> 2) | ld | columns) & 1u) == 0) {
        const uint32_t l = lane & 7u, sub = lane >> 3;
        const bool live = 2u * l < columns;
        float* dst = out + (size_t)sub * ld + 2u * l;
        float2 v[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; i++) {
            const uint32_t r = 4u * i + sub;
            v[i] = *reinterpret_cast<const float2*>(tile + r * 64u + (((l >> 1) ^ ((r >> 1) & 3u)) << 4) + (l & 1u) * 8u);
        }
#pragma unroll
        for (uint32_t i = 0; i < 8; i++, dst += 4u * (size_t)ld)
            if (live && 4u * i + sub < rows) *reinterpret_cast<float2*>(dst) = v[i];
    } else {
        const uint32_t l = lane & 15u, odd = lane >> 4;
        const bool live = l < columns;
        float* dst = out + (size_t)odd * ld + l;
        float v[16];
#pragma unroll
        for (uint32_t i = 0; i < 16; i++) v[i] = *reinterpret_cast<const float*>(tile + (2u * i + odd) * 64u + (((l >> 2) ^ (i & 3u)) << 4) + (l & 3u) * 4u);
#pragma unroll
        for (uint32_t i = 0; i < 16; i++, dst += 2u * (size_t)ld)
            if (live && 2u * i + odd < rows) *dst = v[i];
    }
}

// The SiLU * Mul tail leaves 16 outputs of a 32-channel chunk: this lane's row in y, to out as store_words does.
__device__ __forceinline__ void store_half_words(uint8_t* tile, uint32_t lane, const float (&y)[16], float* out, uint32_t ld,
                                                 uint32_t rows, uint32_t columns, bool aligned) {
    __syncwarp();
#pragma unroll
    for (uint32_t j = 0; j < 4; j++)
        *reinterpret_cast<float4*>(tile + lane * 64u + ((j ^ ((lane >> 1) & 3u)) << 4)) = make_float4(y[4 * j], y[4 * j + 1], y[4 * j + 2], y[4 * j + 3]);
    __syncwarp();
    if (aligned) {
        const uint32_t piece = lane & 3u;
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const uint32_t r = 8u * i + (lane >> 2);
            const float4 v = *reinterpret_cast<const float4*>(tile + r * 64u + ((piece ^ ((r >> 1) & 3u)) << 4));
            if (r < rows) *reinterpret_cast<float4*>(out + (size_t)r * ld + 4u * piece) = v;
        }
    } else {
        flush_half_words(tile, lane, out, ld, rows, columns);
    }
}

}  // namespace vxb
