// Where a reconstructed row chunk goes (dequantise: stored; verify: compared). chunk() takes the lane's 16 weights of chunk
// c of row r as eight BF16x2 words; one() a NIBBLE escape.
#pragma once

#include "decode.cuh"

namespace b16 {
namespace dev {

// chunk c of a gathered row
template <bool BF>
__device__ __forceinline__ void put_row_chunk(char * o, int c, int lane, const uint32_t (&w)[8]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int i = c * CHUNK + 128 * j + 4 * lane;
        if (BF) {
            *(uint2 *) (o + 2 * i) = make_uint2(w[2 * j], w[2 * j + 1]);
        } else {
            *(float4 *) (o + 4 * i) = make_float4(bf16lo_f32(w[2 * j]), bf16hi_f32(w[2 * j]), bf16lo_f32(w[2 * j + 1]), bf16hi_f32(w[2 * j + 1]));
        }
    }
}

struct StoreBF16 { // row-major BF16 output
    uint16_t * out;
    int64_t K;
    __device__ __forceinline__ void chunk(int64_t r, int c, int lane, const uint32_t (&w)[8]) {
        uint16_t * o = out + r * K + c * CHUNK + 4 * lane;
#pragma unroll
        for (int j = 0; j < 4; j++) { *(uint2 *) (o + 128 * j) = make_uint2(w[2 * j], w[2 * j + 1]); }
    }
    __device__ __forceinline__ void one(int64_t r, int col, uint32_t bits) { out[r * K + col] = (uint16_t) bits; }
    __device__ __forceinline__ void finish(int) {}
};

struct CompareBF16 { // count words that differ from src
    const uint16_t * src;
    int64_t K;
    unsigned long long * total;
    unsigned int bad;
    __device__ __forceinline__ void chunk(int64_t r, int c, int lane, const uint32_t (&w)[8]) {
        const uint16_t * o = src + r * K + c * CHUNK + 4 * lane;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint2 s = __ldg((const uint2 *) (o + 128 * j));
            const uint32_t d0 = s.x ^ w[2 * j], d1 = s.y ^ w[2 * j + 1];
            bad += ((d0 & 0xFFFFu) != 0) + ((d0 >> 16) != 0) + ((d1 & 0xFFFFu) != 0) + ((d1 >> 16) != 0);
        }
    }
    // NIBBLE escapes: the dense pass saw +0 where src holds the escaped value, so every escape that matches its source
    // takes back one counted difference (and a wrong one keeps it)
    __device__ __forceinline__ void one(int64_t r, int col, uint32_t bits) {
        const uint32_t s = src[r * K + col];
        if (s != 0) { bad -= 1; }
        if (s != bits) { bad += 1; }
    }
    __device__ __forceinline__ void finish(int lane) {
        unsigned int b = bad;
#pragma unroll
        for (int o = 16; o; o >>= 1) { b += __shfl_xor_sync(FULL, b, o); }
        if (lane == 0 && b) { atomicAdd(total, (unsigned long long) b); }
    }
};

} // namespace dev
} // namespace b16
