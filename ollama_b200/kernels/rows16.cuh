// Activations in 16 bits, in the order that gemm_sk.cu multiplies them.
#pragma once
#include "common.cuh"

constexpr int SG_ROW = 544, SG_CHUNK = 16 * (SG_ROW + 4);      // bytes of a row's 256-block: values and sums of 32; with the scales of 16 rows
constexpr int SG_MAX_ROWS = 64;

// One row's 256-block by a warp, a lane its columns 8 lane .. + 7.  A 256-block of `n` rows: [64 columns][n rows][128 bytes, 16-byte pieces xor row & 7] values, [two parts][n rows][16 bytes] sums of 32 (upper f16 parts of the eight, then
// lower parts), [n] scales.  Place 8 j + 2 t + e of 64 columns holds column 32 (j / 4) + 16 (j / 2 & 1) + 4 t + (j & 1) + 2 e.
__device__ __forceinline__ void store_block16(uint8_t* out, int n, int row, int blk, int lane, const float (&v)[8]) {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) m = fmaxf(m, fabsf(v[i]));
    m = warp_max(m);
    const int e = max((int)(__float_as_uint(m) >> 23), 16);                        // scale 2^(e - 135): the largest value lands in 256..512
    const float inv = __uint_as_float((uint32_t)(262 - e) << 23), scale = __uint_as_float((uint32_t)(e - 8) << 23);
    __half h[8];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        h[i] = __float2half_rn(v[i] * inv);
        sum += __half2float(h[i]);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);                                    // the 32 columns of four lanes
    uint8_t* c = out + (size_t)blk * n * (SG_ROW + 4);
    // lane: columns 8 lane .. + 7 = t values 2 (lane & 1) and + 1 of 16-column group lane / 2
    const int j = 2 * ((lane >> 1) & 3);
    uint8_t* f = c + (size_t)((lane >> 3) * n + row) * 128 + 8 * (lane & 1);
    const __half2 p[4] = {__halves2half2(h[0], h[2]), __halves2half2(h[4], h[6]), __halves2half2(h[1], h[3]), __halves2half2(h[5], h[7])};
    *reinterpret_cast<uint2*>(f + ((j ^ (row & 7)) << 4)) = *reinterpret_cast<const uint2*>(p);
    *reinterpret_cast<uint2*>(f + (((j + 1) ^ (row & 7)) << 4)) = *reinterpret_cast<const uint2*>(p + 2);
    // sums of two neighbouring sub-blocks: lanes 8 i and 8 i + 4 hold them
    const float next = __shfl_down_sync(0xffffffffu, sum, 4);
    if ((lane & 7) == 0) {
        const __half h0 = __float2half_rn(sum), h1 = __float2half_rn(next);
        __half2* s = reinterpret_cast<__half2*>(c + (size_t)n * 512 + row * 16 + (lane >> 3) * 4);
        s[0] = __halves2half2(h0, h1);
        s[n * 4] = __halves2half2(__float2half_rn(sum - __half2float(h0)), __float2half_rn(next - __half2float(h1)));
    }
    if (lane == 0) *reinterpret_cast<float*>(c + (size_t)n * SG_ROW + row * 4) = scale;
}
