// One warp quantises one 256-element block to Q8_K; lane l holds elements 8l..8l+7 in v[].
// Bit-exact with the reference's quantize_row_q8_k (src/kernels/gemm_kernels_q4k_q8k.c:53-103):
// the SIGNED value of the first element with the largest |x| sets the scale (ties: the lowest index), iscale = -127/max and d = 1/iscale are IEEE divisions,
// and iscale*x is rounded to fp32 before the round-to-nearest-even conversion.
#pragma once

#include "device_common.cuh"

namespace ckb {

// the eight quants of this lane (all zero, d = 0 for a block of zeros), their sum, and the block scale (in every lane)
struct Q8kLane { int q[8], s; float d; };
__device__ __forceinline__ Q8kLane quantize_lane_q8k(const float (&v)[8], int lane)
{
    float best = 0.0f, mine = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float ax = fabsf(v[j]);
        if (ax > best) { best = ax; mine = v[j]; }
    }
    // non-negative floats order like their bits: one warp reduction instead of five rounds of (value, index) shuffles, a chain of 250 cycles; the lowest
    // lane that has the maximum holds its first occurrence
    const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(best));
    const float vmax = __shfl_sync(0xffffffffu, mine, __ffs(__ballot_sync(0xffffffffu, __float_as_uint(best) == top)) - 1);
    best = __uint_as_float(top);

    Q8kLane r;
    r.s = 0;
    r.d = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) r.q[j] = 0;
    if (best == 0.0f) return r;
    const float iscale = __fdiv_rn(-127.0f, vmax);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        r.q[j] = max(-128, min(127, __float2int_rn(__fmul_rn(iscale, v[j]))));
        r.s += r.q[j];
    }
    r.d = __fdiv_rn(1.0f, iscale);
    return r;
}

__device__ __forceinline__ void quantize_block_q8k(const float (&v)[8], uint8_t *out, int lane)
{
    const Q8kLane r = quantize_lane_q8k(v, lane);
    const uint32_t w0 = (r.q[0] & 255) | ((r.q[1] & 255) << 8) | ((r.q[2] & 255) << 16) | ((uint32_t)(r.q[3] & 255) << 24);
    const uint32_t w1 = (r.q[4] & 255) | ((r.q[5] & 255) << 8) | ((r.q[6] & 255) << 16) | ((uint32_t)(r.q[7] & 255) << 24);
    reinterpret_cast<uint32_t *>(out + 4)[2 * lane] = w0;
    reinterpret_cast<uint32_t *>(out + 4)[2 * lane + 1] = w1;
    const int s = r.s + __shfl_xor_sync(0xffffffffu, r.s, 1);   // the 16-element sum lives in both lanes of a pair
    if ((lane & 1) == 0) reinterpret_cast<int16_t *>(out + 260)[lane >> 1] = (int16_t)s;
    if (lane == 0) *reinterpret_cast<float *>(out) = r.d;
}

// The same block as operand of the tensor-core product (gemm_tc.cu): token `tok` of a blob of `nt` tokens and this superblock: fp16 quants in 8-element
// k-chunks of nt x 16 bytes (order 0 2 1 3 4 6 5 7 inside a chunk), the 16 sums as two chunks behind them, then the nt block scales.
__host__ __device__ constexpr size_t q8k_tile_bytes(int nt) { return (size_t)nt * (16 * 34 + 4); }
__device__ __forceinline__ void quantize_block_q8k_tile(const float (&v)[8], uint8_t *blob, int nt, int tok, int lane)
{
    const Q8kLane r = quantize_lane_q8k(v, lane);
    constexpr int order[8] = {0, 2, 1, 3, 4, 6, 5, 7};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 h = __floats2half2_rn((float)r.q[order[2 * i]], (float)r.q[order[2 * i + 1]]);
        o[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
    uint8_t *at = blob + tok * 16;
    *reinterpret_cast<uint4 *>(at + (size_t)lane * nt * 16) = make_uint4(o[0], o[1], o[2], o[3]);
    const int s = r.s + __shfl_xor_sync(0xffffffffu, r.s, 1);
    if ((lane & 1) == 0) *reinterpret_cast<__half *>(at + (size_t)(32 + (lane >> 4)) * nt * 16 + (lane >> 1 & 7) * 2) = __int2half_rn(s);
    if (lane == 0) reinterpret_cast<float *>(blob + (size_t)nt * (16 * 34))[tok] = r.d;
}

}  // namespace ckb
