// The weight formats of the one-launch decode step (step_persistent.cu): loading a lane's part of a block, multiplying a pair of rows, quantising 256 elements of
// the input row into the layout that the products read.  In a header because the integer-stage dump (subblock_sums.cu) runs the same functions.
#pragma once

#include "add_rmsnorm_q8k.cuh"
#include "q4p_unit.cuh"
#include "q6p_unit.cuh"

namespace ckb {

__device__ __forceinline__ uint2 ps_pack8(const int (&q)[8])
{
    return make_uint2((q[0] & 255) | ((q[1] & 255) << 8) | ((q[2] & 255) << 16) | ((uint32_t)(q[3] & 255) << 24),
                      (q[4] & 255) | ((q[5] & 255) << 8) | ((q[6] & 255) << 16) | ((uint32_t)(q[7] & 255) << 24));
}

// `pair`: both rows of a lane's pair against its part of a block, the activations read once, with plain loads that the compiler may place early.
struct PsQ4 {                                 // two lanes per superblock
    using W = Q4pW;
    static constexpr int LPS = 2;
    static constexpr bool DEEP = false;       // the next rows in registers of their own while a pair is multiplied (else in the same ones, behind it)
    static __host__ __device__ __forceinline__ size_t row_bytes(int nb) { return (size_t)nb * Q4K_BYTES; }
    static __device__ __forceinline__ void load(W &w, const uint8_t *row, int, int b, int u)
    {
        const uint8_t *pb = row + b * Q4K_BYTES;
        w.hdr = __ldg(reinterpret_cast<const uint4 *>(pb));
        w.a0 = __ldg(reinterpret_cast<const uint4 *>(pb + 16 + 32 * u));
        w.a1 = __ldg(reinterpret_cast<const uint4 *>(pb + 32 + 32 * u));
        w.b0 = __ldg(reinterpret_cast<const uint4 *>(pb + 80 + 32 * u));
        w.b1 = __ldg(reinterpret_cast<const uint4 *>(pb + 96 + 32 * u));
    }
    // 32-element sums of both rows: lo[r][q] and hi[r][q] / 16 are sub-blocks 2 p + 4 q and 2 p + 4 q + 1
    static __device__ __forceinline__ void isums(const Q4pW &w0, const Q4pW &w1, const uint8_t *s, int b, int p, int (&lo)[2][2], int (&hi)[2][2])
    {
        const Q4pW *w[2] = {&w0, &w1};
        const uint8_t *xs = s + (b * Q4P_SLOTS + 4 * p) * 16;
#pragma unroll
        for (int r = 0; r < 2; ++r) lo[r][0] = lo[r][1] = hi[r][0] = hi[r][1] = 0;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint4 *x = reinterpret_cast<const uint4 *>(xs + 128 * q);
            const uint4 l0 = x[0], l1 = x[1], h0 = x[2], h1 = x[3];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint4 c0 = q ? w[r]->b0 : w[r]->a0, c1 = q ? w[r]->b1 : w[r]->a1;
                const uint32_t c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w}, l[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w},
                               h[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    lo[r][q] = dp4a_us(c[i] & 0x0F0F0F0Fu, l[i], lo[r][q]);
                    hi[r][q] = dp4a_us(c[i] & 0xF0F0F0F0u, h[i], hi[r][q]);      // 16 x the high-nibble sum
                }
            }
        }
    }
    static __device__ __forceinline__ void pair(const Q4pW &w0, const Q4pW &w1, const uint8_t *s, int nb, int b, int p, float &a0, float &a1)
    {
        int lo[2][2], hi[2][2];
        const uint8_t *d = s + nb * Q4P_SLOTS * 16, *sums = d + nb * 4 + 4 * (2 * b + p);
        const uint32_t blo = *reinterpret_cast<const uint32_t *>(sums), bhi = *reinterpret_cast<const uint32_t *>(sums + nb * 8);
        const float xd = *reinterpret_cast<const float *>(d + 4 * b);
        isums(w0, w1, s, b, p, lo, hi);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint4 hdr = r ? w1.hdr : w0.hdr;
            const int t = 16 * p;
            const uint32_t a = hdr.y >> t, bb = hdr.z >> t, c = hdr.w >> t;
            const uint32_t scA = a & 0x3F3Fu, mA = bb & 0x3F3Fu, scB = (c & 0x0F0Fu) | ((a >> 2) & 0x3030u), mB = ((c >> 4) & 0x0F0Fu) | ((bb >> 2) & 0x3030u);
            const int isum = (int)(scA & 255u) * lo[r][0] + (int)(scB & 255u) * lo[r][1] + (((int)(scA >> 8) * hi[r][0] + (int)(scB >> 8) * hi[r][1]) >> 4);
            const uint32_t m4 = mA | (mB << 16);
            const int imin = dp4a_us(m4, blo, 0) + 128 * dp4a_us(m4, bhi, 0);
            const float2 dd = __half22float2(*reinterpret_cast<const __half2 *>(&hdr.x));
            (r ? a1 : a0) += (dd.x * xd) * (float)isum - (dd.y * xd) * (float)imin;
        }
    }
    // elements 256 b + 8 lane .. + 7, as q4p_stage_x lays them out
    static __device__ __forceinline__ void put(const float (&v)[8], int b, int nb, int lane, uint8_t *s)
    {
        const Q8kLane r = quantize_lane_q8k(v, lane);
        *reinterpret_cast<uint2 *>(s + (size_t)b * Q4P_SLOTS * 16 + 8 * lane) = ps_pack8(r.q);
        int sum = r.s + __shfl_xor_sync(0xffffffffu, r.s, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        uint8_t *d = s + (size_t)nb * Q4P_SLOTS * 16, *lo = d + nb * 4, *hi = lo + nb * 8;
        if ((lane & 3) == 0) {
            const int j = lane >> 2, at = (b * 2 + ((j >> 1) & 1)) * 4 + ((j & 1) | ((j >> 2) << 1));
            lo[at] = (uint8_t)(sum & 127);
            hi[at] = (uint8_t)(sum >> 7);
        }
        if (lane == 0) reinterpret_cast<float *>(d)[b] = r.d;
    }
};

struct PsQ6 {                                 // four lanes per superblock
    using W = Q6pW;
    static constexpr int LPS = 4;
    static constexpr bool DEEP = true;
    static __host__ __device__ __forceinline__ size_t row_bytes(int nb) { return q6p_row_bytes(nb); }
    static __device__ __forceinline__ void load(W &w, const uint8_t *row, int nb, int b, int u) { q6p_load(w, row, nb, b, u >> 1, u & 1); }
    struct X { uint4 q[4]; uint32_t lo4, hi4; float d; };      // the quarter's activations, its four block sums as 128 hi + lo, the block scale
    static __device__ __forceinline__ X input(const uint8_t *s, int nb, int b, int u)
    {
        const uint8_t *d = s + nb * 320, *sums = d + nb * 4 + 4 * (b * 4 + u);
        const uint4 *x = reinterpret_cast<const uint4 *>(s + b * 320 + (10 * (u >> 1) + (u & 1)) * 16);
        return {{x[0], x[2], x[4], x[6]}, *reinterpret_cast<const uint32_t *>(sums), *reinterpret_cast<const uint32_t *>(sums + nb * 16), *reinterpret_cast<const float *>(d + 4 * b)};
    }
    static __device__ __forceinline__ void pair(const W &w0, const W &w1, const uint8_t *s, int nb, int b, int u, float &a0, float &a1)
    {
        const X x = input(s, nb, b, u);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const W &w = r ? w1 : w0;
            int S1, S2, S3, S4;
            q6k_plane_sums(w.qa, w.qb, w.qh, x.q[0], x.q[1], x.q[2], x.q[3], S1, S2, S3, S4);
            const uint32_t sc4 = (u & 1) ? __byte_perm(w.sc.x, w.sc.y, 0x7531) : __byte_perm(w.sc.x, w.sc.y, 0x6420);      // scales of groups 8 n + h + {0, 2, 4, 6}
            const int s0 = (int)(int8_t)(sc4 & 255u), s1 = (int)(int8_t)((sc4 >> 8) & 255u), s2 = (int)(int8_t)((sc4 >> 16) & 255u), s3 = (int)sc4 >> 24;
            const int center = dp4a_ss(sc4, x.lo4, 0) + 128 * dp4a_ss(sc4, x.hi4, 0);
            const int tot = s0 * S1 + s1 * S2 + s2 * S3 + s3 * S4 - 32 * center;
            (r ? a1 : a0) += (half_bits_to_float(w.d) * x.d) * (float)tot;
        }
    }
    // as ring_stage_x lays them out
    static __device__ __forceinline__ void put(const float (&v)[8], int b, int nb, int lane, uint8_t *s)
    {
        const Q8kLane r = quantize_lane_q8k(v, lane);
        const int c = lane >> 1;
        *reinterpret_cast<uint2 *>(s + (size_t)b * 320 + (c + 2 * (c >> 3)) * 16 + 8 * (lane & 1)) = ps_pack8(r.q);
        const int sum = r.s + __shfl_xor_sync(0xffffffffu, r.s, 1);
        uint8_t *d = s + (size_t)nb * 320, *lo = d + nb * 4, *hi = lo + nb * 16;
        if ((lane & 1) == 0) {
            const int j = c >> 1, at = (b * 4 + (j >> 2) * 2 + (c & 1)) * 4 + (j & 3);
            lo[at] = (uint8_t)(sum & 127);
            hi[at] = (uint8_t)(sum >> 7);
        }
        if (lane == 0) reinterpret_cast<float *>(d)[b] = r.d;
    }
};

struct PsQ5 {                                 // one lane per 32-element block; the input row in Q8_0
    struct W { uint4 qs; uint32_t qh, d; };
    static constexpr int LPS = 1;
    static constexpr bool DEEP = true;
    static __host__ __device__ __forceinline__ size_t row_bytes(int nb) { return ((size_t)nb * Q50_BYTES + 15) & ~(size_t)15; }
    static __device__ __forceinline__ void load(W &w, const uint8_t *row, int nb, int b, int)
    {
        w.qs = __ldg(reinterpret_cast<const uint4 *>(row + (size_t)b * 16));
        w.qh = __ldg(reinterpret_cast<const uint32_t *>(row + (size_t)nb * 16 + (size_t)b * 4));
        w.d = ldg_nc_u16(row + (size_t)nb * 20 + (size_t)b * 2);
    }
    static __device__ __forceinline__ void pair(const W &w0, const W &w1, const uint8_t *s, int, int b, int, float &a0, float &a1)
    {
        a0 += q50_unit_presum(w0.d, w0.qh, w0.qs, smem_u32(s) + 48u * b);
        a1 += q50_unit_presum(w1.d, w1.qh, w1.qs, smem_u32(s) + 48u * b);
    }
    // blocks 8 b .. 8 b + 7: four lanes each, 48-byte slots of quants, scale (rounded to fp16) and sum of the quants
    static __device__ __forceinline__ void put(const float (&v)[8], int b, int nb, int lane, uint8_t *s)
    {
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const float id = amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
        int q[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            q[j] = __float2int_rn(__fmul_rn(v[j], id));
            sum += (int)(int8_t)(q[j] & 255);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        const int blk = 8 * b + (lane >> 2);
        if (blk >= nb) return;
        uint8_t *slot = s + (size_t)blk * 48;
        *reinterpret_cast<uint2 *>(slot + 8 * (lane & 3)) = ps_pack8(q);
        if ((lane & 3) == 0) {
            *reinterpret_cast<float *>(slot + 32) = __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f)));
            *reinterpret_cast<int *>(slot + 36) = sum;
        }
    }
};

}  // namespace ckb
