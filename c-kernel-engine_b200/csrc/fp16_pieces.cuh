// A float as two fp16 pieces: the nearest, and the nearest to what that leaves (22 bits of the mantissa while the value is in fp16's normal range).
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace ckb {

__device__ __forceinline__ void pm_split2(float a, float b, uint32_t &hi, uint32_t &lo)
{
    const __half2 h = __floats2half2_rn(a, b);
    const float2 hf = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - hf.x, b - hf.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
// four in a row, to hi[at .. at + 3] and `arr` halves further on
__device__ __forceinline__ void store_pieces4(__half *at, size_t arr, const float4 &v)
{
    uint2 hi, lo;
    pm_split2(v.x, v.y, hi.x, lo.x);
    pm_split2(v.z, v.w, hi.y, lo.y);
    *reinterpret_cast<uint2 *>(at) = hi;
    *reinterpret_cast<uint2 *>(at + arr) = lo;
}

}  // namespace ckb
