// Attention of a portion of a prompt behind keys that are already in the cache, in fp32: the passes that stand in for decode steps (later turns of a conversation,
// prompts over Q5_0 projections).  q and out [H][T][d], K and V [Hkv][kv_stride][d] with `before` + T rows, query token i sees keys 0 .. before + i; mathematics
// of attention_flash_decode (src/kernels/attention_flash_true.c:142-230).
//
// Such a call has the range and the accuracy of the steps that it replaces, which the fp16 pieces of attention_prefill_mma.cu do not: against 64 bits (512 tokens, 32 / 8
// heads of 128) 1.4e-7 of the result where decode steps give 1.3e-7, in pieces 7.6e-7, and 5.8e-6 for values around 0.003, whose low pieces are below
// fp16's normal range.  Chains of additions are kept short for it: 16 terms in each of two per 32 dimensions of a score, 16 keys of an output.
//
// A CTA owns one kv head and 64 query rows (tokens x the query heads of that kv head), 128 threads in 16 x 8.  Per tile of 64 keys a thread computes 8 x 4
// scores (four dimensions a step: twelve 16-byte loads for 128 multiply-adds) and, with the probabilities passed through shared memory inside its half-warp,
// 8 rows x d / 16 outputs; packed fp32 FMAs, two to an instruction.  16-byte pieces of a row are permuted by the row's low bits, so that the keys of a load lie
// in all banks.  112 KB of shared memory at d = 128, two CTAs per SM: one's copies run under the other's products.  What bounds it is the loads from shared memory
// (640 of a warp and tile for 4096 packed FMAs): 44 % of the fp32 rate behind 16000 keys (512 tokens of the heads above: 4.3 ms; tiles of 4 x 4 a thread, 256 threads: 5.6).
// Few query blocks leave most SMs idle: the keys are then split over CTAs and the parts merged by a second launch (16 tokens behind 16000 keys: 178 us; one CTA per
// kv head would take 4 ms).
#include <math.h>

#include "device_common.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "runtime.h"

namespace ckb {

constexpr int AB_ROWS = 64, AB_BK = 64, AB_THREADS = 128, AB_R = 8;      // rows of a thread
constexpr int AB_MAX_GROUP = 8;      // query heads per kv head on this path
constexpr int AB_MAX_SPLITS = 64;

struct AbParams {
    const float *q, *k, *v;
    float *out, *part;               // part: [split][H][T][AD] unnormalised, then [split][H][T] (maximum, sum)
    int H, Hkv, T, before, kv_stride, BT, splits;
    float scale;                     // log2(e) included
};

__device__ __forceinline__ uint64_t ab_fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t ab_mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t ab_add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t ab_pack(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ float2 ab_unpack(uint64_t v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ void ab_lds2(uint32_t addr, uint64_t &a, uint64_t &b) { asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr)); }
__device__ __forceinline__ void ab_cp16(uint32_t dst, const void *src, uint32_t bytes)     // bytes = 0: sixteen zeros
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
template <int AD> constexpr int ab_smem_bytes() { return (3 * AB_ROWS * AD + AB_ROWS * AB_BK) * 4; }

// row r of the CTA: token t0 + r / G, query head kvh * G + r % G
template <int AD>
__global__ void __launch_bounds__(AB_THREADS, 2) attn_behind_kernel(const __grid_constant__ AbParams p)
{
    constexpr int PC = AD / 4, NP = AD / 32;                 // 16-byte pieces of a row; output pairs of a thread and row
    extern __shared__ __align__(16) float ab_smem[];
    const uint32_t sQ = smem_u32(ab_smem), sK = sQ + AB_ROWS * AD * 4, sV = sK + AB_BK * AD * 4, sP = sV + AB_BK * AD * 4;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int G = p.H / p.Hkv, kvh = blockIdx.y, t0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * p.BT;      // blocks with the most keys first
    const int end = p.before + min(p.T, t0 + p.BT), tiles = (end + AB_BK - 1) / AB_BK, per = (tiles + p.splits - 1) / p.splits;
    const int tile0 = (int)blockIdx.z * per, tile1 = min(tiles, tile0 + per);
    const float *kbase = p.k + (size_t)kvh * p.kv_stride * AD, *vbase = p.v + (size_t)kvh * p.kv_stride * AD;
    pdl_wait();
    pdl_trigger();

    auto load = [&](const float *base, uint32_t dst, int tile, bool permuted) {         // keys past the end of the block's range read as zeros
        const int key0 = tile * AB_BK;
#pragma unroll 4
        for (int i = tid; i < AB_BK * PC; i += AB_THREADS) {
            const int row = i / PC, c = i % PC, key = key0 + row;
            ab_cp16(dst + (uint32_t)(row * PC + (permuted ? c ^ (row & 7) : c)) * 16u, base + (size_t)min(key, end - 1) * AD + 4 * c, key < end ? 16u : 0u);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (tile0 < tile1) {
        load(kbase, sK, tile0, true);
        load(vbase, sV, tile0, false);
    }
    for (int i = tid; i < AB_ROWS * PC; i += AB_THREADS) {
        const int r = i / PC, c = i % PC, t = t0 + r / G;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < p.T && r < p.BT * G) x = __ldcg(reinterpret_cast<const float4 *>(p.q + ((size_t)(kvh * G + r % G) * p.T + t) * AD) + c);
        reinterpret_cast<float4 *>(ab_smem)[r * PC + (c ^ (r & 7))] = make_float4(x.x * p.scale, x.y * p.scale, x.z * p.scale, x.w * p.scale);
    }
    int pos[AB_R];                                           // place of rows ty + 8 i in the sequence
    uint64_t o[AB_R][NP];
    float m[AB_R], l[AB_R];
#pragma unroll
    for (int i = 0; i < AB_R; ++i) {
        pos[i] = p.before + t0 + (ty + 8 * i) / G;
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (int n = 0; n < NP; ++n) o[i][n] = 0;
    }
    const uint32_t qrow = sQ + (uint32_t)ty * AD * 4, krow = sK + (uint32_t)tx * AD * 4, prow = sP + (uint32_t)ty * AB_BK * 4;
    const uint32_t flip = (uint32_t)(ty & 1);                // the two rows of a warp's broadcast loads of probabilities lie in different banks

#pragma unroll 1
    for (int tile = tile0; tile < tile1; ++tile) {
        const int key0 = tile * AB_BK;
        asm volatile("cp.async.wait_group 1;" ::: "memory");                   // the keys have landed
        __syncthreads();
        float s[AB_R][4];
#pragma unroll
        for (int i = 0; i < AB_R; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
#pragma unroll 1
        for (int c0 = 0; c0 < PC; c0 += 8) {                                   // 32 dimensions at a time, two chains of 16
            uint64_t acc[AB_R][4];
#pragma unroll
            for (int i = 0; i < AB_R; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                uint64_t ka[4], kb[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) ab_lds2(krow + (uint32_t)(16 * j * PC + ((c0 + c) ^ (tx & 7))) * 16u, ka[j], kb[j]);
#pragma unroll
                for (int i = 0; i < AB_R; ++i) {
                    uint64_t qa, qb;
                    ab_lds2(qrow + (uint32_t)(8 * i * PC + ((c0 + c) ^ (ty & 7))) * 16u, qa, qb);
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = ab_fma2(qb, kb[j], ab_fma2(qa, ka[j], acc[i][j]));
                }
            }
#pragma unroll
            for (int i = 0; i < AB_R; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) { const float2 a = ab_unpack(acc[i][j]); s[i][j] += a.x + a.y; }
        }
        // In a tile with keys that some row of the CTA does not see those are left out one by one: their weight is 0, but 0 x inf is not.
        const bool edge = key0 + AB_BK > p.before + t0 + 1;
        if (edge) {
#pragma unroll
            for (int i = 0; i < AB_R; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (key0 + tx + 16 * j > pos[i]) s[i][j] = -INFINITY;
        }
        __syncthreads();
        if (tile + 1 < tile1) load(kbase, sK, tile + 1, true);
        else asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int i = 0; i < AB_R; ++i) {
            float top = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
            top = fmaxf(m[i], top);
            const float ref = top == -INFINITY ? 0.0f : top;                   // a row may have seen no key yet
            const float corr = m[i] == -INFINITY ? 0.0f : exp2f(m[i] - ref);
            m[i] = top;
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float pr = s[i][j] == -INFINITY ? 0.0f : exp2f(s[i][j] - ref);
                sum += pr;
                const uint32_t piece = (uint32_t)((tx + 16 * j) >> 2) ^ flip;
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(prow + (uint32_t)(8 * i) * AB_BK * 4 + piece * 16u + (uint32_t)(tx & 3) * 4u), "f"(pr) : "memory");
            }
            l[i] = fmaf(l[i], corr, sum);
            const uint64_t c2 = ab_pack(corr, corr);
#pragma unroll
            for (int n = 0; n < NP; ++n) o[i][n] = ab_mul2(o[i][n], c2);
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");                   // the values have landed
        __syncthreads();
#pragma unroll 1
        for (int kq0 = 0; kq0 < AB_BK / 4; kq0 += 4) {                     // 16 keys at a time
            uint64_t acc[AB_R][NP];
#pragma unroll
            for (int i = 0; i < AB_R; ++i)
#pragma unroll
                for (int n = 0; n < NP; ++n) acc[i][n] = 0;
#pragma unroll 1
            for (int kq = kq0; kq < kq0 + 4; ++kq) {
                float pr[AB_R][4];
#pragma unroll
                for (int i = 0; i < AB_R; ++i)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(pr[i][0]), "=f"(pr[i][1]), "=f"(pr[i][2]), "=f"(pr[i][3]) : "r"(prow + (uint32_t)(8 * i) * AB_BK * 4 + ((uint32_t)kq ^ flip) * 16u));
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint64_t v[NP];
#pragma unroll
                    for (int n = 0; n < NP; n += 2) ab_lds2(sV + (uint32_t)((4 * kq + kk) * AD + 4 * tx + 32 * n) * 4u, v[n], v[n + 1]);
                    if (edge) {
#pragma unroll
                        for (int i = 0; i < AB_R; ++i)
                            if (key0 + 4 * kq + kk <= pos[i]) {
                                const uint64_t w = ab_pack(pr[i][kk], pr[i][kk]);
#pragma unroll
                                for (int n = 0; n < NP; ++n) acc[i][n] = ab_fma2(w, v[n], acc[i][n]);
                            }
                    } else {
#pragma unroll
                        for (int i = 0; i < AB_R; ++i) {
                            const uint64_t w = ab_pack(pr[i][kk], pr[i][kk]);
#pragma unroll
                            for (int n = 0; n < NP; ++n) acc[i][n] = ab_fma2(w, v[n], acc[i][n]);
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < AB_R; ++i)
#pragma unroll
                for (int n = 0; n < NP; ++n) o[i][n] = ab_add2(o[i][n], acc[i][n]);
        }
        __syncthreads();
        if (tile + 1 < tile1) load(vbase, sV, tile + 1, false);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

#pragma unroll
    for (int i = 0; i < AB_R; ++i) {
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], w);
        const int r = ty + 8 * i, t = t0 + r / G, h = kvh * G + r % G;
        if (r >= p.BT * G || t >= p.T) continue;
        const size_t at = (size_t)h * p.T + t, rows = (size_t)p.H * p.T;
        float *dst = p.splits > 1 ? p.part + ((size_t)blockIdx.z * rows + at) * AD : p.out + at * AD;
        if (p.splits > 1 && tx == 0) reinterpret_cast<float2 *>(p.part + (size_t)p.splits * rows * AD)[(size_t)blockIdx.z * rows + at] = make_float2(m[i], l[i]);
#pragma unroll
        for (int n = 0; n < NP; n += 2) {
            const float2 a = ab_unpack(o[i][n]), b = ab_unpack(o[i][n + 1]);
            float4 x = make_float4(a.x, a.y, b.x, b.y);
            const int d = 4 * tx + 32 * n;
            if (p.splits == 1) {
                const float sum = l[i];
                x = sum > 0.0f || sum != sum ? make_float4(x.x / sum, x.y / sum, x.z / sum, x.w / sum) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            *reinterpret_cast<float4 *>(dst + d) = x;
        }
    }
}

// the parts of a split, in their order: a warp per query row
template <int AD>
__global__ void __launch_bounds__(256) attn_behind_merge_kernel(const float *__restrict__ part, float *__restrict__ out, int rows, int splits)
{
    constexpr int E = AD / 32;
    const int lane = threadIdx.x & 31, row = (int)blockIdx.x * 8 + ((int)threadIdx.x >> 5);
    pdl_wait();
    pdl_trigger();
    if (row >= rows) return;
    const float2 *ml = reinterpret_cast<const float2 *>(part + (size_t)splits * rows * AD) + row;
    const float2 a = lane < splits ? __ldcg(ml + (size_t)lane * rows) : make_float2(-INFINITY, 0.0f);
    const float2 b = lane + 32 < splits ? __ldcg(ml + (size_t)(lane + 32) * rows) : make_float2(-INFINITY, 0.0f);
    float top = fmaxf(a.x, b.x);
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
    const float wa = a.x == -INFINITY ? 0.0f : exp2f(a.x - top), wb = b.x == -INFINITY ? 0.0f : exp2f(b.x - top);
    const float sum = group_sum<32>(fmaf(wa, a.y, wb * b.y));
    float acc[E] = {};
    for (int z = 0; z < splits; ++z) {
        const float w = __shfl_sync(0xffffffffu, z < 32 ? wa : wb, z & 31);
        if (w == 0.0f) continue;
        const float *src = part + ((size_t)z * rows + row) * AD + lane * E;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e] = fmaf(w, __ldcg(src + e), acc[e]);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) out[(size_t)row * AD + lane * E + e] = sum > 0.0f || sum != sum ? acc[e] / sum : 0.0f;
}

// Splits of the keys: enough CTAs for two on every SM, two tiles of keys to each at least (a part costs its copy of the queries and its share of the merge;
// 16 tokens behind 1024 keys: 50 us, with four tiles at least 73)
static int ab_splits(int blocks, int num_kv_heads, int keys)
{
    const int units = blocks * num_kv_heads, tiles = (keys + AB_BK - 1) / AB_BK;
    int z = 2 * ckb_sm_count() / units;
    if (z > tiles / 2) z = tiles / 2;
    return z < 1 ? 1 : (z > AB_MAX_SPLITS ? AB_MAX_SPLITS : z);
}

template <int AD>
static int ab_launch(AbParams p, cudaStream_t st)
{
    static bool attr_set = false;
    if (!attr_set) {
        if (ckb_check_cuda((int)cudaFuncSetAttribute(attn_behind_kernel<AD>, cudaFuncAttributeMaxDynamicSharedMemorySize, ab_smem_bytes<AD>()), "attn_behind smem")) return CKB_ERR_CUDA;
        attr_set = true;
    }
    if (int rc = launch_pdl("attn_behind", attn_behind_kernel<AD>, dim3((p.T + p.BT - 1) / p.BT, p.Hkv, p.splits), dim3(AB_THREADS), (size_t)ab_smem_bytes<AD>(), st, p)) return rc;
    if (p.splits == 1) return 0;
    const int rows = p.H * p.T;
    return launch_pdl("attn_behind_merge", attn_behind_merge_kernel<AD>, dim3((rows + 7) / 8), dim3(256), (size_t)0, st, (const float *)p.part, p.out, rows, p.splits);
}

}  // namespace ckb

using namespace ckb;

// A portion of a prompt behind `before` keys of earlier ones, causal, in fp32.  `part`: scratch for the parts of a split, whatever the number of tokens and keys
// (the split fills two CTAs an SM at most, of 64 rows each).
extern "C" size_t ckb_attn_behind_part_bytes(int head_dim) { return (size_t)2 * ckb_sm_count() * AB_ROWS * (head_dim + 2) * sizeof(float); }
extern "C" int ckb_launch_attn_behind(const float *q, const float *k, const float *v, float *out, int num_heads, int num_kv_heads, int num_tokens, int head_dim,
                                      int kv_stride_tokens, int before, float *part, void *stream)
{
    const int G = num_heads / num_kv_heads;
    if (num_heads % num_kv_heads || G > AB_MAX_GROUP || (head_dim != 64 && head_dim != 128) || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out | (uintptr_t)part) & 15))
        return ckb_fail(CKB_ERR_SHAPE, "attention behind earlier keys: %d heads, %d kv heads, head size %d", num_heads, num_kv_heads, head_dim);
    const int BT = AB_ROWS / G;
    const AbParams p = { q, k, v, out, part, num_heads, num_kv_heads, num_tokens, before, kv_stride_tokens, BT, ab_splits((num_tokens + BT - 1) / BT, num_kv_heads, before + num_tokens),
                         1.0f / sqrtf((float)head_dim) * 1.44269504088896340736f };
    return head_dim == 64 ? ab_launch<64>(p, ckb_stream(stream)) : ab_launch<128>(p, ckb_stream(stream));
}
