// Batched Q8_0 x Q8_0 product for prefill: C[M,N] = A_q8[M,K] . B[N,K]^T + bias, the reference's gemm_nt_q8_0_q8_0
// (src/kernels/gemm_batch_int8.c:87-120; the symbol version/v7/src/ck_parallel_prefill.h:44-48 dispatches).
//
// Both operands carry one fp16 scale per 32 elements, so the integer part of the product is a sum of 32 int8 x int8 terms per
// block and every block needs its own scale: C[m][n] = sum_b (sum_32 a q) * (d_a[m][b] * d_w[n][b]).  One integer tensor-core
// instruction (mma.sync m16n8k32, s8 x s8 -> s32) is exactly one block deep, so a warp issues one MMA per (16 x 8 outputs, block),
// converts the int32 block sums and adds them, scaled, to fp32 accumulators - block after block in the reference's order, which
// makes the result bit-identical to the scalar loop (int32 sums are exact, the fp32 operations are the same and in the same order).
//
// Operands come in the row-planar layout of gemv_q80_planar.cu (per row all quants, then all scales; the reference's 34-byte
// blocks are only 2-byte aligned), so tiles move with 16-byte cp.async into shared memory: four blocks (128 bytes of k) per stage, three stages;
// rows padded to 144 bytes in shared memory so that the eight rows a fragment load touches fall into different banks.  Every weight tile is
// read once per token tile instead of once per token.
//
// Q5_0 weights (gemm_nt_q5_0_q8_0, src/kernels/gemm_kernels_q5_0.c:1725-1752) run through the same kernel from their own planes (nibbles | fifth bits |
// scales, gemv_q50_planar.cu): word t of a block's 16 nibble bytes holds elements 4t .. 4t+3 and 16+4t .., exactly the two registers of lane t's fragment;
// five instructions a register make them signed bytes.  The sums are the same int32 and the fp32 steps the same, so these are bit-identical too.
//
// Tiles: 128 tokens x 128 rows, or 64 x 64 where the wide ones leave SMs idle, in their only round (the projections of a 896-wide model: 7 row tiles) or in their last.
#include "device_common.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "runtime.h"

namespace ckb {

constexpr int QM_KB = 4, QM_STAGES = 3, QM_THREADS = 256;
constexpr int QM_ROW = QM_KB * 32 + 16;                       // bytes of one row of signed bytes in shared memory (padded)
constexpr int QM_ROW5 = QM_KB * 16 + 16;                      // of one row of nibbles: 80 bytes, eight rows in different banks again
template <bool Q5, int TILE> struct QmTile {                  // TILE tokens x TILE weight rows
    static constexpr int A = TILE * QM_ROW, B = TILE * (Q5 ? QM_ROW5 : QM_ROW), FIFTH = Q5 ? TILE * QM_KB * 4 : 0, SCALES = TILE * QM_KB * 2;
    static constexpr int OFF_B = A, OFF_FIFTH = OFF_B + B, OFF_DA = OFF_FIFTH + FIFTH, OFF_DB = OFF_DA + SCALES, STAGE = OFF_DB + SCALES, SMEM = QM_STAGES * STAGE;
};

__host__ __device__ inline size_t qm_row_bytes(int nb) { return ((size_t)nb * Q80_BYTES + 15) & ~(size_t)15; }
__host__ __device__ inline size_t qm_row5_bytes(int nb) { return ((size_t)nb * Q50_BYTES + 15) & ~(size_t)15; }

// four elements of a Q5_0 block as signed bytes: nib - 16 * (fifth bit clear); fifth: their four bits, lowest first
__device__ __forceinline__ uint32_t q5_bytes(uint32_t nib, uint32_t fifth) { return nib | ((((~fifth & 15u) * 0x00204081u) & 0x01010101u) * 0xF0u); }

// rows past the end are filled with zeros, not fetched: copies of the last row in their place all went to one L2 slice (65 tokens x 4864 x 896: 44 us, with zeros 23)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool in) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory"); }
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src, bool in) { asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(in ? 8 : 0) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// A: row-planar Q8_0, B: row-planar Q8_0 or Q5_0 (rows of nb blocks, nb a multiple of QM_KB).  grid = (N tiles, M tiles).
template <bool Q5, int TILE>
__global__ void __launch_bounds__(QM_THREADS) gemm_q80_mma_kernel(const uint8_t *__restrict__ A, const uint8_t *__restrict__ B, const float *__restrict__ bias,
                                                                  float *__restrict__ C, int ldc, int M, int N, int nb, int weights_ready)
{
    using L = QmTile<Q5, TILE>;
    constexpr int MI = TILE / 32, NJ = TILE / 32;             // 16-token and 8-row fragments of a warp: 2 x 4 warps of TILE / 2 tokens x TILE / 4 rows
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t s_base = smem_u32(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp >> 2, wn = warp & 3;
    const int g = lane >> 2, t = lane & 3;
    const int m0 = blockIdx.y * TILE, n0 = blockIdx.x * TILE;
    const size_t ra = qm_row_bytes(nb), rb = Q5 ? qm_row5_bytes(nb) : ra;
    const int nchunks = nb / QM_KB;
    pdl_trigger();

    auto issue_b = [&](int chunk) {
        const uint32_t st = s_base + (uint32_t)(chunk % QM_STAGES) * L::STAGE;
        const int kb = chunk * QM_KB;
        constexpr int PIECES = Q5 ? 4 : 8;                    // 16-byte pieces of a row
#pragma unroll
        for (int i = 0; i < TILE * PIECES / QM_THREADS; ++i) {
            const int idx = tid + i * QM_THREADS, row = idx / PIECES, piece = idx % PIECES;
            cp_async16(st + L::OFF_B + (uint32_t)(row * (Q5 ? QM_ROW5 : QM_ROW) + piece * 16), B + (size_t)min(n0 + row, N - 1) * rb + (size_t)kb * (Q5 ? 16 : 32) + piece * 16, n0 + row < N);
        }
        if (tid < TILE) {
            const uint8_t *src = B + (size_t)min(n0 + tid, N - 1) * rb;
            if (Q5) cp_async16(st + L::OFF_FIFTH + (uint32_t)(tid * 16), src + (size_t)nb * 16 + (size_t)kb * 4, n0 + tid < N);
            cp_async8(st + L::OFF_DB + (uint32_t)(tid * 8), src + (size_t)nb * (Q5 ? 20 : 32) + (size_t)kb * 2, n0 + tid < N);
        }
    };
    auto issue_a = [&](int chunk) {
        const uint32_t st = s_base + (uint32_t)(chunk % QM_STAGES) * L::STAGE;
        const int kb = chunk * QM_KB;
#pragma unroll
        for (int i = 0; i < TILE * 8 / QM_THREADS; ++i) {
            const int idx = tid + i * QM_THREADS, row = idx >> 3, piece = idx & 7;
            cp_async16(st + (uint32_t)(row * QM_ROW + piece * 16), A + (size_t)min(m0 + row, M - 1) * ra + (size_t)kb * 32 + piece * 16, m0 + row < M);
        }
        if (tid >= QM_THREADS - TILE) {
            const int row = tid - (QM_THREADS - TILE);
            cp_async8(st + L::OFF_DA + (uint32_t)(row * 8), A + (size_t)min(m0 + row, M - 1) * ra + (size_t)nb * 32 + (size_t)kb * 2, m0 + row < M);
        }
    };

    float acc[MI][NJ][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;

    if (!weights_ready) pdl_wait();                           // resident weights are nobody's output; a copy re-laid by the kernel before this one is
    for (int c = 0; c < QM_STAGES - 1; ++c)
        if (c < nchunks) issue_b(c);
    pdl_wait();
    for (int c = 0; c < QM_STAGES - 1; ++c) {
        if (c < nchunks) issue_a(c);
        cp_async_commit();                                    // the first group holds the weights of both chunks
    }
    for (int c = 0; c < nchunks; ++c) {
        cp_async_wait<QM_STAGES - 2>();
        __syncthreads();                                      // chunk c has landed for everyone, and chunk c - 1's stage is free
        if (c + QM_STAGES - 1 < nchunks) { issue_b(c + QM_STAGES - 1); issue_a(c + QM_STAGES - 1); }
        cp_async_commit();
        const uint32_t st = s_base + (uint32_t)(c % QM_STAGES) * L::STAGE;
        const uint32_t sA = st + (uint32_t)((wm * (TILE / 2) + g) * QM_ROW + t * 4), sB = st + L::OFF_B + (uint32_t)((wn * (TILE / 4) + g) * (Q5 ? QM_ROW5 : QM_ROW) + t * 4);
        const uint32_t sF = st + L::OFF_FIFTH + (uint32_t)((wn * (TILE / 4) + g) * 16);
        const uint32_t sDA = st + L::OFF_DA + (uint32_t)((wm * (TILE / 2) + g) * 8), sDB = st + L::OFF_DB + (uint32_t)((wn * (TILE / 4) + 2 * t) * 8);
#pragma unroll
        for (int b = 0; b < QM_KB; ++b) {
            uint32_t af[MI][4], bf[NJ][2];
            float da[MI][2], db[NJ][2];
#pragma unroll
            for (int i = 0; i < MI; ++i) {                    // token rows 16 i + g and + 8
                const uint32_t p = sA + (uint32_t)(i * 16 * QM_ROW + b * 32);
                af[i][0] = lds_u32(p);
                af[i][1] = lds_u32(p + 8 * QM_ROW);
                af[i][2] = lds_u32(p + 16);
                af[i][3] = lds_u32(p + 8 * QM_ROW + 16);
                da[i][0] = half_bits_to_float(lds_u16(sDA + (uint32_t)(i * 16 * 8 + b * 2)));
                da[i][1] = half_bits_to_float(lds_u16(sDA + (uint32_t)((i * 16 + 8) * 8 + b * 2)));
            }
#pragma unroll
            for (int j = 0; j < NJ; ++j) {                    // weight rows 8 j + g (fragment), outputs 8 j + 2 t and + 1
                if (Q5) {
                    const uint32_t w = lds_u32(sB + (uint32_t)(j * 8 * QM_ROW5 + b * 16)), f = lds_u32(sF + (uint32_t)(j * 8 * 16 + b * 4));
                    bf[j][0] = q5_bytes(w & 0x0F0F0F0Fu, f >> (4 * t));
                    bf[j][1] = q5_bytes((w >> 4) & 0x0F0F0F0Fu, f >> (16 + 4 * t));
                } else {
                    const uint32_t p = sB + (uint32_t)(j * 8 * QM_ROW + b * 32);
                    bf[j][0] = lds_u32(p);
                    bf[j][1] = lds_u32(p + 16);
                }
                db[j][0] = half_bits_to_float(lds_u16(sDB + (uint32_t)(j * 8 * 8 + b * 2)));
                db[j][1] = half_bits_to_float(lds_u16(sDB + (uint32_t)((j * 8 + 1) * 8 + b * 2)));
            }
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    int s[4] = {0, 0, 0, 0};
                    mma_s8(s, af[i], bf[j]);
                    // sumf += (float)sumi * (d_w * d_x), the reference's operations in the reference's order
                    acc[i][j][0] = __fadd_rn(acc[i][j][0], __fmul_rn((float)s[0], __fmul_rn(db[j][0], da[i][0])));
                    acc[i][j][1] = __fadd_rn(acc[i][j][1], __fmul_rn((float)s[1], __fmul_rn(db[j][1], da[i][0])));
                    acc[i][j][2] = __fadd_rn(acc[i][j][2], __fmul_rn((float)s[2], __fmul_rn(db[j][0], da[i][1])));
                    acc[i][j][3] = __fadd_rn(acc[i][j][3], __fmul_rn((float)s[3], __fmul_rn(db[j][1], da[i][1])));
                }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int col = n0 + wn * (TILE / 4) + j * 8 + 2 * t;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = m0 + wm * (TILE / 2) + i * 16 + g + 8 * h;
                if (row < M) {
                    if (col < N) C[(size_t)row * ldc + col] = acc[i][j][2 * h] + (bias ? bias[col] : 0.0f);
                    if (col + 1 < N) C[(size_t)row * ldc + col + 1] = acc[i][j][2 * h + 1] + (bias ? bias[col + 1] : 0.0f);
                }
            }
        }
}

template <bool Q5, int TILE>
static int qm_launch(const void *A, const void *B, const float *bias, float *C, int ldc, int M, int N, int nb, int weights_ready, cudaStream_t st)
{
    auto kernel = gemm_q80_mma_kernel<Q5, TILE>;
    constexpr int smem = QmTile<Q5, TILE>::SMEM;
    static int attr_set = 0;
    if (!attr_set) {
        if (ckb_check_cuda((int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "gemm_q80_mma smem attr")) return CKB_ERR_CUDA;
        attr_set = 1;
    }
    return launch_pdl("gemm_q80_mma", kernel, dim3((N + TILE - 1) / TILE, (M + TILE - 1) / TILE), dim3(QM_THREADS), (size_t)smem, st, (const uint8_t *)A, (const uint8_t *)B, bias,
                      C, ldc, M, N, nb, weights_ready);
}

template <bool Q5>
static int qm_pick(const void *A, const void *B, const float *bias, float *C, int ldc, int M, int N, int K, int weights_ready, void *stream)
{
    if (K % (32 * QM_KB) || M <= 0 || N <= 0 || (((uintptr_t)A | (uintptr_t)B) & 15)) return -1;
    // Rounds of wide tiles, one on an SM, against rounds of narrow ones, two on an SM, each of which takes 0.6 of a wide one's time (K of 4096: 61 against 103 us; of 896:
    // 15 against 21).  9728 x 896 at 256 tokens is 152 wide tiles: two rounds, 43 us, narrow 33; at 130 tokens 38 and 26; 4096 x 4096 at 512 tokens 104 and 119.
    const long sms = ckb_sm_count(), wide = (long)((N + 127) / 128) * ((M + 127) / 128), narrow = (long)((N + 63) / 64) * ((M + 63) / 64);
    int tile = ckb_tune_get("gemm_q80_tile", 0);
    if (tile != 64 && tile != 128) tile = 10 * ((wide + sms - 1) / sms) < 6 * ((narrow + 2 * sms - 1) / (2 * sms)) ? 128 : 64;
    cudaStream_t st = ckb_stream(stream);
    return tile == 128 ? qm_launch<Q5, 128>(A, B, bias, C, ldc, M, N, K / 32, weights_ready, st) : qm_launch<Q5, 64>(A, B, bias, C, ldc, M, N, K / 32, weights_ready, st);
}

}  // namespace ckb

using namespace ckb;

// A_planar [M rows], B_planar [N rows]: row-planar Q8_0 (ckb200_dev_q8_0_to_planar), or for q50 the weights row-planar Q5_0 (ckb200_dev_q5_0_to_planar);
// rows of C are ldc floats apart; weights_ready: no kernel of this stream wrote B lately (it is read ahead of the dependency wait).  Returns -1 when the shape is not handled (K not a multiple of 128).
extern "C" int ckb_launch_gemm_q80_mma(const void *A_planar, const void *B_planar, const float *bias, float *C, int ldc, int M, int N, int K, int weights_ready, void *stream)
{
    return qm_pick<false>(A_planar, B_planar, bias, C, ldc, M, N, K, weights_ready, stream);
}
extern "C" int ckb_launch_gemm_q50_mma(const void *A_planar, const void *B_planar, const float *bias, float *C, int ldc, int M, int N, int K, int weights_ready, void *stream)
{
    return qm_pick<true>(A_planar, B_planar, bias, C, ldc, M, N, K, weights_ready, stream);
}
