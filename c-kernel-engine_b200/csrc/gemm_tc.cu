// Prefill / batched-decode GEMM on the 5th-generation tensor cores: C[M,N] = A_q8[M,K] . W[N,K]^T (+ bias), M >= 16,
// for Q4_K weights (the reference's block_q4_K rows) and Q6_K weights (row-planar layout, gemv_q6k_planar.cu).
// Replaces gemm_nt_q4_k_q8_k (src/kernels/gemm_kernels_q4k_q8k.c:301-326) and gemm_nt_q6_k_q8_k
// (src/kernels/gemm_kernels_q6k_q8k.c:1243-1268), which the reference computes as one GEMV per token.
//
// Exact-integer formulation.  For one 256-element Q4_K superblock b the reference adds
//     d_x[m,b] * ( d[n,b] * sum_j sc[n,j] * S[m,n,j]  -  dmin[n,b] * sum_j mn[n,j] * bsum[m,j] )
// where S are int32 sub-block dots (gemm_kernels_q4k_q8k.c:144-173).  Here
//     T [n,m] = sum_k (sc[n,k/32] * q4[n,k]) * q8[m,k]        256-deep f16 MMA, every operand an exact integer
//     T2[n,m] = sum_i  mn[n,i/2]  * bsum16[m,i]               16-deep f16 MMA (one k-step)
// are accumulated in fp32 in tensor memory (integers below 2^24 stay exact), read back with tcgen05.ld once per
// superblock and combined with the fp32 scales in registers: acc += d_x * (d * T - dmin * T2).
// Q6_K: A = (q6 - 32) * sc (src/kernels/gemm_kernels_q6k_q8k.c:86-116), the offset is inside the operand, so there
// is no T2.  The product is an exact fp16 integer whenever |q6 - 32| * |sc| <= 2048, always for |sc| <= 64.  Above that fp16 holds the even integers
// only: the operand is the nearest of them, and what it lacks (-1, 0 or 1) is an operand of its own, multiplied into the same accumulator.  Files made by a
// quantiser that scales a superblock to its largest sub-scale have such scales in every superblock; whether there are rests is found per stage and 32 rows
// (4096 x 14336 at 512 tokens: 110 us without, 125 with; 108 when the products stayed rounded, 1.3e-4 off).
//
// Two kernels:
//  * gemm_x_tiles_kernel expands the Q8_K activations once into fp16 operand tiles in the exact shared-memory
//    layout of the MMA (K-major, no swizzle, 8 x 16-byte core matrices), one contiguous blob per (token tile,
//    superblock), so the GEMM fetches them with plain 1-D bulk copies.
//  * gemm_kq_tc_kernel<WF, NT>: one CTA owns 128 weight rows (the M = 128 operand, one TMEM lane each) and one tile of NT tokens
//    (the N operand, TMEM columns; fewer tokens are zero-padded).  Warp-specialised:
//        warp 0       loader of activations: bulk copies of 128-deep stages, of the bsum tile and of the block scales of each superblock
//        warp 1       issuer: tcgen05.mma from one elected lane; tcgen05.commit frees stages and publishes accumulators
//        warp 2       Q4_K: the 16-deep tile of mins and the (d, dmin) pairs of a superblock
//        warp 3       loader of weights: the raw superblocks of all 128 rows, one tiled bulk copy each (Q6_K: one per plane)
//        warps 4-11   two expander sets, thread = row: raw bytes -> fp16 operand, alternate 64-deep k-stages
//        warps 12-    drain: tcgen05.ld of T and T2, fp32 sums in registers
//    Every wait is bounded; a timeout sets the device error word, the CTA drains, frees TMEM and returns.
//
// What bounds it, and why it is split like this.  The MMAs of a superblock take 17 x 64 cycles at NT = 128.  With the expanded weights in
// shared memory the data pipe alone would need about 3700 (uncoalesced weight loads 1536 tag cycles, operand tile written 512 and read
// 512, activations written 512 and read 512), and the kernel took 5100.  So the expanded weights never touch shared memory: an expander
// thread owns a row, a row is a TMEM lane, and tcgen05.st puts its 64 halves where the MMA reads its A operand.  Nor is a proxy
// fence needed between the two.  The raw weights come as 144-byte rows by tiled copies (coalesced, and conflict-free to read at that pitch).
// A nibble becomes a half with one AND-OR (0x6400 | n = 1024 + n, or 1024 + 16 n for the upper one) and one fused multiply-add; the halves of a
// register are then elements 0, 2 and 1, 3 of a 4-byte word, and the activation tiles are written in that order: k is a summation index.
// The 512 TMEM columns at NT = 128: two T buffers (256), one T2 (128), four weight stages (128).
// A superblock now takes about 1960 cycles: issuer, expanders and drain are each busy for 1500 of them and share four schedulers.
// Measured (28672 x 4096 Q4_K at 512 / 2048 tokens): 142 / 512 us = 847 / 940 TFLOP/s, with the operand through shared memory 268 / 1055 us; 4096 x 14336 Q6_K
// at 512 tokens 110 us (181 before); 333 tokens of 28672 x 4096: 126 us against 205 with activations quantised.
#include <cuda.h>

#include "q8k_block.cuh"
#include "quant_units.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "runtime.h"
#include "tcgen05.cuh"

namespace ckb {

constexpr int TC_ROWS = 128;                          // rows of the weight operand per MMA
constexpr int TC_AUX = TC_ROWS * 32;                  // 16-deep tile of the mins: 4 KB
constexpr int TC_ASLOTS = 4, TC_BSLOTS = 4, TC_RSLOTS = 3, TC_XSLOTS = 4;   // rings: 64-deep weight stages in TMEM, 128-deep activation stages, raw
                                                                          // superblocks, per-superblock extras (mins, bsums, scales)
enum { TC_W_Q4K = 0, TC_W_Q6K_PLANAR = 1 };           // weight operand formats

// Activation blob of one (tile of NT tokens, superblock): four 64-deep k-stages, the 16-deep bsum tile, NT block scales.
template <int NT>
struct TcTile {
    static constexpr int CHUNK = NT * 16;                     // one 8-element k-chunk of NT tokens
    static constexpr int STAGE = 8 * CHUNK;                   // 64-deep
    static constexpr int AUX = 2 * CHUNK;
    static constexpr int XBLOB_B2 = 4 * STAGE, XBLOB_DX = XBLOB_B2 + AUX, XBLOB = XBLOB_DX + NT * 4;   // a multiple of 16
    static_assert(XBLOB == q8k_tile_bytes(NT), "the layout that quantize_block_q8k_tile writes");
};

// Everything that depends on the width NT of the token tile and on the weight format.  NT = 32: the accumulators and the staging shrink so far that
// two CTAs share an SM and each covers the other's latencies.
template <int WF, int NT>
struct TcCfg : TcTile<NT> {
    static constexpr bool Q4 = WF == TC_W_Q4K;
    // raw superblocks of 128 rows: 144-byte rows, or the planes ql | qh | scales (1024-byte aligned: they are written swizzled)
    static constexpr int RAW_QH = TC_ROWS * 128, RAW_SC = RAW_QH + TC_ROWS * 64, RAW = Q4 ? TC_ROWS * Q4K_BYTES : RAW_SC + TC_ROWS * 16;
    static constexpr int OFF_RAW = 0;
    static constexpr int OFF_B = OFF_RAW + TC_RSLOTS * RAW;
    static constexpr int OFF_A2 = OFF_B + TC_BSLOTS * 2 * TcTile<NT>::STAGE;
    static constexpr int OFF_B2 = OFF_A2 + (Q4 ? TC_XSLOTS * TC_AUX : 0);
    static constexpr int OFF_DX = OFF_B2 + (Q4 ? TC_XSLOTS * TcTile<NT>::AUX : 0);
    static constexpr int OFF_DD = OFF_DX + TC_XSLOTS * NT * 4;                     // fp16 d | dmin of the rows
    static constexpr int OFF_BAR = OFF_DD + (Q4 ? TC_XSLOTS * TC_ROWS * 4 : 0);
    static constexpr int A_FULL = 0, A_EMPTY = A_FULL + TC_ASLOTS, B_FULL = A_EMPTY + TC_ASLOTS, B_EMPTY = B_FULL + TC_BSLOTS, R_FULL = B_EMPTY + TC_BSLOTS,
                         R_EMPTY = R_FULL + TC_RSLOTS, X_FULL = R_EMPTY + TC_RSLOTS, X_EMPTY = X_FULL + TC_XSLOTS, T_FULL = X_EMPTY + TC_XSLOTS, T_EMPTY = T_FULL + 2,
                         T2_EMPTY = T_EMPTY + 2, DONE = T2_EMPTY + 1, BARS = DONE + 1;
    static constexpr int OFF_WIDE = OFF_BAR + BARS * 8 + 16;                       // Q6_K: a byte per (weight stage, lane quarter): there are rests
    static constexpr int SMEM = OFF_WIDE + 4 * TC_ASLOTS;
    static constexpr int DRAIN_WARPS = NT > 32 ? 8 : 4;       // 4 TMEM lane quarters x column halves
    static constexpr int DRAIN_COLS = NT / (DRAIN_WARPS / 4); // token columns per drain thread
    static constexpr int THREADS = (12 + DRAIN_WARPS) * 32, CTAS_PER_SM = NT > 32 ? 1 : 2;
    // Register counts per role after setmaxnreg.  setmaxnreg.inc blocks until the CTA's own pool (threads x registers
    // at launch) can supply the registers, so 128 * CTL + 256 * EXP + 32 * DRAIN_WARPS * DRAIN must not exceed
    // THREADS * LAUNCH; the launcher checks the compiled register count against LAUNCH before the first launch.
    static constexpr int REGS_LAUNCH = NT > 32 ? 96 : 64, REGS_CTL = 48, REGS_EXP = 72, REGS_DRAIN = NT > 32 ? 144 : 64;
    static_assert(128 * REGS_CTL + 256 * REGS_EXP + 32 * DRAIN_WARPS * REGS_DRAIN <= THREADS * REGS_LAUNCH, "setmaxnreg targets exceed the CTA's register pool");
    static_assert(THREADS * REGS_LAUNCH * CTAS_PER_SM <= 65536, "register plan");
    // T buffer u at column u * NT.  Q6_K has no T2; what its stages lack goes behind them, a slot per stage or (two CTAs on an SM) per expander set.
    static constexpr uint32_t TM_T2 = 2 * NT, TM_A = (Q4 ? 3 : 2) * NT, TM_R = TM_A + 32 * TC_ASLOTS, TMEM_COLS = NT > 32 ? 512 : 256;
    static constexpr uint32_t RESTS = Q4 ? 0 : (NT > 32 ? TC_ASLOTS : 2);
    static_assert(TM_R + 32 * RESTS <= TMEM_COLS && CTAS_PER_SM * TMEM_COLS <= 512, "tensor memory plan");
    // instruction descriptor: f16 x f16 -> f32, both operands K-major, M = 128, N = NT
    static constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(TC_ROWS >> 4) << 24);
    static_assert(NT % 32 == 0 && NT <= 128 && RAW % (Q4 ? 16 : 1024) == 0 && OFF_BAR % 8 == 0 && OFF_B % 128 == 0, "layout");
    static_assert(CTAS_PER_SM * (SMEM + 1024) <= 228 * 1024 && SMEM <= 227 * 1024, "shared memory plan");
};

// shared-memory matrix descriptor: K-major, no swizzle; LBO = distance between the two 8-element k-chunks of
// one MMA (rows x 16 B), SBO = distance between 8-row groups (128 B); version 1 (Blackwell)
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t addr, uint32_t chunk_bytes)
{
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(chunk_bytes >> 4) << 16;
    d |= (uint64_t)(128 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
// (a & mask) | bits in one instruction
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits)
{
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(bits));
    return r;
}

// eight int8 -> 8 fp16, exact, in the order 0 2 1 3 4 6 5 7: (x ^ 0x80) is x + 128 as an unsigned byte; 0x6400 | that is 1152 + x
__device__ __forceinline__ uint4 s8_chunk_to_half(uint32_t w0, uint32_t w1)
{
    const __half2 off = __floats2half2_rn(1152.0f, 1152.0f);
    const uint32_t u0 = w0 ^ 0x80808080u, u1 = w1 ^ 0x80808080u;
    return make_uint4(h2_bits(__hsub2(bits_h2(and_or(u0, 0x00FF00FFu, 0x64006400u)), off)), h2_bits(__hsub2(bits_h2(and_or(u0 >> 8, 0x00FF00FFu, 0x64006400u)), off)),
                      h2_bits(__hsub2(bits_h2(and_or(u1, 0x00FF00FFu, 0x64006400u)), off)), h2_bits(__hsub2(bits_h2(and_or(u1 >> 8, 0x00FF00FFu, 0x64006400u)), off)));
}

template <int NT>
__device__ __forceinline__ uint32_t tc_xtile_offset(int tok, int kchunk) { return (uint32_t)(kchunk * TcTile<NT>::CHUNK + (tok >> 3) * 128 + (tok & 7) * 16); }

// A operand in tensor memory (one lane per row, two k per column)
__device__ __forceinline__ void tc_mma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u));
}
// 32 columns of this warp's 32 lanes
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tc_tma(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

// two fp32 at a time (Blackwell's packed fp32 instructions: half the issue slots)
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi)); return r; }
__device__ __forceinline__ uint64_t pack2f(float lo, float hi) { return pack2(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }

// The 64 weights of one row in k-stage s of a Q4_K superblock (sub-blocks 2s and 2s + 1: 32 nibble bytes) times their 6-bit scales:
// (1024 + n) * sc - 1024 * sc and (1024 + 16 n) * sc / 16 - 64 * sc, exact: only the result (at most 945) is rounded
__device__ __forceinline__ void q4k_expand(const uint4 &hdr, const uint4 &qa, const uint4 &qb, int s, uint32_t (&o)[32])
{
    uint32_t sc2, m2;
    q4k_scales(hdr.y, hdr.z, hdr.w, s, sc2, m2);
    const __half2 k1024 = __floats2half2_rn(1024.0f, 1024.0f);
    const __half2 s_lo = __hsub2(bits_h2(__byte_perm(sc2, 0x64646464u, 0x4040)), k1024), s_hi = __hsub2(bits_h2(__byte_perm(sc2, 0x64646464u, 0x4141)), k1024);
    const __half2 b_lo = __hmul2(s_lo, __floats2half2_rn(-1024.0f, -1024.0f)), b_hi = __hmul2(s_hi, __floats2half2_rn(-64.0f, -64.0f));
    const __half2 s_hi16 = __hmul2(s_hi, __floats2half2_rn(0.0625f, 0.0625f));
    const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t v = w[i], v8 = v >> 8;
        o[2 * i] = h2_bits(__hfma2(bits_h2(and_or(v, 0x000F000Fu, 0x64006400u)), s_lo, b_lo));
        o[2 * i + 1] = h2_bits(__hfma2(bits_h2(and_or(v8, 0x000F000Fu, 0x64006400u)), s_lo, b_lo));
        o[16 + 2 * i] = h2_bits(__hfma2(bits_h2(and_or(v, 0x00F000F0u, 0x64006400u)), s_hi16, b_hi));
        o[16 + 2 * i + 1] = h2_bits(__hfma2(bits_h2(and_or(v8, 0x00F000F0u, 0x64006400u)), s_hi16, b_hi));
    }
}

// The same for Q6_K: k-stage 2 n + hi holds weights 128 n + 64 hi .. + 63: nibbles `hi` of the 64 ql bytes of half n, 2-bit planes 2 hi and
// 2 hi + 1 of its 32 qh bytes, scales 8 n + 4 hi .. + 3.  raw: the row's planes as the swizzled copies left them.
__device__ __forceinline__ void q6k_expand(const uint8_t *raw_ql, const uint8_t *raw_qh, uint32_t scw, int row, int n, int hi, uint32_t (&o)[32])
{
    const __half2 c66 = __floats2half2_rn(66.0f, 66.0f);
    uint32_t qhw[8];
#pragma unroll
    for (int j = 0; j < 2; ++j) {            // 64-byte swizzle: 16-byte pieces permuted by bits 1-2 of the row
        const uint4 v = *reinterpret_cast<const uint4 *>(raw_qh + row * 64 + (((2 * n + j) ^ ((row >> 1) & 3)) << 4));
        qhw[4 * j] = v.x >> (4 * hi); qhw[4 * j + 1] = v.y >> (4 * hi); qhw[4 * j + 2] = v.z >> (4 * hi); qhw[4 * j + 3] = v.w >> (4 * hi);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {            // 128-byte swizzle: 16-byte pieces permuted by the row's low three bits
        const uint4 v = *reinterpret_cast<const uint4 *>(raw_ql + row * 128 + (((4 * n + j) ^ (row & 7)) << 4));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        const float scf = 16.0f * (float)(int)(int8_t)((scw >> (8 * j)) & 255u);      // 16 weights per scale = one 16-byte piece
        const __half2 sc2 = __floats2half2_rn(scf, scf);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t nib = (w[i] >> (4 * hi)) & 0x0F0F0F0Fu, h = qhw[4 * (j & 1) + i];
            const uint32_t q = nib | ((j < 2 ? h << 4 : h << 2) & 0x30303030u);
            // 0x5400 | q is the fp16 bit pattern of 64 + q / 16: (q - 32) / 16 * 16 sc
            o[8 * j + 2 * i] = h2_bits(__hmul2(__hsub2(bits_h2(and_or(q, 0x00FF00FFu, 0x54005400u)), c66), sc2));
            o[8 * j + 2 * i + 1] = h2_bits(__hmul2(__hsub2(bits_h2(and_or(q >> 8, 0x00FF00FFu, 0x54005400u)), c66), sc2));
        }
    }
}
// Half a stage (16-byte pieces 2 P and 2 P + 1) as the rounded products and what they lack, which one fused multiply-add gives exactly
template <int P>
__device__ __forceinline__ void q6k_expand_rests(const uint8_t *raw_ql, const uint8_t *raw_qh, uint32_t scw, int row, int n, int hi, uint32_t (&o)[16], uint32_t (&t)[16])
{
    const __half2 c66 = __floats2half2_rn(66.0f, 66.0f);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const uint4 g = *reinterpret_cast<const uint4 *>(raw_qh + row * 64 + (((2 * n + j) ^ ((row >> 1) & 3)) << 4));
        const uint4 v = *reinterpret_cast<const uint4 *>(raw_ql + row * 128 + (((4 * n + 2 * P + j) ^ (row & 7)) << 4));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w}, qh[4] = {g.x, g.y, g.z, g.w};
        const float scf = 16.0f * (float)(int)(int8_t)((scw >> (8 * (2 * P + j))) & 255u);
        const __half2 sc2 = __floats2half2_rn(scf, scf);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t h = qh[i] >> (4 * hi), q = ((w[i] >> (4 * hi)) & 0x0F0F0F0Fu) | ((P == 0 ? h << 4 : h << 2) & 0x30303030u);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const __half2 a = __hsub2(bits_h2(and_or(e ? q >> 8 : q, 0x00FF00FFu, 0x54005400u)), c66), p = __hmul2(a, sc2);
                o[8 * j + 2 * i + e] = h2_bits(p);
                t[8 * j + 2 * i + e] = h2_bits(__hfma2(a, sc2, __hneg2(p)));
            }
        }
    }
}
// whether one of four scales is outside [-64, 63]
__device__ __forceinline__ bool q6k_wide(uint32_t scw) { return ((((scw & 0x7F7F7F7Fu) + 0x40404040u) ^ scw) & 0x80808080u) != 0; }

// ---------------------------------------------------------------- activation tiles

// grid (superblocks, token tiles, parts of the 32 k-chunks).  The quants of a token's block are read as they lie (consecutive
// threads, consecutive words) into shared memory and leave it token-major: consecutive threads take consecutive tokens of one
// k-chunk, so every warp writes 512 contiguous bytes of the blob.  (Reading token-major straight from global memory fetched a
// 32-byte sector per 8 bytes used and took 12 us for 512 tokens of 4096 elements.)
template <int NT>
__global__ void __launch_bounds__(256) gemm_x_tiles_kernel(const uint8_t *__restrict__ A_q8, uint8_t *__restrict__ xt, int M, int nb)
{
    using Cfg = TcTile<NT>;
    constexpr int PITCH = 66;                                  // words per token in shared memory: 64 + 2, 8-byte reads two-way at worst
    __shared__ __align__(8) uint32_t q[NT * PITCH];
    const int b = blockIdx.x, mt = blockIdx.y;
    pdl_wait();
    pdl_trigger();                                             // the product reads weights ahead of its own wait: whatever re-laid them is complete by now
    const int kcz = 32 / (int)gridDim.z, kc0 = (int)blockIdx.z * kcz;     // this CTA's k-chunks [kc0, kc0 + kcz)
    uint8_t *blob = xt + ((size_t)mt * nb + b) * Cfg::XBLOB;
    for (int it = threadIdx.x; it < NT * kcz * 2; it += 256) {
        const int t = it / (2 * kcz), w = it - t * (2 * kcz), m = mt * NT + t;
        uint32_t v = 0;
        if (m < M) v = __ldcg(reinterpret_cast<const uint32_t *>(A_q8 + ((size_t)m * nb + b) * Q8K_BYTES) + 1 + 2 * kc0 + w);
        q[t * PITCH + w] = v;
    }
    __syncthreads();
    for (int it = threadIdx.x; it < NT * kcz; it += 256) {
        const int t = it % NT, kl = it / NT, kc = kc0 + kl;
        const uint2 w = *reinterpret_cast<const uint2 *>(&q[t * PITCH + 2 * kl]);
        *reinterpret_cast<uint4 *>(blob + (kc >> 3) * Cfg::STAGE + tc_xtile_offset<NT>(t, kc & 7)) = s8_chunk_to_half(w.x, w.y);
    }
    if (blockIdx.z != 0) return;
    if (threadIdx.x < 2 * NT) {
        const int t = threadIdx.x % NT, g = threadIdx.x / NT, m = mt * NT + t;    // bsums[8g .. 8g+7], |bsum| <= 2048: exact
        uint32_t o[4] = {0u, 0u, 0u, 0u};
        float d = 0.0f;
        if (m < M) {
            const uint32_t *blk = reinterpret_cast<const uint32_t *>(A_q8 + ((size_t)m * nb + b) * Q8K_BYTES);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t v = __ldcg(blk + 65 + 4 * g + c);
                const __half2 h = __floats2half2_rn((float)(short)(v & 0xffffu), (float)(short)(v >> 16));
                o[c] = *reinterpret_cast<const uint32_t *>(&h);
            }
            d = __uint_as_float(__ldcg(blk));
        }
        *reinterpret_cast<uint4 *>(blob + Cfg::XBLOB_B2 + tc_xtile_offset<NT>(t, g)) = make_uint4(o[0], o[1], o[2], o[3]);
        if (g == 0) reinterpret_cast<float *>(blob + Cfg::XBLOB_DX)[t] = d;
    }
}

// ---------------------------------------------------------------- GEMM

template <uint32_t V> struct TcConst { static constexpr uint32_t value = V; };
struct TcMaps { CUtensorMap w[3]; };                  // Q4_K: rows; Q6_K: planes ql, qh, scales

// Work of a launch: units of (K slice, row tile, token tile), token tiles innermost, dealt round-robin to persistent CTAs.  A slice z takes the superblocks
// [z * nbz, z * nbz + nbz) and writes its partial sums to C + z * cz (the launcher adds the slices up in a fixed order); a single slice writes C
// itself, bias included.  Only the loaders and the drain know where a unit ends; the other roles see one run of superblocks, so that the next unit's
// weights are expanded and multiplied while the last one's sums are stored (a CTA per unit spent 6 us of 23 starting and storing).
struct TcWork {
    int units, mtiles, ntiles, nb_row, nbz;
    __device__ __forceinline__ int mt(int u) const { return u % mtiles; }
    __device__ __forceinline__ int nt(int u) const { return u / mtiles % ntiles; }
    __device__ __forceinline__ int z(int u) const { return u / mtiles / ntiles; }
    __device__ __forceinline__ int kb0(int u) const { return z(u) * nbz; }
    __device__ __forceinline__ int nb(int u) const { return min(nbz, nb_row - kb0(u)); }
};

template <int WF, int NT>
__global__ void __launch_bounds__(TcCfg<WF, NT>::THREADS, TcCfg<WF, NT>::CTAS_PER_SM)
gemm_kq_tc_kernel(const __grid_constant__ TcMaps maps, const TcWork work, const uint8_t *__restrict__ xt, const uint8_t *__restrict__ B, const float *__restrict__ bias,
                  float *__restrict__ C, int ldc, size_t cz, int M, int N, int *__restrict__ dev_err)
{
    using Cfg = TcCfg<WF, NT>;
    constexpr bool Q4 = Cfg::Q4;
    uint32_t total = 0;                               // superblocks of all this CTA's units
    for (int u = blockIdx.x; u < work.units; u += gridDim.x) total += (uint32_t)work.nb(u);
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t s_base = smem_u32(smem), s_bar = s_base + Cfg::OFF_BAR;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + Cfg::OFF_BAR + Cfg::BARS * 8);
#define BAR(i) (s_bar + 8u * (uint32_t)(i))

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid == 0) {
        for (int i = 0; i < TC_ASLOTS; ++i) { mbar_init(BAR(Cfg::A_FULL + i), 4); mbar_init(BAR(Cfg::A_EMPTY + i), 1); }
        for (int i = 0; i < TC_BSLOTS; ++i) { mbar_init(BAR(Cfg::B_FULL + i), 1); mbar_init(BAR(Cfg::B_EMPTY + i), 1); }
        for (int i = 0; i < TC_RSLOTS; ++i) { mbar_init(BAR(Cfg::R_FULL + i), 1); mbar_init(BAR(Cfg::R_EMPTY + i), Q4 ? 9 : 8); }     // expander warps and warp 2
        for (int i = 0; i < TC_XSLOTS; ++i) {
            mbar_init(BAR(Cfg::X_FULL + i), Q4 ? 2 : 1);                            // loader (and its bytes), warp 2
            mbar_init(BAR(Cfg::X_EMPTY + i), Cfg::DRAIN_WARPS + (Q4 ? 1 : 0));      // drain, T2's MMA
        }
        for (int i = 0; i < 2; ++i) { mbar_init(BAR(Cfg::T_FULL + i), 1); mbar_init(BAR(Cfg::T_EMPTY + i), Cfg::DRAIN_WARPS); }
        mbar_init(BAR(Cfg::T2_EMPTY), Cfg::DRAIN_WARPS);
        mbar_init(BAR(Cfg::DONE), 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(Cfg::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();

#define TC_SETMAXNREG(op, n) asm volatile("setmaxnreg." op ".sync.aligned.u32 %0;" ::"n"(n))
#define TC_WAIT(bar, parity, code)                                        \
    if (!mbar_wait_spin(bar, parity)) { atomicExch(dev_err, code); break; }

    if (warp < 4) {
        TC_SETMAXNREG("dec", Cfg::REGS_CTL);
        if (warp == 0) {
            // ------------------------------------------------------------ activations
            pdl_wait();                                // the tiles are what the kernel before this one writes; weights are nobody's output
            uint32_t g = 0, issued = 0, extras = 0;
            bool go = true;
            for (int u = blockIdx.x; u < work.units && go; u += gridDim.x) {
                const uint8_t *blob = xt + ((size_t)work.mt(u) * work.nb_row + work.kb0(u)) * Cfg::XBLOB;
                for (int nb = work.nb(u); nb > 0 && go; --nb, ++g, blob += Cfg::XBLOB) {
                    const uint32_t x = g % TC_XSLOTS;
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) {
                        const uint32_t i = 2 * (g & 1u) + h;
                        if (!mbar_wait_spin(BAR(Cfg::B_EMPTY + i), ((g >> 1) & 1u) ^ 1u)) { go = false; break; }
                        if (tc_elect_one()) {
                            mbar_arrive_expect_tx(BAR(Cfg::B_FULL + i), 2 * Cfg::STAGE);
                            bulk_g2s(s_base + Cfg::OFF_B + i * 2 * Cfg::STAGE, blob + h * 2 * Cfg::STAGE, 2 * Cfg::STAGE, BAR(Cfg::B_FULL + i));
                        }
                        ++issued;
                    }
                    if (!go || !mbar_wait_spin(BAR(Cfg::X_EMPTY + x), ((g / TC_XSLOTS) & 1u) ^ 1u)) { go = false; break; }
                    if (tc_elect_one()) {
                        mbar_arrive_expect_tx(BAR(Cfg::X_FULL + x), NT * 4 + (Q4 ? Cfg::AUX : 0));
                        bulk_g2s(s_base + Cfg::OFF_DX + x * NT * 4, blob + Cfg::XBLOB_DX, NT * 4, BAR(Cfg::X_FULL + x));
                        if (Q4) bulk_g2s(s_base + Cfg::OFF_B2 + x * Cfg::AUX, blob + Cfg::XBLOB_B2, Cfg::AUX, BAR(Cfg::X_FULL + x));
                    }
                    ++extras;
                }
            }
            if (!go) atomicExch(dev_err, DEV_ERR_EMPTY_WAIT);
            // copies still in flight land before the CTA's shared memory goes away, whatever became of the roles that wait for them
            for (uint32_t j = issued > TC_BSLOTS ? issued - TC_BSLOTS : 0; j < issued; ++j) mbar_wait_spin(BAR(Cfg::B_FULL + j % TC_BSLOTS), (j / TC_BSLOTS) & 1u);
            for (uint32_t b = extras > TC_XSLOTS ? extras - TC_XSLOTS : 0; b < extras; ++b) mbar_wait_spin(BAR(Cfg::X_FULL + b % TC_XSLOTS), (b / TC_XSLOTS) & 1u);
        } else if (warp == 1) {
            // ------------------------------------------------------------ issuer: the warp runs the loop and the waits uniformly, one lane issues.  This
            // warp is a chain of short dependent steps, and the MMAs of a 64-deep stage take 256 cycles: two superblocks are unrolled so that
            // slots, descriptors and most parities are constants (with them computed in a loop of stages the chain took 900 cycles a stage).
            const uint64_t dB = tc_smem_desc(s_base + Cfg::OFF_B, Cfg::CHUNK), dA2 = tc_smem_desc(s_base + Cfg::OFF_A2, TC_ROWS * 16), dB2 = tc_smem_desc(s_base + Cfg::OFF_B2, Cfg::CHUNK);
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const bool leader = tc_elect_one();
            auto superblock = [&](auto odd, uint32_t b) -> bool {
                constexpr uint32_t u = decltype(odd)::value;
                const uint32_t p = (b >> 1) & 1u, x [[maybe_unused]] = b % TC_XSLOTS;
                if (!mbar_wait_spin(BAR(Cfg::T_EMPTY + u), p ^ 1u)) return false;
#pragma unroll
                for (uint32_t s = 0; s < 4; ++s) {
                    constexpr uint32_t half = Cfg::STAGE >> 4;
                    const uint32_t i = 2 * u + (s >> 1);
                    if (!(s & 1u) && !mbar_wait_spin(BAR(Cfg::B_FULL + i), p)) return false;
                    if (!mbar_wait_spin(BAR(Cfg::A_FULL + s), u)) return false;
                    tc_fence_after();                  // the expanders' stores, and (s = 0) the drain's loads of this accumulator, come before these MMAs
                    if (leader) {
                        uint32_t wide = 0;
                        if constexpr (!Q4) wide = *reinterpret_cast<const volatile uint32_t *>(smem + Cfg::OFF_WIDE + 4 * s);
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k)
                            tc_mma_ta(tm + NT * u, tm + Cfg::TM_A + 32 * s + 8 * k, dB + (uint64_t)(half * (2 * i + (s & 1u)) + k * (2 * Cfg::CHUNK >> 4)), Cfg::IDESC, (s | k) ? 1u : 0u);
                        if constexpr (!Q4) {
                            if (wide) {
#pragma unroll
                                for (uint32_t k = 0; k < 4; ++k)
                                    tc_mma_ta(tm + NT * u, tm + Cfg::TM_R + 32 * (s % Cfg::RESTS) + 8 * k, dB + (uint64_t)(half * (2 * i + (s & 1u)) + k * (2 * Cfg::CHUNK >> 4)), Cfg::IDESC, 1u);
                            }
                        }
                        tc_commit(BAR(Cfg::A_EMPTY + s));
                        if (s & 1u) tc_commit(BAR(Cfg::B_EMPTY + i));
                    }
                    __syncwarp();
                }
                if constexpr (Q4) {
                    if (!mbar_wait_spin(BAR(Cfg::T2_EMPTY), u ^ 1u) || !mbar_wait_spin(BAR(Cfg::X_FULL + x), (b / TC_XSLOTS) & 1u)) return false;
                    tc_fence_after();
                }
                if (leader) {
                    if constexpr (Q4) {
                        tc_mma(tm + Cfg::TM_T2, dA2 + (uint64_t)(x * (TC_AUX >> 4)), dB2 + (uint64_t)(x * (Cfg::AUX >> 4)), Cfg::IDESC, 0u);
                        tc_commit(BAR(Cfg::X_EMPTY + x));
                    }
                    tc_commit(BAR(Cfg::T_FULL + u));
                }
                __syncwarp();
                return true;
            };
            for (uint32_t b = 0; b < total; b += 2)
                if (!superblock(TcConst<0>(), b) || (b + 1 < total && !superblock(TcConst<1>(), b + 1))) {
                    atomicExch(dev_err, DEV_ERR_MMA_WAIT);
                    break;
                }
            if (leader) tc_commit(BAR(Cfg::DONE));          // MMAs in flight finish before the tensor memory is freed
            mbar_wait_spin(BAR(Cfg::DONE), 0);
        } else if (warp == 2) {
            // ------------------------------------------------------------ Q4_K: mins (each doubled: bsums come per 16 elements) and block scales
            if constexpr (Q4) {
                for (uint32_t b = 0; b < total; ++b) {
                    const uint32_t r = b % TC_RSLOTS, x = b % TC_XSLOTS;
                    TC_WAIT(BAR(Cfg::X_EMPTY + x), ((b / TC_XSLOTS) & 1u) ^ 1u, DEV_ERR_EMPTY_WAIT);
                    TC_WAIT(BAR(Cfg::R_FULL + r), (b / TC_RSLOTS) & 1u, DEV_ERR_FULL_WAIT);
#pragma unroll 1
                    for (int row = lane; row < TC_ROWS; row += 32) {
                        const uint4 hdr = *reinterpret_cast<const uint4 *>(smem + Cfg::OFF_RAW + r * Cfg::RAW + row * Q4K_BYTES);
                        const __half2 k1024 = __floats2half2_rn(1024.0f, 1024.0f);
                        uint32_t o[8];
#pragma unroll
                        for (int s = 0; s < 4; ++s) {
                            uint32_t sc2, m2;
                            q4k_scales(hdr.y, hdr.z, hdr.w, s, sc2, m2);
                            o[2 * s] = h2_bits(__hsub2(bits_h2(__byte_perm(m2, 0x64646464u, 0x4040)), k1024));
                            o[2 * s + 1] = h2_bits(__hsub2(bits_h2(__byte_perm(m2, 0x64646464u, 0x4141)), k1024));
                        }
                        uint8_t *a2 = smem + Cfg::OFF_A2 + x * TC_AUX + (row >> 3) * 128 + (row & 7) * 16;
                        *reinterpret_cast<uint4 *>(a2) = make_uint4(o[0], o[1], o[2], o[3]);
                        *reinterpret_cast<uint4 *>(a2 + TC_ROWS * 16) = make_uint4(o[4], o[5], o[6], o[7]);
                        *reinterpret_cast<uint32_t *>(smem + Cfg::OFF_DD + (x * TC_ROWS + row) * 4) = hdr.x;
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes -> visible to the tensor core
                    __threadfence_block();
                    __syncwarp();
                    if (lane == 0) { mbar_arrive(BAR(Cfg::X_FULL + x)); mbar_arrive(BAR(Cfg::R_EMPTY + r)); }
                }
            }
        } else {
            // ------------------------------------------------------------ raw weights
            uint32_t issued = 0, r = 0, ph = 1;
            bool go = true;
            for (int u = blockIdx.x; u < work.units && go; u += gridDim.x) {
                const int n0 = work.nt(u) * TC_ROWS, kb0 = work.kb0(u), end = kb0 + work.nb(u);
                for (int kb = kb0; kb < end; ++kb) {
                    if (!mbar_wait_spin(BAR(Cfg::R_EMPTY + r), ph)) { atomicExch(dev_err, DEV_ERR_EMPTY_WAIT); go = false; break; }
                    if (tc_elect_one()) {
                        const uint32_t dst = s_base + Cfg::OFF_RAW + r * Cfg::RAW;
                        mbar_arrive_expect_tx(BAR(Cfg::R_FULL + r), Cfg::RAW);
                        if constexpr (Q4) {
                            tc_tma(dst, &maps.w[0], kb * Q4K_BYTES, n0, BAR(Cfg::R_FULL + r));
                        } else {
                            tc_tma(dst, &maps.w[0], kb * 128, n0, BAR(Cfg::R_FULL + r));
                            tc_tma(dst + Cfg::RAW_QH, &maps.w[1], kb * 64, n0, BAR(Cfg::R_FULL + r));
                            tc_tma(dst + Cfg::RAW_SC, &maps.w[2], kb * 16, n0, BAR(Cfg::R_FULL + r));
                        }
                    }
                    ++issued;
                    if (++r == TC_RSLOTS) { r = 0; ph ^= 1u; }
                }
            }
            for (uint32_t b = issued > TC_RSLOTS ? issued - TC_RSLOTS : 0; b < issued; ++b) mbar_wait_spin(BAR(Cfg::R_FULL + b % TC_RSLOTS), (b / TC_RSLOTS) & 1u);
        }
    } else if (warp < 12) {
        // ------------------------------------------------------------ weight expanders: thread = row = TMEM lane; set e takes the k-stages e and e + 2
        if constexpr (Cfg::REGS_EXP < Cfg::REGS_LAUNCH) TC_SETMAXNREG("dec", Cfg::REGS_EXP);
        else TC_SETMAXNREG("inc", Cfg::REGS_EXP);
        const int set = (warp - 4) >> 2, row = tid & 127;
        const uint32_t ta = tmem + Cfg::TM_A + ((uint32_t)(row & 96) << 16);
        bool go = true;
        uint32_t rests [[maybe_unused]] = 3;       // Q6_K, bit per stage of the set: not known to be zeros in this warp's rows
        for (uint32_t b = 0; b < total && go; ++b) {
            const uint32_t r = b % TC_RSLOTS;
            const uint8_t *raw = smem + Cfg::OFF_RAW + r * Cfg::RAW;
            TC_WAIT(BAR(Cfg::R_FULL + r), (b / TC_RSLOTS) & 1u, DEV_ERR_FULL_WAIT);
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int s = 2 * h + set;
                if constexpr (Q4) {
                    uint32_t o[32];
                    const uint8_t *p = raw + row * Q4K_BYTES;
                    q4k_expand(*reinterpret_cast<const uint4 *>(p), *reinterpret_cast<const uint4 *>(p + 16 + 32 * s), *reinterpret_cast<const uint4 *>(p + 32 + 32 * s), s, o);
                    if (!mbar_wait_spin(BAR(Cfg::A_EMPTY + s), (b & 1u) ^ 1u)) { atomicExch(dev_err, DEV_ERR_EMPTY_WAIT); go = false; break; }
                    tc_fence_after();
                    tc_st32(ta + 32 * s, o);
                } else {
                    const uint2 sc8 = *reinterpret_cast<const uint2 *>(raw + Cfg::RAW_SC + row * 16 + 8 * h);
                    const uint32_t scw = set ? sc8.y : sc8.x;
                    const bool wide = __any_sync(0xffffffffu, q6k_wide(scw));
                    if (!wide && !rests) {
                        uint32_t o[32];
                        q6k_expand(raw, raw + Cfg::RAW_QH, scw, row, h, set, o);
                        if (!mbar_wait_spin(BAR(Cfg::A_EMPTY + s), (b & 1u) ^ 1u)) { atomicExch(dev_err, DEV_ERR_EMPTY_WAIT); go = false; break; }
                        tc_fence_after();
                        tc_st32(ta + 32 * s, o);
                    } else {
                        // The issuer multiplies a slot of rests when any warp of the set has some, so a warp without leaves zeros in its rows, once.
                        // A slot per stage is free when the stage is; a slot per set when the set's stage before this one has been multiplied.
                        const uint32_t tr = ta + Cfg::TM_R - Cfg::TM_A + 32 * (s % Cfg::RESTS);
                        uint32_t o[16], t[16];
                        q6k_expand_rests<0>(raw, raw + Cfg::RAW_QH, scw, row, h, set, o, t);
                        if (!mbar_wait_spin(BAR(Cfg::A_EMPTY + s), (b & 1u) ^ 1u) ||
                            (Cfg::RESTS < TC_ASLOTS && !mbar_wait_spin(BAR(Cfg::A_EMPTY + (s ^ 2)), (b & 1u) ^ (h ? 0u : 1u)))) { atomicExch(dev_err, DEV_ERR_EMPTY_WAIT); go = false; break; }
                        tc_fence_after();
                        tc_st16(ta + 32 * s, o);
                        tc_st16(tr, t);
                        q6k_expand_rests<1>(raw, raw + Cfg::RAW_QH, scw, row, h, set, o, t);
                        tc_st16(ta + 32 * s + 16, o);
                        tc_st16(tr + 16, t);
                        rests = wide ? rests | (1u << h) : rests & ~(1u << h);
                        if (lane == 0) *(volatile uint8_t *)(smem + Cfg::OFF_WIDE + 4 * s + (warp & 3)) = wide;
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(BAR(Cfg::A_FULL + s));
                    if (h) mbar_arrive(BAR(Cfg::R_EMPTY + r));       // every lane's reads of the superblock have gone into what it stored
                }
            }
        }
    } else {
        // ------------------------------------------------------------ accumulator drain: thread = TMEM lane (weight row), DRAIN_COLS token columns
        if constexpr (Cfg::REGS_DRAIN < Cfg::REGS_LAUNCH) TC_SETMAXNREG("dec", Cfg::REGS_DRAIN);
        else TC_SETMAXNREG("inc", Cfg::REGS_DRAIN);
        constexpr int COLS = Cfg::DRAIN_COLS;
        const int dw = warp - 12;
        const int q = dw & 3, ch = dw >> 2;           // warp % 4 is the TMEM lane quarter this warp may read (12 % 4 == 0)
        const int row = 32 * q + lane;
        const size_t rb6 = ((size_t)work.nb_row * Q6K_BYTES + 15) & ~(size_t)15;
        uint32_t b = 0;
        bool go = true;
        for (int u = blockIdx.x; u < work.units && go; u += gridDim.x) {
            const int n = work.nt(u) * TC_ROWS + row, m0 = work.mt(u) * NT, nb = work.nb(u);
            const uint8_t *d_plane = Q4 ? nullptr : B + (size_t)min(n, N - 1) * rb6 + (size_t)work.nb_row * 208 + (size_t)work.kb0(u) * 2;
            uint64_t acc[COLS / 2];
#pragma unroll
            for (int i = 0; i < COLS / 2; ++i) acc[i] = 0;
            uint32_t d_next = 0;
            if constexpr (!Q4) d_next = ldg_nc_u16(d_plane);
            for (int kb = 0; kb < nb; ++kb, ++b) {
                const uint32_t buf = b & 1u, x = b % TC_XSLOTS;
                uint32_t dd_bits = d_next;
                if constexpr (!Q4) { if (kb + 1 < nb) d_next = ldg_nc_u16(d_plane + 2 * (size_t)(kb + 1)); }
                if (!mbar_wait_spin(BAR(Cfg::X_FULL + x), (b / TC_XSLOTS) & 1u)) { go = false; break; }
                if constexpr (Q4) dd_bits = *reinterpret_cast<const uint32_t *>(smem + Cfg::OFF_DD + (x * TC_ROWS + row) * 4);
                const float2 dd = __half22float2(bits_h2(dd_bits));
                const uint64_t d2 = pack2f(dd.x, dd.x), m2 = pack2f(-dd.y, -dd.y);
                const uint32_t dx = s_base + Cfg::OFF_DX + (x * NT + COLS * ch) * 4;
                if (!mbar_wait_spin(BAR(Cfg::T_FULL + buf), (b >> 1) & 1u)) { go = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(COLS * ch);
#pragma unroll
                for (int c = 0; c < COLS / 16; ++c) {
                    uint32_t t1[16], t2[16];
                    tc_ld16(taddr + NT * buf + 16 * c, t1);
                    if constexpr (Q4) tc_ld16(taddr + Cfg::TM_T2 + 16 * c, t2);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c == COLS / 16 - 1) {             // the accumulators are in registers: the next superblocks may overwrite them
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(BAR(Cfg::T_EMPTY + buf));
                            if (Q4) mbar_arrive(BAR(Cfg::T2_EMPTY));
                        }
                    }
#pragma unroll
                    for (int i4 = 0; i4 < 4; ++i4) {
                        uint64_t dxp[2];
                        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(dxp[0]), "=l"(dxp[1]) : "r"(dx + 64 * c + 16 * i4));
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint64_t t = pack2(t1[4 * i4 + 2 * i], t1[4 * i4 + 2 * i + 1]);
                            uint64_t &a = acc[8 * c + 2 * i4 + i];
                            if constexpr (Q4) a = fma2(dxp[i], fma2(d2, t, mul2(m2, pack2(t2[4 * i4 + 2 * i], t2[4 * i4 + 2 * i + 1]))), a);
                            else a = fma2(mul2(dxp[i], d2), t, a);
                        }
                    }
                }
                // Every lane has read block scales from shared memory with plain loads, and lane 0's arrival below tells the loader that
                // the buffer may be overwritten (by a bulk copy, which neither the compiler nor the warp barrier knows about).  The fence
                // makes each lane's loads complete before the warp barrier, so that none of them can still be in flight when the copy
                // lands.  Without it a pipeline that is not starved elsewhere corrupts a few 4-token groups of a 32-row quarter per call.
                __threadfence_block();
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(Cfg::X_EMPTY + x));
            }
            if (go && n < N) {
                const float bv = bias && work.nbz == work.nb_row ? bias[n] : 0.0f;
                float *Cz = C + (size_t)work.z(u) * cz;
#pragma unroll
                for (int i = 0; i < COLS / 2; ++i) {
                    const int m = m0 + COLS * ch + 2 * i;
                    float lo, hi;
                    unpack2(acc[i], lo, hi);
                    if (m < M) Cz[(size_t)m * ldc + n] = lo + bv;
                    if (m + 1 < M) Cz[(size_t)(m + 1) * ldc + n] = hi + bv;
                }
            }
        }
        if (!go) atomicExch(dev_err, DEV_ERR_MMA_WAIT);
    }
#undef TC_WAIT
#undef TC_SETMAXNREG
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::TMEM_COLS));
#undef BAR
}

// sum of the split-K slices in slice order, plus bias: C[m * ldc + n] = sum_z part[z][m][n] + bias[n]
template <bool VEC>
__global__ void __launch_bounds__(256) gemm_splitk_sum_kernel(const float *__restrict__ part, int Z, const float *__restrict__ bias, float *__restrict__ C, int ldc,
                                                              int M, int N)
{
    const size_t mn = (size_t)M * N;
    if (VEC) {                                                 // N and ldc multiples of 4, C and bias 16-byte aligned: four outputs per thread
        for (size_t i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4; i < mn; i += (size_t)gridDim.x * 1024) {
            const int m = (int)(i / N), n = (int)(i - (size_t)m * N);
            float4 s = __ldcg(reinterpret_cast<const float4 *>(part + i));
            for (int z = 1; z < Z; ++z) {                      // slices in a fixed order
                const float4 v = __ldcg(reinterpret_cast<const float4 *>(part + (size_t)z * mn + i));
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
            if (bias) {
                const float4 b = *reinterpret_cast<const float4 *>(bias + n);
                s.x += b.x; s.y += b.y; s.z += b.z; s.w += b.w;
            } else {
                s.x += 0.0f; s.y += 0.0f; s.z += 0.0f; s.w += 0.0f;
            }
            *reinterpret_cast<float4 *>(C + (size_t)m * ldc + n) = s;
        }
        return;
    }
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < mn; i += (size_t)gridDim.x * 256) {
        const int m = (int)(i / N), n = (int)(i - (size_t)m * N);
        float s = __ldcg(part + i);
        for (int z = 1; z < Z; ++z) s += __ldcg(part + (size_t)z * mn + i);
        C[(size_t)m * ldc + n] = s + (bias ? bias[n] : 0.0f);
    }
}

}  // namespace ckb

using namespace ckb;

// How many K slices: enough CTAs to fill the resident slots (SMs x CTAs per SM) in whole waves.  Few tokens only (the
// partial sums cost Z * M * N * 4 bytes of traffic), slices of at least 4 superblocks, at most 16.
static int tc_pick_slices(int tiles, int nb, int slots)
{
    int best = 1;
    double best_eff = 0.0;
    for (int z = 1; z <= 16 && nb / z >= 4; ++z) {
        const long ctas = (long)tiles * z, waves = (ctas + slots - 1) / slots;
        const double eff = (double)ctas / (double)(waves * slots);
        if (eff > best_eff * 1.08) { best_eff = eff; best = z; }      // a larger Z must pay for its partial sums
    }
    return best;
}

// How a product is cut: K slices of nbz superblocks, and row tiles that go to a second launch with K split.
struct TcPlan { int mtiles, ntiles, Z, nbz, tail_nt, Zt, nbzt; double us; };
static TcPlan tc_plan(int wf, int width, int M, int N, int nb, int ctas_per_sm, bool may_tail)
{
    TcPlan p = {(M + width - 1) / width, (N + TC_ROWS - 1) / TC_ROWS, 1, nb, 0, 1, nb, 0.0};
    const int slots = ckb_sm_count() * ctas_per_sm, tiles = p.ntiles * p.mtiles;
    // K is split for a handful of tokens, and for any product whose tiles leave more than half of the SMs without a CTA (the k and
    // v projections of a prompt: 8 x 4 tiles)
    const int splitk = ckb_tune_get("gemm_tc_splitk", 1);
    if (splitk && (M <= 128 || (splitk != 2 && 2 * tiles <= slots))) p.Z = tc_pick_slices(tiles, nb, slots);
    const int forced = ckb_tune_get("gemm_tc_slices", 0);
    if (forced > 0 && forced <= nb) p.Z = forced;
    p.nbz = (nb + p.Z - 1) / p.Z;
    p.Z = (nb + p.nbz - 1) / p.nbz;                    // no empty slice
    // A grid of whole waves plus a few units pays a full wave for those few (28672 x 4096 at 512 tokens: 896 tiles = 6 waves of 148
    // and 8 tiles).  The row tiles behind that remainder then go to a second launch with K split, which fills the SMs for a
    // fraction of a wave; its partial sums are added as for any split.  The two extra launches cost about 10 us, so not where a unit takes
    // less (9728 x 1024 at 129 tokens: 25.7 us with the second launch, 19 without).  Library workspace only (a caller's workspace is sized for one launch).
    if (p.Z == 1 && may_tail && nb >= 8 && ckb_tune_get("gemm_tc_tail", 1)) {
        const int rem = tiles % slots;
        if (tiles > slots && rem > 0 && 4 * rem <= slots && rem % p.mtiles == 0 && rem / p.mtiles < p.ntiles && N % TC_ROWS == 0) {
            p.Zt = tc_pick_slices(rem, nb, slots);
            if (p.Zt > 1) p.tail_nt = rem / p.mtiles;
        }
    }
    p.nbzt = (nb + p.Zt - 1) / p.Zt;
    if (p.tail_nt) p.Zt = (nb + p.nbzt - 1) / p.nbzt;
    // time: rounds of units, a superblock of a unit at the measured rate (us, by width and format), its stores, and the launches of a split
    const double per_sb = wf == TC_W_Q4K ? (width == 128 ? 1.06 : (width == 96 ? 0.98 : 0.78)) : (width == 128 ? 1.32 : (width == 96 ? 1.26 : 1.13));
    const int units = (p.ntiles - p.tail_nt) * p.mtiles * p.Z, rounds = (units + slots - 1) / slots;
    p.us = rounds * (p.nbz * per_sb + 1.5 * width / 128) + (p.Z > 1 ? 4.0 : 0.0) + (p.tail_nt ? 10.0 + p.nbzt * per_sb : 0.0);
    return p;
}

static size_t tc_part_bytes(const TcPlan &p, int M, int N)
{
    return p.Z > 1 ? (size_t)p.Z * M * N * sizeof(float) : (p.tail_nt ? (size_t)p.Zt * M * p.tail_nt * TC_ROWS * sizeof(float) : 0);
}

typedef CUresult (*tc_encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                 CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// `rows` rows of row_bytes bytes (a multiple of 16), boxes of box_bytes x 128 rows; rows past the end read as zeros
static bool tc_make_map(CUtensorMap *map, const void *base, size_t row_bytes, size_t rows, unsigned box_bytes, CUtensorMapSwizzle swizzle)
{
    static tc_encode_fn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return false;
        }
        fn = (tc_encode_fn)p;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {box_bytes, TC_ROWS}, estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// weights of a launch over rows [0, N); Q6_K: the planes lie behind one another in every row
template <int WF>
static bool tc_maps(TcMaps *maps, const uint8_t *B, int N, int nb)
{
    if (WF == TC_W_Q4K) {
        if (!tc_make_map(&maps->w[0], B, (size_t)nb * Q4K_BYTES, (size_t)N, Q4K_BYTES, CU_TENSOR_MAP_SWIZZLE_NONE)) return false;
        maps->w[1] = maps->w[2] = maps->w[0];
        return true;
    }
    const size_t rb = ((size_t)nb * Q6K_BYTES + 15) & ~(size_t)15;
    return tc_make_map(&maps->w[0], B, rb, (size_t)N, 128, CU_TENSOR_MAP_SWIZZLE_128B) &&
           tc_make_map(&maps->w[1], B + (size_t)nb * 128, rb, (size_t)N, 64, CU_TENSOR_MAP_SWIZZLE_64B) &&
           tc_make_map(&maps->w[2], B + (size_t)nb * 192, rb, (size_t)N, 16, CU_TENSOR_MAP_SWIZZLE_NONE);
}

// The product over operand tiles: xt holds them (tiles of NT tokens), part the partial sums of a K split (part_bytes at hand).
template <int WF, int NT>
static int launch_tc(const uint8_t *xt, const void *B, const float *bias, float *C, int ldc, int M, int N, int nb, const TcPlan &plan, float *part, size_t part_bytes, cudaStream_t st)
{
    using Cfg = TcCfg<WF, NT>;
    auto kernel = gemm_kq_tc_kernel<WF, NT>;
    static int attr_set = 0;
    if (!attr_set) {
        cudaFuncAttributes fa;
        if (ckb_check_cuda((int)cudaFuncGetAttributes(&fa, kernel), "func attributes")) return CKB_ERR_CUDA;
        if (fa.numRegs != Cfg::REGS_LAUNCH)     // a different allocation at launch would make setmaxnreg.inc wait for registers that never come
            return ckb_fail(CKB_ERR_LIMIT, "gemm_kq_tc: kernel compiled with an unexpected register count");
        if (ckb_check_cuda((int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM), "smem attr")) return CKB_ERR_CUDA;
        attr_set = 1;
    }
    TcMaps maps;
    if (!tc_maps<WF>(&maps, (const uint8_t *)B, N, nb)) return ckb_fail(CKB_ERR_SHAPE, "gemm_kq_tc: no tensor map for %d rows of %d superblocks", N, nb);
    if (tc_part_bytes(plan, M, N) > part_bytes)
        return ckb_fail(CKB_ERR_LIMIT, "gemm_kq_tc: the workspace holds %zu bytes of partial sums, this call needs %zu", part_bytes, tc_part_bytes(plan, M, N));
    const int slots = ckb_sm_count() * Cfg::CTAS_PER_SM;
    const int mtiles = plan.mtiles, ntiles = plan.ntiles, Z = plan.Z, nbz = plan.nbz, tail_nt = plan.tail_nt, Zt = plan.Zt, nbzt = plan.nbzt;
    const int Nt = tail_nt * TC_ROWS;                  // rows (output columns) of the tail launch
    TcWork work = {(ntiles - tail_nt) * mtiles * Z, mtiles, ntiles - tail_nt, nb, nbz};
    dim3 grid((unsigned)(work.units < slots ? work.units : slots));
    if (Z == 1) {
        if (int rc = launch_pdl("gemm_kq_tc", kernel, grid, dim3(Cfg::THREADS), (size_t)Cfg::SMEM, st, maps, work, xt, (const uint8_t *)B, bias, C, ldc, (size_t)0, M, N - Nt,
                                ckb_device_error_word()))
            return rc;
        if (!tail_nt) return 0;
        const int n0 = N - Nt;
        const size_t rb = WF == TC_W_Q4K ? (size_t)nb * Q4K_BYTES : (((size_t)nb * Q6K_BYTES + 15) & ~(size_t)15);
        const uint8_t *Bt = (const uint8_t *)B + (size_t)n0 * rb;
        if (!tc_maps<WF>(&maps, Bt, Nt, nb)) return ckb_fail(CKB_ERR_SHAPE, "gemm_kq_tc: no tensor map for %d rows of %d superblocks", Nt, nb);
        work = {tail_nt * mtiles * Zt, mtiles, tail_nt, nb, nbzt};
        grid = dim3((unsigned)(work.units < slots ? work.units : slots));
        if (int rc = launch_pdl("gemm_kq_tc tail", kernel, grid, dim3(Cfg::THREADS), (size_t)Cfg::SMEM, st, maps, work, xt, Bt, nullptr, part, Nt, (size_t)M * Nt, M, Nt,
                                ckb_device_error_word()))
            return rc;
        const size_t mnt = (size_t)M * Nt;
        const unsigned tb = (unsigned)((mnt + 1023) / 1024 < 1184 ? (mnt + 1023) / 1024 : 1184);
        const float *bt = bias ? bias + n0 : nullptr;
        if (ldc % 4 == 0 && (((uintptr_t)(C + n0) | (uintptr_t)bt) & 15) == 0) gemm_splitk_sum_kernel<true><<<tb, 256, 0, st>>>(part, Zt, bt, C + n0, ldc, M, Nt);
        else gemm_splitk_sum_kernel<false><<<tb, 256, 0, st>>>(part, Zt, bt, C + n0, ldc, M, Nt);
        return ckb_check_launch("gemm_splitk_sum");
    }
    if (int rc = launch_pdl("gemm_kq_tc", kernel, grid, dim3(Cfg::THREADS), (size_t)Cfg::SMEM, st, maps, work, xt, (const uint8_t *)B, nullptr, part, N, (size_t)M * N, M, N,
                            ckb_device_error_word()))
        return rc;
    const size_t mn = (size_t)M * N;
    const unsigned blocks = (unsigned)((mn + 1023) / 1024 < 1184 ? (mn + 1023) / 1024 : 1184);
    if (N % 4 == 0 && ldc % 4 == 0 && (((uintptr_t)C | (uintptr_t)bias) & 15) == 0) gemm_splitk_sum_kernel<true><<<blocks, 256, 0, st>>>(part, Z, bias, C, ldc, M, N);
    else gemm_splitk_sum_kernel<false><<<blocks, 256, 0, st>>>(part, Z, bias, C, ldc, M, N);
    return ckb_check_launch("gemm_splitk_sum");
}

static int tc_launch(int wf, int nt, const uint8_t *xt, const void *B, const float *bias, float *C, int ldc, int M, int N, int nb, const TcPlan &plan, float *part,
                     size_t part_bytes, cudaStream_t st)
{
#define TC_GO(WF, NT) return launch_tc<WF, NT>(xt, B, bias, C, ldc, M, N, nb, plan, part, part_bytes, st)
    if (wf == TC_W_Q6K_PLANAR) switch (nt) { case 32: TC_GO(TC_W_Q6K_PLANAR, 32); case 64: TC_GO(TC_W_Q6K_PLANAR, 64); case 96: TC_GO(TC_W_Q6K_PLANAR, 96); default: TC_GO(TC_W_Q6K_PLANAR, 128); }
    switch (nt) { case 32: TC_GO(TC_W_Q4K, 32); case 64: TC_GO(TC_W_Q4K, 64); case 96: TC_GO(TC_W_Q4K, 96); default: TC_GO(TC_W_Q4K, 128); }
#undef TC_GO
}
static int tc_make_tiles(const void *A_q8, uint8_t *xt, int nt, int M, int nb, cudaStream_t st)
{
    const int mtiles = (M + nt - 1) / nt, xz = nb * mtiles >= 2 * ckb_sm_count() ? 1 : (nb * mtiles >= ckb_sm_count() ? 2 : 4);      // enough CTAs for every SM
    auto kernel = nt == 32 ? gemm_x_tiles_kernel<32> : (nt == 64 ? gemm_x_tiles_kernel<64> : (nt == 96 ? gemm_x_tiles_kernel<96> : gemm_x_tiles_kernel<128>));
    return launch_pdl("gemm_x_tiles", kernel, dim3(nb, mtiles, xz), dim3(256), (size_t)0, st, (const uint8_t *)A_q8, xt, M, nb);
}

// Token tile: 32 for batched decode (up to 64 tokens: two CTAs per SM), else the width whose plan takes least.
static int tc_width(int wf, int M, int N, int nb, bool may_tail)
{
    if (M <= ckb_tune_get("gemm_tc_small_max", 64)) return 32;
    const int forced = ckb_tune_get("gemm_tc_nt", 0);
    if (forced == 64 || forced == 96 || forced == 128) return forced;
    const TcPlan wide = tc_plan(wf, 128, M, N, nb, 1, may_tail);
    double best = wide.us;
    int width = 128;
    for (int w = 96; w >= 64 && !wide.tail_nt; w -= 32) {
        const double us = tc_plan(wf, w, M, N, nb, 1, may_tail).us;
        if (us < 0.97 * best) { best = us; width = w; }
    }
    return width;
}

// A caller that quantises rows straight into operand tiles (quantize_block_q8k_tile: one blob per tile of nt tokens and superblock) asks for the width
// and the sizes first.  Products over the same rows share one width: the one that suits the largest of them.
extern "C" int ckb_gemm_tc_width(int wf, int M, int N, int K) { return tc_width(wf, M, N, K / QK_K, true); }
extern "C" size_t ckb_gemm_tc_tile_bytes(int nt, int M, int K) { return (size_t)((M + nt - 1) / nt) * (K / QK_K) * q8k_tile_bytes(nt); }
extern "C" size_t ckb_gemm_tc_part_bytes(int wf, int nt, int M, int N, int K) { return tc_part_bytes(tc_plan(wf, nt, M, N, K / QK_K, nt == 32 ? 2 : 1, true), M, N); }
extern "C" int ckb_launch_gemm_tc_tiles(int wf, const void *tiles, int nt, const void *B, float *C, int ldc, int M, int N, int K, void *part, size_t part_bytes, void *stream)
{
    if (K % QK_K || ((uintptr_t)B & 15) || ((uintptr_t)tiles & 15)) return -1;
    return tc_launch(wf, nt, (const uint8_t *)tiles, B, nullptr, C, ldc, M, N, K / QK_K, tc_plan(wf, nt, M, N, K / QK_K, nt == 32 ? 2 : 1, true), (float *)part, part_bytes,
                     ckb_stream(stream));
}

// C[m * ldc + n] = A_q8[m] . W[n] (+ bias[n]).  wf: TC_W_Q4K (the reference's block_q4_K rows) or TC_W_Q6K_PLANAR.
// Returns -1 when the shape is not handled here (caller falls back to the per-token path).  min_tokens: smallest M
// worth the tensor-core path (tokens past M are zeros).
extern "C" int ckb_launch_gemm_tc_ws(int wf, const void *A_q8, const void *B, const float *bias, float *C, int ldc, int M, int N, int K, int min_tokens,
                                     void *ws, size_t ws_bytes, void *stream)
{
    if (M < min_tokens || K % QK_K || ((uintptr_t)B & 15) || ((uintptr_t)A_q8 & 3) || ((uintptr_t)ws & 255) || ckb_tune_get("gemm_tc", 1) == 0) return -1;
    const int nb = K / QK_K, nt = tc_width(wf, M, N, nb, ws == nullptr);
    const TcPlan plan = tc_plan(wf, nt, M, N, nb, nt == 32 ? 2 : 1, ws == nullptr);
    const size_t xt_bytes = (ckb_gemm_tc_tile_bytes(nt, M, K) + 255) & ~(size_t)255, part_bytes = tc_part_bytes(plan, M, N);
    // A caller that records the launch in a CUDA graph brings its own workspace: the library's pool may be freed and
    // regrown by any later call that needs more, which would leave a captured pointer dangling.
    if (ws && xt_bytes + part_bytes > ws_bytes)
        return ckb_fail(CKB_ERR_LIMIT, "gemm_kq_tc: the caller's workspace holds %zu bytes, this call needs %zu", ws_bytes, xt_bytes + part_bytes);
    uint8_t *xt = ws ? (uint8_t *)ws : (uint8_t *)ckb_scratch(CKB_SLOT_G, xt_bytes + part_bytes);
    if (!xt) return CKB_ERR_CUDA;
    cudaStream_t st = ckb_stream(stream);
    if (int rc = tc_make_tiles(A_q8, xt, nt, M, nb, st)) return rc;
    return tc_launch(wf, nt, xt, B, bias, C, ldc, M, N, nb, plan, reinterpret_cast<float *>(xt + xt_bytes), part_bytes, st);
}

extern "C" int ckb_launch_gemm_tc(int wf, const void *A_q8, const void *B, const float *bias, float *C, int ldc, int M, int N, int K, int min_tokens,
                                  void *stream)
{
    return ckb_launch_gemm_tc_ws(wf, A_q8, B, bias, C, ldc, M, N, K, min_tokens, NULL, 0, stream);
}

// Upper bound of the workspace one call with these sizes can need (activation tiles plus the partial sums of the largest
// K split the launcher picks by itself), for callers that allocate it once.
extern "C" size_t ckb_gemm_tc_workspace_bytes(int M, int N, int K)
{
    if (M <= 0 || N <= 0 || K <= 0 || K % QK_K) return 0;
    const int nb = K / QK_K;
    const size_t blob = TcTile<128>::XBLOB;
    const size_t mtiles = (size_t)(M + 31) / 32;
    const size_t xt = (mtiles * nb * blob + 255) & ~(size_t)255;
    int zmax = nb / 4 < 1 ? 1 : (nb / 4 > 16 ? 16 : nb / 4);
    size_t part = zmax > 1 ? (size_t)zmax * M * N * sizeof(float) : 0;
    if (M > 128) {                                     // split only while the tiles leave half of the SMs idle
        const size_t most = (size_t)zmax * (ckb_sm_count() / 2) * TC_ROWS * 128 * sizeof(float);
        if (part > most) part = most;
    }
    return xt + part + 256;
}

extern "C" int ckb_launch_gemm_q4k_tc(const void *A_q8, const void *B, const float *bias, float *C, int M, int N, int K, void *stream)
{
    return ckb_launch_gemm_tc(TC_W_Q4K, A_q8, B, bias, C, N, M, N, K, ckb_tune_get("gemm_tc_min_tokens", 16), stream);
}

// gemm_nt_q6_k_q8_k (src/kernels/gemm_kernels_q6k_q8k.c:1243-1268) over weights in the row-planar layout
extern "C" int ckb200_dev_gemv_q6_k_planar_q8_k(float *, const void *, const void *, int, int, void *);
extern "C" int ckb200_dev_add_bias_rows(float *, const float *, int, int, void *);
extern "C" int ckb_launch_gemm_q6k_mma(const void *A_q8, const void *B_planar, const float *bias, float *C, int ldc, int M, int N, int K, void *stream);
extern "C" int ckb200_dev_gemm_nt_q6_k_planar_q8_k(const void *A_q8, const void *B_planar, const float *bias, float *C, int M, int N, int K, void *stream)
{
    if (!A_q8 || !B_planar || !C || M <= 0 || N <= 0 || K <= 0) return 0;
    if (ckb_ensure_init()) return CKB_ERR_NO_DEVICE;
    int rc = ckb_launch_gemm_q6k_mma(A_q8, B_planar, bias, C, N, M, N, K, stream);        // 4 to 64 tokens: integer MMA over the planes (gemm_q6k_mma.cu)
    if (rc >= 0) return rc;
    rc = ckb_launch_gemm_tc(TC_W_Q6K_PLANAR, A_q8, B_planar, bias, C, N, M, N, K, ckb_tune_get("gemm_tc_min_tokens", 16), stream);
    if (rc >= 0) return rc;
    for (int m = 0; m < M; ++m) {
        const int r2 = ckb200_dev_gemv_q6_k_planar_q8_k(C + (size_t)m * N, B_planar, (const uint8_t *)A_q8 + (size_t)m * (K / QK_K) * Q8K_BYTES, N, K, stream);
        if (r2) return r2;
    }
    return bias ? ckb200_dev_add_bias_rows(C, bias, M, N, stream) : 0;
}
