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
// are accumulated in fp32 in tensor memory, read back with tcgen05.ld once per
// superblock and combined with the fp32 scales in registers: acc += d_x * (d * T - dmin * T2).
// The accumulators hold every integer below 2^24, and no sum of a superblock is larger as long as its terms do not pile up on one side: the largest products all of one
// sign make 3.1e7 (Q4_K) and 1.3e8 (Q6_K).  Beyond 2^24 each MMA cuts the running sum off at its last place: 3e-7 and 7e-7 from 64 bits on rows of one sign,
// where the integer-MMA kernels, with 32-bit sums rounded once, are at 2e-7; on ordinary rows both are at 5e-8 (2-norm; 200 x 1280, 64 tokens).
// Q6_K: A = (q6 - 32) * sc (src/kernels/gemm_kernels_q6k_q8k.c:86-116), the offset is inside the operand, so there
// is no T2.  The product is an exact fp16 integer whenever |q6 - 32| * |sc| <= 2048, always for |sc| <= 64.  Above that fp16 holds the even integers
// only: the operand is the nearest of them, and what it lacks (-1, 0 or 1) is an operand of its own, multiplied into the same accumulator.  Files made by a
// quantiser that scales a superblock to its largest sub-scale have such scales in every superblock; whether there are rests is found per stage and 32 rows
// (multiplying them costs about a seventh of the time).
//
// Two kernels:
//  * gemm_x_tiles_kernel expands the Q8_K activations once into fp16 operand tiles in the exact shared-memory
//    layout of the MMA (K-major, no swizzle, 8 x 16-byte core matrices), one contiguous blob per (token tile,
//    superblock), so the GEMM fetches them with plain 1-D bulk copies.
//  * gemm_kq_tc_kernel<WF, NT>: one CTA owns 128 weight rows (the M = 128 operand, one TMEM lane each) and one tile of NT tokens
//    (the N operand, TMEM columns; fewer tokens are zero-padded).  Warp-specialised:
//        warp 0       loader of activations: bulk copies of 128-deep stages (256-deep up to 64 tokens), of the bsum tile and of the block scales of each superblock
//        warp 1       issuer: tcgen05.mma from one elected lane; tcgen05.commit frees stages and publishes accumulators
//        warp 2       loader of weights: the raw superblocks of all 128 rows, one tiled bulk copy each (Q6_K: one per plane)
//        warps 4-11   two expander sets, thread = row: raw bytes -> fp16 operand in 64-deep k-stages; Q4_K: also the 16-deep tile of mins and the (d, dmin) pairs
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
// The 512 TMEM columns at NT = 128: two T buffers (256), one T2 (128), four weight stages (128); up to 96 tokens T2 has two buffers, up to 64 eight stages fit.
//
// No unit of the SM is full (57344 x 8192 at 32 tokens / 28672 x 4096 at 333: issue slots 53 / 56 %, logic 40 / 33 %, fp16 27 / 16 %, fp32 21 / 26 %, tensor 23 / 55 %;
// fp16 arithmetic and logic issue every other cycle): what a superblock takes is instructions, and how far the warps' code lies apart, for eight kinds of work share one instruction cache.  So: the
// mins are made by the threads that have the header in registers (a warp of its own took 800 cycles a superblock and held up the drain), expander sets take superblocks in turn,
// waits are four instructions, the sums of a unit leave sixteen columns at a time (see there).  Before and after these, us, from Q8_K rows (the launch that makes tiles of
// them included), 40 calls in a row on a cool GPU (the power cap makes long runs up to a sixth slower: 333 tokens 118 to 125, 512 tokens 153):
//   28672 x 4096 Q4_K:  77 tokens 52.4 -> 45, 129: 80.6 -> 58, 333: 115 -> 108, 512: 140 -> 129 to 142
//   4096 x 14336 Q6_K:  129 tokens 60.4 -> 48, 512: 111 -> 95
//   57344 x 8192 Q4_K:  32 tokens 111 -> 74, 64: 222 -> 88;  8192 x 28672 Q6_K: 76 -> 61, 126 -> 70;  128256 x 8192 Q6_K at 32: 213 (4.05 TB/s of weights)
// (with the operand through shared memory 28672 x 4096 at 512 tokens took 268).
#include <cuda.h>
#include <pthread.h>

#include "q8k_block.cuh"
#include "quant_units.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "runtime.h"
#include "tcgen05.cuh"

namespace ckb {

constexpr int TC_ROWS = 128;                          // rows of the weight operand per MMA
constexpr int TC_AUX = TC_ROWS * 32;                  // 16-deep tile of the mins: 4 KB
constexpr int TC_BSLOTS = 4, TC_XSLOTS = 4;           // rings: activation stages, per-superblock extras (mins, bsums, scales)
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

// Everything that depends on the width NT of the token tile and on the weight format.
template <int WF, int NT>
struct TcCfg : TcTile<NT> {
    static constexpr bool Q4 = WF == TC_W_Q4K;
    // raw superblocks of 128 rows: 144-byte rows, or the planes ql | qh | scales (1024-byte aligned: they are written swizzled)
    static constexpr int RAW_QH = TC_ROWS * 128, RAW_SC = RAW_QH + TC_ROWS * 64, RAW = Q4 ? TC_ROWS * Q4K_BYTES : RAW_SC + TC_ROWS * 16;
    static constexpr int RSLOTS = NT > 96 || NT == 64 ? 3 : (NT == 96 ? (Q4 ? 5 : 4) : (Q4 ? 7 : 5));        // ring of raw superblocks: what is left of shared memory
    static constexpr int BDEEP = NT > 64 ? 2 : 4;                    // 64-deep stages in a slot of the activation ring: half a superblock or all of it
    static constexpr int BSLOT = BDEEP * TcTile<NT>::STAGE;
    static constexpr int ADEEP = NT > 64 ? 1 : 2, ASLOTS = 4;        // ring of weight stages in tensor memory, 64-deep or 128-deep: one superblock or two
    // Q4_K: the expander sets take superblocks in turn; where they share the slots, each has barriers of its own for them.  Q6_K: a half of every superblock each.
    static constexpr int AEMPTIES = Q4 && ADEEP == 1 ? 2 * ASLOTS : ASLOTS, TAKERS = Q4 ? 4 : 8;      // warps that read a raw superblock
    // A Q4_K set skips every other superblock, so it must not come to the wait for superblock b before b - RSLOTS has landed: to a waiter two phases ahead a phase parity
    // reads as complete.  Where the sets share the weight slots b - 1 has to be multiplied first anyway; with slots of its own a set gets three superblocks ahead
    // (its raw wait of b comes behind its stores of b - 2, which need b - 4 multiplied, while b - 3 may still be in flight).  A ring of three then needs b - 2 multiplied first.
    static constexpr bool RAW_BEHIND_MMA = Q4 && ADEEP == 2 && RSLOTS <= 3;
    static constexpr int OFF_RAW = 0;
    static constexpr int OFF_B = OFF_RAW + RSLOTS * RAW;
    static constexpr int OFF_A2 = OFF_B + TC_BSLOTS * BSLOT;
    static constexpr int OFF_B2 = OFF_A2 + (Q4 ? TC_XSLOTS * TC_AUX : 0);
    static constexpr int OFF_DX = OFF_B2 + (Q4 ? TC_XSLOTS * TcTile<NT>::AUX : 0);
    static constexpr int OFF_DD = OFF_DX + TC_XSLOTS * NT * 4;                     // fp16 d | dmin of the rows
    static constexpr int OFF_BAR = OFF_DD + (Q4 ? TC_XSLOTS * TC_ROWS * 4 : 0);
    static constexpr int A_FULL = 0, A_EMPTY = A_FULL + ASLOTS, B_FULL = A_EMPTY + AEMPTIES, B_EMPTY = B_FULL + TC_BSLOTS, R_FULL = B_EMPTY + TC_BSLOTS,
                         R_EMPTY = R_FULL + RSLOTS, X_FULL = R_EMPTY + RSLOTS, X_EMPTY = X_FULL + TC_XSLOTS, T_FULL = X_EMPTY + TC_XSLOTS, T_EMPTY = T_FULL + 2,
                         T2_EMPTY = T_EMPTY + 2, DONE = T2_EMPTY + 1, BARS = DONE + 1;
    // Q6_K, a byte per (weight stage, lane quarter): there are rests
    static constexpr int OFF_WIDE = OFF_BAR + BARS * 8 + 16, SMEM = OFF_WIDE + 4 * ASLOTS * ADEEP;
    static constexpr int DRAIN_WARPS = NT > 32 ? 8 : 4;       // 4 TMEM lane quarters x column halves
    static constexpr int DRAIN_COLS = NT / (DRAIN_WARPS / 4); // token columns per drain thread
    static constexpr int THREADS = (12 + DRAIN_WARPS) * 32;
    // Register counts per role after setmaxnreg.  setmaxnreg.inc blocks until the CTA's own pool (threads x registers
    // at launch) can supply the registers, so 128 * CTL + 256 * EXP + 32 * DRAIN_WARPS * DRAIN must not exceed
    // THREADS * LAUNCH; the launcher checks the compiled register count against LAUNCH before the first launch.
    static constexpr int REGS_LAUNCH = NT > 32 ? 96 : 128, REGS_CTL = NT > 32 ? 48 : 128, REGS_EXP = NT > 32 ? 72 : 128, REGS_DRAIN = NT > 32 ? 144 : 128;
    static_assert(128 * REGS_CTL + 256 * REGS_EXP + 32 * DRAIN_WARPS * REGS_DRAIN <= THREADS * REGS_LAUNCH, "setmaxnreg targets exceed the CTA's register pool");
    static_assert(THREADS * REGS_LAUNCH <= 65536, "register plan");
    // T buffer u at column u * NT; T2 has two buffers too where they fit.  Q6_K has no T2; what its stages lack goes behind them, a slot for each stage of a superblock.
    static constexpr bool T2_TWICE = NT <= 96;
    static constexpr uint32_t TM_T2 = 2 * NT, TM_A = Q4 ? (T2_TWICE ? 4 : 3) * NT : 2 * NT, TM_R = TM_A + 32 * ADEEP * ASLOTS, TMEM_COLS = 512;
    static_assert(TM_R + (Q4 ? 0 : 32 * 4) <= TMEM_COLS, "tensor memory plan");
    // instruction descriptor: f16 x f16 -> f32, both operands K-major, M = 128, N = NT
    static constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(TC_ROWS >> 4) << 24);
    static_assert(NT % 32 == 0 && NT <= 128 && RAW % (Q4 ? 16 : 1024) == 0 && OFF_BAR % 8 == 0 && OFF_B % 128 == 0, "layout");
    static_assert(SMEM <= 227 * 1024, "shared memory plan");
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

// mbar_wait_spin in fewer instructions: it stands in loops of warps that share an instruction cache.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity)
{
    if (mbar_try_wait(bar, parity)) return true;
    uint32_t t0, t;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(t0));
#pragma unroll 1
    do {
        if (mbar_try_wait(bar, parity)) return true;
        asm volatile("mov.u32 %0, %%clock;" : "=r"(t));
    } while (t - t0 < (1u << 31));
    return false;
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
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate));
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

// 6-bit scales (or mins) of sub-blocks 4 n .. 4 n + 3 of a Q4_K superblock as bytes: their own word, and the four bits that lie with the other kind's
__device__ __forceinline__ uint32_t q4k_scales4(uint32_t six, uint32_t four, int n) { return n ? (four & 0x0F0F0F0Fu) | ((six >> 2) & 0x30303030u) : six & 0x3F3F3F3Fu; }

// The 64 weights of one row in a k-stage of a Q4_K superblock (two sub-blocks: 32 nibble bytes) times their scales (bytes 2 hi and 2 hi + 1 of sc):
// (1024 + n) * sc - 1024 * sc and (1024 + 16 n) * sc / 16 - 64 * sc, exact: only the result (at most 945) is rounded
__device__ __forceinline__ void q4k_expand(uint32_t sc, const uint4 &qa, const uint4 &qb, uint32_t (&o)[32])
{
    const __half2 k1024 = __floats2half2_rn(1024.0f, 1024.0f);
    const __half2 s_lo = __hsub2(bits_h2(__byte_perm(sc, 0x64646464u, 0x4040)), k1024), s_hi = __hsub2(bits_h2(__byte_perm(sc, 0x64646464u, 0x4141)), k1024);
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

// The same for Q6_K: k-stage 2 n + hi holds weights 128 n + 64 hi .. + 63: nibbles hi of the 64 ql bytes of half n, 2-bit planes 2 hi and
// 2 hi + 1 of its 32 qh bytes, scales 8 n + 4 hi .. + 3 (scw), one for each 16-byte piece of ql.  The row's planes lie as the swizzled copies left them.
struct Q6kStage {
    const uint8_t *ql, *qh;
    uint32_t scw;
    int n, row, shift, plane;         // right shift of ql; left rotation of qh that brings plane 2 hi to bits 4 and 5
    __device__ __forceinline__ Q6kStage(const uint8_t *raw_ql, const uint8_t *raw_qh, uint32_t scales, int r, int half, int hi)
        : ql(raw_ql + r * 128), qh(raw_qh + r * 64), scw(scales), n(half), row(r), shift(4 * hi), plane(4 - 4 * hi) {}
    // 16-byte pieces are permuted by the row's low three bits (128-byte swizzle) and by its bits 1-2 (64-byte swizzle)
    __device__ __forceinline__ uint4 low(int j) const { return *reinterpret_cast<const uint4 *>(ql + (((4 * n + j) ^ (row & 7)) << 4)); }
    __device__ __forceinline__ uint4 high(int j) const { return *reinterpret_cast<const uint4 *>(qh + (((2 * n + j) ^ ((row >> 1) & 3)) << 4)); }
    // four weights + 32 out of a word of each, piece J: bytes 0 .. 63
    template <int J>
    __device__ __forceinline__ uint32_t bytes(uint32_t l, uint32_t h) const { return ((l >> shift) & 0x0F0F0F0Fu) | (__funnelshift_l(h, h, J < 2 ? plane : plane - 2) & 0x30303030u); }
    // scale of piece J, exact: 1152 + scale, less 1152
    template <int J>
    __device__ __forceinline__ __half2 scale() const { return __hsub2(bits_h2(__byte_perm(scw ^ 0x80808080u, 0x64646464u, 0x4040 + 0x0101 * J)), __floats2half2_rn(1152.0f, 1152.0f)); }
    // weights of the bytes 0 2 (e = 0) or 1 3
    static __device__ __forceinline__ __half2 weight(uint32_t q, int e) { return __hsub2(bits_h2(__byte_perm(q, 0x64646464u, e ? 0x4341 : 0x4240)), __floats2half2_rn(1056.0f, 1056.0f)); }

    template <int J>
    __device__ __forceinline__ void piece(const uint4 &l, const uint4 &h, uint32_t *o) const
    {
        const __half2 sc = scale<J>();
        const uint32_t w[4] = {l.x, l.y, l.z, l.w}, g[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t q = bytes<J>(w[i], g[i]);
            o[2 * i] = h2_bits(__hmul2(weight(q, 0), sc));
            o[2 * i + 1] = h2_bits(__hmul2(weight(q, 1), sc));
        }
    }
    __device__ __forceinline__ void expand(uint32_t (&o)[32]) const
    {
        const uint4 h0 = high(0), h1 = high(1);
        piece<0>(low(0), h0, o);
        piece<1>(low(1), h1, o + 8);
        piece<2>(low(2), h0, o + 16);
        piece<3>(low(3), h1, o + 24);
    }
    // Pieces 2 h and 2 h + 1 as the rounded products and what they lack, which one fused multiply-add gives exactly.  Rarely run, so short rather than fast.
    __device__ __forceinline__ void rests(int h, uint32_t (&o)[16], uint32_t (&t)[16]) const
    {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint4 l = low(2 * h + j), g4 = high(j);
            const uint32_t w[4] = {l.x, l.y, l.z, l.w}, g[4] = {g4.x, g4.y, g4.z, g4.w};
            const __half2 sc = __hsub2(bits_h2(__byte_perm(scw ^ 0x80808080u, 0x64646464u, 0x4040u + 0x0101u * (uint32_t)(2 * h + j))), __floats2half2_rn(1152.0f, 1152.0f));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t q = ((w[i] >> shift) & 0x0F0F0F0Fu) | (__funnelshift_l(g[i], g[i], plane - 2 * h) & 0x30303030u);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const __half2 v = weight(q, e), p = __hmul2(v, sc);
                    o[8 * j + 2 * i + e] = h2_bits(p);
                    t[8 * j + 2 * i + e] = h2_bits(__hfma2(v, sc, __hneg2(p)));
                }
            }
        }
    }
};
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

struct TcMaps { CUtensorMap w[3]; };                  // Q4_K: rows of one matrix, or of two; Q6_K: planes ql, qh, scales

// Work of a product: units dealt round-robin to persistent CTAs, token tiles innermost; a launch does those from `begin` on.  First `whole` units, a tile of the first row tiles and all of K each,
// which write C, bias included; then the last split_nt row tiles in K slices of nbz superblocks, which write partial sums (the launcher adds them up in a fixed
// order).  Only the loaders and the drain know where a unit ends; the other roles see one run of superblocks, so that the next unit's
// weights are expanded and multiplied while the last one's sums are stored (a CTA per unit spent 6 us of 23 starting and storing).
struct TcWork {
    int begin, units, whole, mtiles, split_nt, nb_row, nbz;
    int rows0;                                         // rows of the first matrix, a multiple of TC_ROWS; a second one behind it, or INT_MAX
    __device__ __forceinline__ int mt(int u) const { return u % mtiles; }
    __device__ __forceinline__ int nt(int u) const { return u < whole ? u / mtiles : whole / mtiles + (u - whole) / mtiles % split_nt; }
    __device__ __forceinline__ int z(int u) const { return u < whole ? 0 : (u - whole) / mtiles / split_nt; }
    __device__ __forceinline__ int kb0(int u) const { return z(u) * nbz; }
    __device__ __forceinline__ int nb(int u) const { return u < whole ? nb_row : min(nbz, nb_row - kb0(u)); }
};

template <int WF, int NT>
__global__ void __launch_bounds__(TcCfg<WF, NT>::THREADS, 1)
gemm_kq_tc_kernel(const __grid_constant__ TcMaps maps, const TcWork work, const uint8_t *__restrict__ xt, const uint8_t *__restrict__ B, const float *__restrict__ bias,
                  float *__restrict__ C, int ldc, float *__restrict__ part, int M, int N, int *__restrict__ dev_err)
{
    using Cfg = TcCfg<WF, NT>;
    constexpr bool Q4 = Cfg::Q4;
    uint32_t total = 0;                               // superblocks of all this CTA's units
    for (int u = work.begin + blockIdx.x; u < work.units; u += gridDim.x) total += (uint32_t)work.nb(u);
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t s_base = smem_u32(smem), s_bar = s_base + Cfg::OFF_BAR;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + Cfg::OFF_BAR + Cfg::BARS * 8);
#define BAR(i) (s_bar + 8u * (uint32_t)(i))

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid == 0) {
        for (int i = 0; i < Cfg::ASLOTS; ++i) { mbar_init(BAR(Cfg::A_FULL + i), 4); }
        for (int i = 0; i < Cfg::AEMPTIES; ++i) mbar_init(BAR(Cfg::A_EMPTY + i), 1);
        for (int i = 0; i < TC_BSLOTS; ++i) { mbar_init(BAR(Cfg::B_FULL + i), 1); mbar_init(BAR(Cfg::B_EMPTY + i), 1); }
        for (int i = 0; i < Cfg::RSLOTS; ++i) { mbar_init(BAR(Cfg::R_FULL + i), 1); mbar_init(BAR(Cfg::R_EMPTY + i), Cfg::TAKERS); }
        for (int i = 0; i < TC_XSLOTS; ++i) {
            mbar_init(BAR(Cfg::X_FULL + i), Q4 ? 5 : 1);                            // loader (and its bytes), the set that writes the mins
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
#define TC_REGISTERS(n)                                                          \
    do {                                                                         \
        if constexpr ((n) < Cfg::REGS_LAUNCH) TC_SETMAXNREG("dec", n);           \
        else if constexpr ((n) > Cfg::REGS_LAUNCH) TC_SETMAXNREG("inc", n);      \
    } while (0)
#define TC_WAIT(bar, parity, code)                                        \
    if (!tc_wait(bar, parity)) { atomicExch(dev_err, code); break; }

    if (warp < 4) {
        TC_REGISTERS(Cfg::REGS_CTL);
        if (warp == 0) {
            // ------------------------------------------------------------ activations
            pdl_wait();                                // the tiles are what the kernel before this one writes; weights are nobody's output
            uint32_t g = 0, issued = 0, extras = 0;
            bool go = true;
            for (int u = work.begin + blockIdx.x; u < work.units && go; u += gridDim.x) {
                const uint8_t *blob = xt + ((size_t)work.mt(u) * work.nb_row + work.kb0(u)) * Cfg::XBLOB;
                for (int nb = work.nb(u); nb > 0 && go; --nb, ++g, blob += Cfg::XBLOB) {
                    const uint32_t x = g % TC_XSLOTS;
                    constexpr uint32_t PARTS = 4 / Cfg::BDEEP;
#pragma unroll
                    for (uint32_t h = 0; h < PARTS; ++h, ++issued) {
                        const uint32_t i = issued % TC_BSLOTS;
                        if (!tc_wait(BAR(Cfg::B_EMPTY + i), ((issued / TC_BSLOTS) & 1u) ^ 1u)) { go = false; break; }
                        if (tc_elect_one()) {
                            mbar_arrive_expect_tx(BAR(Cfg::B_FULL + i), Cfg::BSLOT);
                            bulk_g2s(s_base + Cfg::OFF_B + i * Cfg::BSLOT, blob + h * Cfg::BSLOT, Cfg::BSLOT, BAR(Cfg::B_FULL + i));
                        }
                    }
                    if (!go || !tc_wait(BAR(Cfg::X_EMPTY + x), ((g / TC_XSLOTS) & 1u) ^ 1u)) { go = false; break; }
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
            for (uint32_t j = issued > TC_BSLOTS ? issued - TC_BSLOTS : 0; j < issued; ++j) tc_wait(BAR(Cfg::B_FULL + j % TC_BSLOTS), (j / TC_BSLOTS) & 1u);
            for (uint32_t b = extras > TC_XSLOTS ? extras - TC_XSLOTS : 0; b < extras; ++b) tc_wait(BAR(Cfg::X_FULL + b % TC_XSLOTS), (b / TC_XSLOTS) & 1u);
        } else if (warp == 1) {
            // ------------------------------------------------------------ issuer: the warp runs the loop and the waits uniformly, one lane issues.  This
            // warp is a chain of short dependent steps that the MMAs of a 64-deep stage (64 to 260 cycles) have to cover: the stages of a superblock are unrolled
            // (in a loop they took a fifth longer); two superblocks unrolled as well were not faster and crowd the instruction cache.
            const uint64_t dB = tc_smem_desc(s_base + Cfg::OFF_B, Cfg::CHUNK), dA2 = tc_smem_desc(s_base + Cfg::OFF_A2, TC_ROWS * 16), dB2 = tc_smem_desc(s_base + Cfg::OFF_B2, Cfg::CHUNK);
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const bool leader = tc_elect_one();
            bool go = true;
#pragma unroll 1
            for (uint32_t b = 0; b < total && go; ++b) {
                const uint32_t u = b & 1u, p = (b >> 1) & 1u, x [[maybe_unused]] = b % TC_XSLOTS;
                const uint32_t a0 = Cfg::ADEEP == 2 ? 2 * u : 0, pa = Cfg::ADEEP == 2 ? p : u;
                const uint32_t pb = Cfg::BDEEP == 4 ? (b >> 2) & 1u : p, b0 = Cfg::BDEEP == 4 ? b & 3u : 2 * u;
                if (!tc_wait(BAR(Cfg::T_EMPTY + u), p ^ 1u)) { go = false; break; }
#pragma unroll
                for (uint32_t s = 0; s < 4; ++s) {
                    constexpr uint32_t half = Cfg::STAGE >> 4;
                    const uint32_t i = b0 + s / Cfg::BDEEP, a = a0 + s / Cfg::ADEEP;
                    if (s % Cfg::BDEEP == 0 && !tc_wait(BAR(Cfg::B_FULL + i), pb)) { go = false; break; }
                    if (s % Cfg::ADEEP == 0 && !tc_wait(BAR(Cfg::A_FULL + a), pa)) { go = false; break; }
                    tc_fence_after();                  // the expanders' stores, and (s = 0) the drain's loads of this accumulator, come before these MMAs
                    if (leader) {
                        uint32_t wide = 0;
                        if constexpr (!Q4) wide = *reinterpret_cast<const volatile uint32_t *>(smem + Cfg::OFF_WIDE + 4 * (Cfg::ADEEP * a0 + s));
                        const uint64_t d = dB + (uint64_t)(half * (Cfg::BDEEP * b0 + s));
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k)
                            tc_mma_ta(tm + NT * u, tm + Cfg::TM_A + 32 * (Cfg::ADEEP * a0 + s) + 8 * k, d + (uint64_t)(k * (2 * Cfg::CHUNK >> 4)), Cfg::IDESC, (s | k) ? 1u : 0u);
                        if constexpr (!Q4) {
                            if (wide) {
#pragma unroll 1
                                for (uint32_t k = 0; k < 4; ++k)
                                    tc_mma_ta(tm + NT * u, tm + Cfg::TM_R + 32 * s + 8 * k, d + (uint64_t)(k * (2 * Cfg::CHUNK >> 4)), Cfg::IDESC, 1u);
                            }
                        }
                        if (s % Cfg::ADEEP == Cfg::ADEEP - 1) tc_commit(BAR(Cfg::A_EMPTY + (Cfg::AEMPTIES > 4 ? 4 * (u ^ 1u) : 0) + a));       // to the set that writes there next
                        if (s % Cfg::BDEEP == Cfg::BDEEP - 1) tc_commit(BAR(Cfg::B_EMPTY + i));
                    }
                    __syncwarp();
                }
                if (!go) break;
                if constexpr (Q4) {
                    if ((!Cfg::T2_TWICE && !tc_wait(BAR(Cfg::T2_EMPTY), u ^ 1u)) || !tc_wait(BAR(Cfg::X_FULL + x), (b / TC_XSLOTS) & 1u)) { go = false; break; }
                    tc_fence_after();
                }
                if (leader) {
                    if constexpr (Q4) {
                        tc_mma(tm + Cfg::TM_T2 + (Cfg::T2_TWICE ? NT * u : 0), dA2 + (uint64_t)(x * (TC_AUX >> 4)), dB2 + (uint64_t)(x * (Cfg::AUX >> 4)), Cfg::IDESC, 0u);
                        tc_commit(BAR(Cfg::X_EMPTY + x));
                    }
                    tc_commit(BAR(Cfg::T_FULL + u));
                }
                __syncwarp();
            }
            if (!go) atomicExch(dev_err, DEV_ERR_MMA_WAIT);
            if (leader) tc_commit(BAR(Cfg::DONE));          // MMAs in flight finish before the tensor memory is freed
            tc_wait(BAR(Cfg::DONE), 0);
        } else if (warp == 2) {
            // ------------------------------------------------------------ raw weights
            uint32_t issued = 0, r = 0, ph = 1;
            bool go = true;
            for (int u = work.begin + blockIdx.x; u < work.units && go; u += gridDim.x) {
                const int n0 = work.nt(u) * TC_ROWS, kb0 = work.kb0(u), end = kb0 + work.nb(u);
                for (int kb = kb0; kb < end; ++kb) {
                    if (!tc_wait(BAR(Cfg::R_EMPTY + r), ph)) { atomicExch(dev_err, DEV_ERR_EMPTY_WAIT); go = false; break; }
                    if (tc_elect_one()) {
                        const uint32_t dst = s_base + Cfg::OFF_RAW + r * Cfg::RAW;
                        mbar_arrive_expect_tx(BAR(Cfg::R_FULL + r), Cfg::RAW);
                        if constexpr (Q4) {
                            tc_tma(dst, &maps.w[n0 < work.rows0 ? 0 : 1], kb * Q4K_BYTES, n0 < work.rows0 ? n0 : n0 - work.rows0, BAR(Cfg::R_FULL + r));
                        } else {
                            tc_tma(dst, &maps.w[0], kb * 128, n0, BAR(Cfg::R_FULL + r));
                            tc_tma(dst + Cfg::RAW_QH, &maps.w[1], kb * 64, n0, BAR(Cfg::R_FULL + r));
                            tc_tma(dst + Cfg::RAW_SC, &maps.w[2], kb * 16, n0, BAR(Cfg::R_FULL + r));
                        }
                    }
                    ++issued;
                    if (++r == Cfg::RSLOTS) { r = 0; ph ^= 1u; }
                }
            }
            for (uint32_t b = issued > Cfg::RSLOTS ? issued - Cfg::RSLOTS : 0; b < issued; ++b) tc_wait(BAR(Cfg::R_FULL + b % Cfg::RSLOTS), (b / Cfg::RSLOTS) & 1u);
        }
    } else if (warp < 12) {
        // ------------------------------------------------------------ weight expanders: thread = row = TMEM lane.  A stage is stored while the next one is expanded: what
        // is stored is waited for, and its barrier arrived at, behind that.
        TC_REGISTERS(Cfg::REGS_EXP);
        const uint32_t set = (uint32_t)(warp - 4) >> 2;
        const int row = tid & 127;
        bool go = true;
        auto publish = [&](uint32_t slot) {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(Cfg::A_FULL + slot));
        };
        if constexpr (Q4) {
            // The two sets take superblocks in turn: what a superblock costs beside its weights (waits, header, addresses, mins) is paid by four warps only
            // (sets that made half of every superblock each executed 1.4 times the instructions and took 1.15 times as long at 32 tokens).
            const uint32_t ta = tmem + Cfg::TM_A + ((uint32_t)(row & 96) << 16) + (Cfg::ADEEP == 2 ? 128 * set : 0);
            const uint32_t full = Cfg::ADEEP == 2 ? 2 * set : 0, empty = BAR(Cfg::A_EMPTY + (Cfg::ADEEP == 2 ? 2 : 4) * set);
            uint32_t r = set, rp = 0, pa = Cfg::ADEEP == 2 ? 1u : set ^ 1u;
            // slot for stage s: what was stored before has been published, the slot is empty
            auto acquire = [&](int s) -> bool {
                if (s % Cfg::ADEEP) return true;
                if (s) publish(full + (uint32_t)(s / Cfg::ADEEP - 1));
                if (!tc_wait(empty + 8u * (uint32_t)(s / Cfg::ADEEP), pa)) return false;
                tc_fence_after();
                return true;
            };
            for (uint32_t b = set; b < total; b += 2, pa ^= 1u) {
                const uint8_t *raw = smem + Cfg::OFF_RAW + r * Cfg::RAW;
                if constexpr (Cfg::RAW_BEHIND_MMA) TC_WAIT(empty, pa, DEV_ERR_EMPTY_WAIT);
                TC_WAIT(BAR(Cfg::R_FULL + r), rp, DEV_ERR_FULL_WAIT);
                const uint4 *p = reinterpret_cast<const uint4 *>(raw + row * Q4K_BYTES);
                const uint4 hdr = p[0];
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    uint32_t o[32];
                    q4k_expand(q4k_scales4(hdr.y, hdr.w, s >> 1) >> (16 * (s & 1)), p[1 + 2 * s], p[2 + 2 * s], o);
                    if (!acquire(s)) { go = false; break; }
                    tc_st32(ta + 32 * s, o);
                    if (s == 0) {
                        // The row's mins (each doubled: bsums come per 16 elements) and its block scales, for the MMA of T2 and the drain.  What lay there four superblocks
                        // ago has been read: the MMAs that emptied this slot were issued after the drain had taken the sums of that superblock.
                        const __half2 k1024 = __floats2half2_rn(1024.0f, 1024.0f);
                        const uint32_t x = b % TC_XSLOTS;
                        uint4 *a2 = reinterpret_cast<uint4 *>(smem + Cfg::OFF_A2 + x * TC_AUX + row * 16);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t mins = q4k_scales4(hdr.z, hdr.w >> 4, h);
                            uint32_t m[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) m[j] = h2_bits(__hsub2(bits_h2(__byte_perm(mins, 0x64646464u, 0x4040 + 0x0101 * j)), k1024));
                            a2[h * TC_ROWS] = make_uint4(m[0], m[1], m[2], m[3]);
                        }
                        *reinterpret_cast<uint32_t *>(smem + Cfg::OFF_DD + (x * TC_ROWS + row) * 4) = hdr.x;
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes -> visible to the tensor core
                    }
                }
                if (!go) { atomicExch(dev_err, DEV_ERR_EMPTY_WAIT); break; }
                // every lane's reads of the superblock have gone into what it stored
                publish(full + (uint32_t)(4 / Cfg::ADEEP - 1));
                if (lane == 0) {
                    mbar_arrive(BAR(Cfg::R_EMPTY + r));
                    mbar_arrive(BAR(Cfg::X_FULL + b % TC_XSLOTS));
                }
                r += 2;
                if (r >= Cfg::RSLOTS) { r -= Cfg::RSLOTS; rp ^= 1u; }
            }
        } else {
            // Set n makes stages 2 n and 2 n + 1 of every superblock.  (In turn, as above: every stage's code once more and both sets behind one ring, 1.3 times slower.)
            const uint32_t ta = tmem + Cfg::TM_A + ((uint32_t)(row & 96) << 16);
            uint32_t rests = 3, r = 0, rp = 0;        // rests, a bit per stage of the set: not known to be zeros in this warp's rows
            int stored = -1;                          // slot whose stores have not been published
            for (uint32_t b = 0; b < total; ++b) {
                const uint8_t *raw = smem + Cfg::OFF_RAW + r * Cfg::RAW;
                const uint32_t first = (Cfg::ADEEP == 2 ? 4 * (b & 1u) : 0) + 2 * set, pa = ((Cfg::ADEEP == 2 ? b >> 1 : b) & 1u) ^ 1u;      // 64-deep stage of the ring
                TC_WAIT(BAR(Cfg::R_FULL + r), rp, DEV_ERR_FULL_WAIT);
                const uint2 sc8 = *reinterpret_cast<const uint2 *>(raw + Cfg::RAW_SC + row * 16 + 8 * set);
                auto acquire = [&](int hi) -> bool {
                    if (hi % Cfg::ADEEP) return true;
                    if (stored >= 0) publish((uint32_t)stored);
                    stored = -1;
                    if (!tc_wait(BAR(Cfg::A_EMPTY + (first + (uint32_t)hi) / Cfg::ADEEP), pa)) return false;
                    tc_fence_after();
                    return true;
                };
#pragma unroll
                for (int hi = 0; hi < 2; ++hi) {
                    const uint32_t k = first + hi;
                    const Q6kStage st(raw, raw + Cfg::RAW_QH, hi ? sc8.y : sc8.x, row, set, hi);
                    const bool wide = __any_sync(0xffffffffu, q6k_wide(st.scw));
                    if (!wide && !(rests & (1u << hi))) {
                        uint32_t o[32];
                        st.expand(o);
                        if (!acquire(hi)) { go = false; break; }
                        tc_st32(ta + 32 * k, o);
                    } else {
                        // The issuer multiplies a slot of rests when any warp of the set has some, so a warp without leaves zeros in its rows, once.
                        // A slot of rests is free when the same stage of the superblock before this one has been multiplied.
                        if (!acquire(hi) || (Cfg::ADEEP == 2 && b > 0 && !tc_wait(BAR(Cfg::A_EMPTY + ((k / 2) ^ 2u)), ((b - 1) >> 1) & 1u))) { go = false; break; }
                        tc_fence_after();
#pragma unroll 1
                        for (int h = 0; h < 2; ++h) {
                            uint32_t o[16], f[16];
                            st.rests(h, o, f);
                            tc_st16(ta + 32 * k + 16 * h, o);
                            tc_st16(ta + Cfg::TM_R - Cfg::TM_A + 32 * (2 * set + hi) + 16 * h, f);
                        }
                        rests = wide ? rests | (1u << hi) : rests & ~(1u << hi);
                    }
                    if (lane == 0) *(volatile uint8_t *)(smem + Cfg::OFF_WIDE + 4 * k + (warp & 3)) = wide;
                    stored = (int)(k / Cfg::ADEEP);
                }
                if (!go) { atomicExch(dev_err, DEV_ERR_EMPTY_WAIT); break; }
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(Cfg::R_EMPTY + r));
                if (++r == Cfg::RSLOTS) { r = 0; rp ^= 1u; }
            }
            if (stored >= 0) publish((uint32_t)stored);
        }
    } else {
        // ------------------------------------------------------------ accumulator drain: thread = TMEM lane (weight row), DRAIN_COLS token columns
        TC_REGISTERS(Cfg::REGS_DRAIN);
        constexpr int COLS = Cfg::DRAIN_COLS;
        const int dw = warp - 12;
        const int q = dw & 3, ch = dw >> 2;           // warp % 4 is the TMEM lane quarter this warp may read (12 % 4 == 0)
        const int row = 32 * q + lane;
        const size_t rb6 = ((size_t)work.nb_row * Q6K_BYTES + 15) & ~(size_t)15;
        uint32_t b = 0;
        bool go = true;
        for (int u = work.begin + blockIdx.x; u < work.units && go; u += gridDim.x) {
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
                if (!tc_wait(BAR(Cfg::X_FULL + x), (b / TC_XSLOTS) & 1u)) { go = false; break; }
                if constexpr (Q4) dd_bits = *reinterpret_cast<const uint32_t *>(smem + Cfg::OFF_DD + (x * TC_ROWS + row) * 4);
                const float2 dd = __half22float2(bits_h2(dd_bits));
                const uint64_t d2 = pack2f(dd.x, dd.x), m2 = pack2f(-dd.y, -dd.y);
                const uint32_t dx = s_base + Cfg::OFF_DX + (x * NT + COLS * ch) * 4;
                if (!tc_wait(BAR(Cfg::T_FULL + buf), (b >> 1) & 1u)) { go = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(COLS * ch);
#pragma unroll
                for (int c = 0; c < COLS / 16; ++c) {
                    uint32_t t1[16], t2[16];
                    tc_ld16(taddr + NT * buf + 16 * c, t1);
                    if constexpr (Q4) tc_ld16(taddr + Cfg::TM_T2 + (Cfg::T2_TWICE ? NT * buf : 0) + 16 * c, t2);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c == COLS / 16 - 1) {             // the accumulators are in registers: the next superblocks may overwrite them
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(BAR(Cfg::T_EMPTY + buf));
                            if (Q4 && !Cfg::T2_TWICE) mbar_arrive(BAR(Cfg::T2_EMPTY));
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
                const bool whole = u < work.whole;
                const int m = m0 + COLS * ch, first = work.whole / work.mtiles * TC_ROWS;         // first row (column of C) of the split tiles
                const float bv = whole && bias ? bias[n] : 0.0f;
                const size_t ld = (size_t)(whole ? ldc : N - first);
                float *Cz = whole ? C + (size_t)m * ld + n : part + (size_t)work.z(u) * M * ld + (size_t)m * ld + (n - first);
                // This runs once per unit and comes from memory each time, 128 bytes of code at an L2 round trip each (a store per column, unrolled, took 17500 cycles a unit
                // of 32 tokens): so sixteen columns at a time, the others moved down.
#pragma unroll 1
                for (int left = M - m; left > 0 && left > M - m - COLS; left -= 16) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        float lo, hi;
                        unpack2(acc[i], lo, hi);
                        if (2 * i < left) *Cz = lo + bv;
                        Cz += ld;
                        if (2 * i + 1 < left) *Cz = hi + bv;
                        Cz += ld;
                    }
#pragma unroll
                    for (int i = 0; i + 8 < COLS / 2; ++i) acc[i] = acc[i + 8];
                }
            }
        }
        if (!go) atomicExch(dev_err, DEV_ERR_MMA_WAIT);
    }
#undef TC_WAIT
#undef TC_REGISTERS
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
    pdl_wait();
    pdl_trigger();
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

// How a product is cut: the first row tiles whole, the last split_nt of them in Z slices of nbz superblocks.
struct TcPlan { int mtiles, ntiles, split_nt, Z, nbz; double us; };
// us a superblock of a unit takes: units of 16 and 32 superblocks of one to five rounds, at 32, 64, 96 and 128 tokens
static double tc_superblock_us(int wf, int width)
{
    static const double q4[4] = {0.74, 0.90, 1.07, 1.30}, q6[4] = {1.14, 1.49, 1.80, 1.85};
    return (wf == TC_W_Q4K ? q4 : q6)[width / 32 - 1];
}
static void tc_slice(TcPlan *p, int nb, int z)
{
    p->nbz = (nb + z - 1) / z;
    p->Z = (nb + p->nbz - 1) / p->nbz;                 // no empty slice
}
static TcPlan tc_plan(int wf, int width, int M, int N, int nb)
{
    TcPlan p = {(M + width - 1) / width, (N + TC_ROWS - 1) / TC_ROWS, 0, 1, nb, 0.0};
    const int slots = ckb_sm_count(), tiles = p.ntiles * p.mtiles;
    const double per_sb = tc_superblock_us(wf, width), store = 1.5 * width / 128;
    p.us = (tiles + slots - 1) / slots * (nb * per_sb + store);
    const int forced = ckb_tune_get("gemm_tc_slices", 0), splitk = ckb_tune_get("gemm_tc_splitk", 1);
    if (forced > 0 && forced <= nb) {
        p.split_nt = p.ntiles;
        tc_slice(&p, nb, forced);
        return p;
    }
    // K is split where that takes less time, with what the partial sums cost: a launch that adds them, 3 us behind the product, and their way to L2 and
    // back at 3 TB/s.  Considered for up to 128 tokens and for any product whose tiles leave more than half of the SMs without a CTA (the k and
    // v projections of a prompt: 8 x 4 tiles); slices of at least 4 superblocks, at most 16.
    if (splitk && (M <= 128 || (splitk != 2 && 2 * tiles <= slots)))
        for (int z = 2; z <= 16 && nb / z >= 4; ++z) {
            TcPlan q = p;
            q.split_nt = p.ntiles;
            tc_slice(&q, nb, z);
            q.us = (tiles * q.Z + slots - 1) / slots * (q.nbz * per_sb + store) + 3.0 + (double)q.Z * M * N * 8e-6 / 3.0;
            if (q.us < p.us) p = q;
        }
    // A grid of whole waves plus a few units pays a full wave for those few (28672 x 4096 at 512 tokens: 896 tiles = 6 waves of 148
    // and 8 tiles; 57344 rows at 32 tokens: 3 waves and 4).  The row tiles behind that remainder then go to a second launch with K split, which fills the SMs for a
    // fraction of a wave; its partial sums are added as for any split.  The two extra launches cost about 8 us, so not where a unit takes
    // less (9728 x 1024 at 129 tokens: 25.7 us with the second launch, 19 without).
    const int rem = tiles % slots;
    if (!p.split_nt && nb >= 8 && tiles > slots && rem > 0 && 4 * rem <= slots && rem % p.mtiles == 0 && rem / p.mtiles < p.ntiles && N % TC_ROWS == 0 && ckb_tune_get("gemm_tc_tail", 1)) {
        int z = 1;
        double best = 0.0;
        for (int i = 1; i <= 16 && nb / i >= 4; ++i) {
            const double us = (rem * i + slots - 1) / slots * ((nb + i - 1) / i * per_sb + store);
            if (best == 0.0 || us < 0.93 * best) { best = us; z = i; }
        }
        if (z > 1) {
            p.split_nt = rem / p.mtiles;
            tc_slice(&p, nb, z);
            p.us = tiles / slots * (nb * per_sb + store) + best + 8.0;
        }
    }
    return p;
}

static size_t tc_part_bytes(const TcPlan &p, int M, int N)
{
    const int rest = N - (p.ntiles - p.split_nt) * TC_ROWS;
    return p.split_nt ? (size_t)p.Z * M * rest * sizeof(float) : 0;
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

struct TcSecond { const void *w; int rows0; };      // Q4_K: rows from rows0 on (a multiple of TC_ROWS) are those of a matrix of its own
// The product over operand tiles: xt holds them (tiles of NT tokens), part the partial sums of a K split (part_bytes at hand).
template <int WF, int NT>
static int launch_tc(const uint8_t *xt, const void *B, TcSecond second, const float *bias, float *C, int ldc, int M, int N, int nb, const TcPlan &plan, float *part, size_t part_bytes,
                     cudaStream_t st)
{
    using Cfg = TcCfg<WF, NT>;
    auto kernel = gemm_kq_tc_kernel<WF, NT>;
    static int attr_set = 0;
    if (!attr_set) {
        cudaFuncAttributes fa;
        if (ckb_check_cuda((int)cudaFuncGetAttributes(&fa, kernel), "func attributes")) return CKB_ERR_CUDA;
        if (Cfg::REGS_DRAIN != Cfg::REGS_LAUNCH && fa.numRegs != Cfg::REGS_LAUNCH)     // a different allocation at launch would make setmaxnreg.inc wait for registers that never come
            return ckb_fail(CKB_ERR_LIMIT, "gemm_kq_tc: kernel compiled with an unexpected register count");
        if (ckb_check_cuda((int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM), "smem attr")) return CKB_ERR_CUDA;
        attr_set = 1;
    }
    TcMaps maps;
    TcMaps more;
    if (!tc_maps<WF>(&maps, (const uint8_t *)B, second.w ? second.rows0 : N, nb) || (second.w && !tc_maps<WF>(&more, (const uint8_t *)second.w, N - second.rows0, nb)))
        return ckb_fail(CKB_ERR_SHAPE, "gemm_kq_tc: no tensor map for %d rows of %d superblocks", N, nb);
    if (second.w) maps.w[1] = more.w[0];
    if (tc_part_bytes(plan, M, N) > part_bytes)
        return ckb_fail(CKB_ERR_LIMIT, "gemm_kq_tc: the workspace holds %zu bytes of partial sums, this call needs %zu", part_bytes, tc_part_bytes(plan, M, N));
    const int slots = ckb_sm_count(), first = (plan.ntiles - plan.split_nt) * TC_ROWS, rest = N - first;
    const int whole = (plan.ntiles - plan.split_nt) * plan.mtiles;
    TcWork work = {0, whole, whole, plan.mtiles, plan.split_nt ? plan.split_nt : 1, nb, plan.nbz, second.w ? second.rows0 : 0x7fffffff};
    for (int i = 0; i < 2; ++i) {                      // whole tiles; slices
        if (i) { work.begin = whole; work.units = whole + plan.split_nt * plan.mtiles * plan.Z; }
        const int units = work.units - work.begin;
        if (units == 0) continue;
        if (int rc = launch_pdl(i ? "gemm_kq_tc slices" : "gemm_kq_tc", kernel, dim3((unsigned)(units < slots ? units : slots)), dim3(Cfg::THREADS), (size_t)Cfg::SMEM, st, maps, work, xt,
                                (const uint8_t *)B, bias, C, ldc, part, M, N, ckb_device_error_word()))
            return rc;
    }
    if (!plan.split_nt) return 0;
    const size_t mn = (size_t)M * rest;
    const unsigned blocks = (unsigned)((mn + 1023) / 1024 < 1184 ? (mn + 1023) / 1024 : 1184);
    const float *b2 = bias ? bias + first : nullptr;
    auto sum = rest % 4 == 0 && ldc % 4 == 0 && (((uintptr_t)(C + first) | (uintptr_t)b2 | (uintptr_t)part) & 15) == 0 ? gemm_splitk_sum_kernel<true> : gemm_splitk_sum_kernel<false>;
    return launch_pdl("gemm_splitk_sum", sum, dim3(blocks), dim3(256), (size_t)0, st, (const float *)part, plan.Z, b2, C + first, ldc, M, rest);
}

static int tc_launch(int wf, int nt, const uint8_t *xt, const void *B, TcSecond second, const float *bias, float *C, int ldc, int M, int N, int nb, const TcPlan &plan, float *part,
                     size_t part_bytes, cudaStream_t st)
{
#define TC_GO(WF, NT) return launch_tc<WF, NT>(xt, B, second, bias, C, ldc, M, N, nb, plan, part, part_bytes, st)
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

// Token tile: the width whose plan takes least, a wider one where two are alike.  Up to 32 tokens there is no choice.
static int tc_width(int wf, int M, int N, int nb)
{
    const int forced = ckb_tune_get("gemm_tc_nt", 0);
    if (M > 32 && (forced == 64 || forced == 96 || forced == 128)) return forced;
    if (M <= ckb_tune_get("gemm_tc_small_max", 32)) return 32;
    const TcPlan wide = tc_plan(wf, 128, M, N, nb);
    double best = wide.us;
    int width = 128;
    // One wave of the widest tiles and a few behind it, more than 96 tokens: narrower tiles are not tried, the plan's times do not tell the two apart there (22016 x 2048
    // Q4_K at 112 tokens: 29 us, with the 64-token tiles that the plan prefers 32; 9728 x 4096 at 150: 38 and 36).  Fewer tokens take the narrower tile that holds them
    // (22016 x 4096 at 64: 35 against 28 us, at 77: 36 against 33; Q6_K 22016 x 2048 at 64: 31 against 26).
    const bool one_wave = M > 96 && wide.split_nt && wide.split_nt < wide.ntiles && (wide.ntiles - wide.split_nt) * wide.mtiles <= ckb_sm_count();
    for (int w = 96; w >= 32 && !one_wave; w -= 32) {
        const double us = tc_plan(wf, w, M, N, nb).us;
        if (us < 0.97 * best) { best = us; width = w; }
    }
    return width;
}
// Whether this kernel takes a product from Q8_K rows in less time than an integer-MMA kernel that needs other_us; 3 us for the launch that makes operand tiles.
extern "C" int ckb_gemm_tc_beats(int wf, int M, int N, int K, double other_us)
{
    if (ckb_tune_get("gemm_tc", 1) == 0 || M < ckb_tune_get("gemm_tc_min_tokens", 16)) return 0;
    return tc_plan(wf, tc_width(wf, M, N, K / QK_K), M, N, K / QK_K).us + 3.0 < other_us;
}

// A caller that quantises rows straight into operand tiles (quantize_block_q8k_tile: one blob per tile of nt tokens and superblock) asks for the width
// and the sizes first.  Products over the same rows share one width: the one that suits the largest of them.
extern "C" int ckb_gemm_tc_width(int wf, int M, int N, int K) { return tc_width(wf, M, N, K / QK_K); }
extern "C" size_t ckb_gemm_tc_tile_bytes(int nt, int M, int K) { return (size_t)((M + nt - 1) / nt) * (K / QK_K) * q8k_tile_bytes(nt); }
extern "C" size_t ckb_gemm_tc_part_bytes(int wf, int nt, int M, int N, int K) { return tc_part_bytes(tc_plan(wf, nt, M, N, K / QK_K), M, N); }
extern "C" int ckb_launch_gemm_tc_tiles(int wf, const void *tiles, int nt, const void *B, float *C, int ldc, int M, int N, int K, void *part, size_t part_bytes, void *stream)
{
    if (K % QK_K || ((uintptr_t)B & 15) || ((uintptr_t)tiles & 15)) return -1;
    return tc_launch(wf, nt, (const uint8_t *)tiles, B, TcSecond{nullptr, 0}, nullptr, C, ldc, M, N, K / QK_K, tc_plan(wf, nt, M, N, K / QK_K), (float *)part, part_bytes,
                     ckb_stream(stream));
}

// Two Q4_K products over the same rows as one launch, the second's columns of C behind the first's: for products that are one round of whole tiles together (split along K,
// or in several rounds, they run side by side faster).  -1: not such.
extern "C" int ckb_gemm_tc_pairs(int nt, int M, int N, int N2, int K)
{
    const TcPlan p = tc_plan(TC_W_Q4K, nt, M, N + N2, K / QK_K), a = tc_plan(TC_W_Q4K, nt, M, N, K / QK_K), b = tc_plan(TC_W_Q4K, nt, M, N2, K / QK_K);
    return N % TC_ROWS == 0 && !p.split_nt && !a.split_nt && !b.split_nt && p.mtiles * p.ntiles <= ckb_sm_count();
}
extern "C" int ckb_launch_gemm_tc_pair(const void *tiles, int nt, const void *B, int N, const void *B2, int N2, float *C, int ldc, int M, int K, void *stream)
{
    if (K % QK_K || (((uintptr_t)B | (uintptr_t)B2 | (uintptr_t)tiles) & 15) || !ckb_gemm_tc_pairs(nt, M, N, N2, K)) return -1;
    return tc_launch(TC_W_Q4K, nt, (const uint8_t *)tiles, B, TcSecond{B2, N}, nullptr, C, ldc, M, N + N2, K / QK_K, tc_plan(TC_W_Q4K, nt, M, N + N2, K / QK_K), nullptr, 0, ckb_stream(stream));
}

// What a product from Q8_K rows needs: the operand tiles, and behind them the partial sums.
struct TcRows { int nt; TcPlan plan; size_t xt_bytes, part_bytes; };
static TcRows tc_rows(int wf, int M, int N, int K)
{
    TcRows r;
    r.nt = tc_width(wf, M, N, K / QK_K);
    r.plan = tc_plan(wf, r.nt, M, N, K / QK_K);
    r.xt_bytes = (ckb_gemm_tc_tile_bytes(r.nt, M, K) + 255) & ~(size_t)255;
    r.part_bytes = tc_part_bytes(r.plan, M, N);
    return r;
}
static int tc_launch_rows(int wf, const TcRows &r, const void *A_q8, const void *B, const float *bias, float *C, int ldc, int M, int N, int K, uint8_t *ws, cudaStream_t st)
{
    if (int rc = tc_make_tiles(A_q8, ws, r.nt, M, K / QK_K, st)) return rc;
    return tc_launch(wf, r.nt, ws, B, TcSecond{nullptr, 0}, bias, C, ldc, M, N, K / QK_K, r.plan, reinterpret_cast<float *>(ws + r.xt_bytes), r.part_bytes, st);
}
static bool tc_takes_rows(const void *A_q8, const void *B, int M, int K, int min_tokens)
{
    return !(M < min_tokens || K % QK_K || ((uintptr_t)B & 15) || ((uintptr_t)A_q8 & 3) || ckb_tune_get("gemm_tc", 1) == 0);
}

// C[m * ldc + n] = A_q8[m] . W[n] (+ bias[n]).  wf: TC_W_Q4K (the reference's block_q4_K rows) or TC_W_Q6K_PLANAR.
// Returns -1 when the shape is not handled here (caller falls back to the per-token path).  min_tokens: smallest M
// worth the tensor-core path (tokens past M are zeros).
extern "C" int ckb_launch_gemm_tc_ws(int wf, const void *A_q8, const void *B, const float *bias, float *C, int ldc, int M, int N, int K, int min_tokens,
                                     void *ws, size_t ws_bytes, void *stream)
{
    if (!tc_takes_rows(A_q8, B, M, K, min_tokens) || ((uintptr_t)ws & 255)) return -1;
    const TcRows r = tc_rows(wf, M, N, K);
    // A caller that records the launch in a CUDA graph brings its own workspace: the library's pool may be freed and
    // regrown by any later call that needs more, which would leave a captured pointer dangling.
    if (ws && r.xt_bytes + r.part_bytes > ws_bytes)
        return ckb_fail(CKB_ERR_LIMIT, "gemm_kq_tc: the caller's workspace holds %zu bytes, this call needs %zu", ws_bytes, r.xt_bytes + r.part_bytes);
    uint8_t *xt = ws ? (uint8_t *)ws : (uint8_t *)ckb_scratch(CKB_SLOT_G, r.xt_bytes + r.part_bytes);
    if (!xt) return CKB_ERR_CUDA;
    return tc_launch_rows(wf, r, A_q8, B, bias, C, ldc, M, N, K, xt, ckb_stream(stream));
}

// The same for a product that needs no workspace elsewhere (the integer-MMA kernels take it), whose callers therefore use any stream and thread, record it in graphs
// and call it on a full device.  It comes here where none of that matters: on the library's own stream, outside a capture, over a workspace that no call on another
// stream touches, all launches of a call behind one another whichever thread makes them.  -1: elsewhere, or no room.
extern "C" int ckb_launch_gemm_tc_own(int wf, const void *A_q8, const void *B, const float *bias, float *C, int M, int N, int K, void *stream)
{
    static pthread_mutex_t lock = PTHREAD_MUTEX_INITIALIZER;
    if (ckb_ensure_init()) return CKB_ERR_NO_DEVICE;
    if (!ckb_on_own_stream(stream) || !tc_takes_rows(A_q8, B, M, K, 0)) return -1;
    const TcRows r = tc_rows(wf, M, N, K);
    pthread_mutex_lock(&lock);
    uint8_t *ws = (uint8_t *)ckb_scratch_if_room(CKB_SLOT_O, r.xt_bytes + r.part_bytes);
    const int rc = ws ? tc_launch_rows(wf, r, A_q8, B, bias, C, N, M, N, K, ws, ckb_stream(stream)) : -1;
    pthread_mutex_unlock(&lock);
    return rc;
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
extern "C" int ckb_gemm_q6k_mma_takes(const void *A_q8, const void *B_planar, int M, int N, int K);
extern "C" int ckb_gemm_q6k_mma_best(const void *A_q8, const void *B_planar, int M, int N, int K);
extern "C" int ckb200_dev_gemm_nt_q6_k_planar_q8_k(const void *A_q8, const void *B_planar, const float *bias, float *C, int M, int N, int K, void *stream)
{
    if (!A_q8 || !B_planar || !C || M <= 0 || N <= 0 || K <= 0) return 0;
    if (ckb_ensure_init()) return CKB_ERR_NO_DEVICE;
    int rc = -1;
    if (ckb_gemm_q6k_mma_takes(A_q8, B_planar, M, N, K)) {                                // up to 64 tokens: integer MMA over the planes (gemm_q6k_mma.cu), or as for Q4_K
        if (!ckb_gemm_q6k_mma_best(A_q8, B_planar, M, N, K)) rc = ckb_launch_gemm_tc_own(TC_W_Q6K_PLANAR, A_q8, B_planar, bias, C, M, N, K, stream);
        if (rc < 0) rc = ckb_launch_gemm_q6k_mma(A_q8, B_planar, bias, C, N, M, N, K, stream);
    }
    if (rc >= 0) return rc;
    rc = ckb_launch_gemm_tc(TC_W_Q6K_PLANAR, A_q8, B_planar, bias, C, N, M, N, K, ckb_tune_get("gemm_tc_min_tokens", 16), stream);
    if (rc >= 0) return rc;
    for (int m = 0; m < M; ++m) {
        const int r2 = ckb200_dev_gemv_q6_k_planar_q8_k(C + (size_t)m * N, B_planar, (const uint8_t *)A_q8 + (size_t)m * (K / QK_K) * Q8K_BYTES, N, K, stream);
        if (r2) return r2;
    }
    return bias ? ckb200_dev_add_bias_rows(C, bias, M, N, stream) : 0;
}
