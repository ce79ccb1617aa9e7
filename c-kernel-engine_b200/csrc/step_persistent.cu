// One decode step of one sequence as ONE launch: all layers and the LM head.
//
// The reference's generated decode function issues, per layer, residual add, RMSNorm, quantisation, q / k / v projections, RoPE, cache store, attention,
// ... one call after another (version/v7/scripts/codegen_v7.py:569-931).  As a launch each, thirteen to a layer, the step was the chain of their latencies:
// a token of the Qwen2-0.5B shape (1024 keys) reads 0.4 GB, 60 us at HBM speed, and took 829 us; of the Llama-3-8B shape (4096 keys) 6 GB, 0.9 ms, and took 2.28 ms.
//
// Here one CTA per SM stays for the whole step and a layer is five phases with a grid-wide barrier behind each:
//
//   0  x += down, RMSNorm, quantise | q, k, v products | RoPE, query row and cache rows written
//   1  attention: a CTA takes a run of keys of one kv head; the last CTA of a kv head to finish merges the runs
//   2  quantise the attention row   | o product
//   3  x += o, RMSNorm, quantise    | gate and up products | SwiGLU
//   4  quantise the SwiGLU row      | down product
//
// Every CTA keeps the residual row and repeats norm and quantisation into its own shared memory: a few KB out of L2 against a launch.  What hides the latencies
// of a barrier and of a prologue is that weights do not depend on them: the first rows of the coming product are loaded into registers ahead of them.
// The arithmetic of each piece is that of the stand-alone kernels (the same integer sums and rounding calls); sums over warps and keys are taken in another order.
//
// The two shapes above take 615 us and 1.79 ms in this form (603 and 1.74 as a cooperative launch that needs every SM), Qwen2-0.5B with Q5_0 projections 1020 -> 640 us (2000 keys).  What is left is five barriers a layer (1 us each: release, poll) and
// the pieces that wait for one another behind them; products run at 24 B a cycle and SM, which is both the integer-issue rate and the SM's share of HBM.
//
// Barriers need every CTA that takes part to be on an SM, and the step does not ask for the whole GPU: CTAs enrol as they start, and those that have done so when all
// are there, or a short while after the first, do the step between them (the deal of rows and keys is made for p.ctas CTAs, and a CTA takes several shares where there are
// fewer: the same results, bit for bit).  One that comes later leaves at once.  So the step runs beside a kernel that holds SMs, and in a context that has fewer of
// them.
//
// Every wait is bounded: a CTA that gives up sets the error word and leaves, the others follow; the last to leave zeroes the counters and, as every step does
// whatever came of it, moves the position on.
#include "add_rmsnorm_q8k.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "runtime.h"
#include "step_persistent.h"
#include "step_units.cuh"

namespace ckb {

constexpr int PS_NW = 16, PS_THREADS = PS_NW * 32;
constexpr int PS_R = 2;                       // rows per lane group: the pair that RoPE and SwiGLU need
constexpr int PS_KEYS = 4;                    // keys a warp scores at a time: 4 keys x 8 heads = one score per lane
constexpr int PS_MIN_RUN = 32, PS_MERGE = 32; // attention: fewest keys of a CTA, runs of keys merged at a time
constexpr int PS_MAX_CTAS = 256, PS_MAX_HALF = 64;
constexpr int PS_JOIN_CYCLES = 40000;          // how long the first CTA waits for the others: they all start within 2 us on SMs that are free
constexpr uint32_t PS_CLOSED = 0x80000000u;
enum { PS_ARRIVALS = 0, PS_LEFT, PS_JOINED, PS_MEMBERS, PS_HEADS };      // words of p.sync; PS_HEADS + g: runs of keys of kv head g that are done
constexpr int PS_MAX_SMEM = 219 * 1024;       // dynamic; the rest of the 227 KB holds PsShared
enum { PS_EPI_ROPE_Q, PS_EPI_ROPE_K, PS_EPI_STORE_V, PS_EPI_SWIGLU, PS_EPI_STORE };

#ifdef CKB_STEP_TRACE
// Tuning aid (build with -DCKB_STEP_TRACE): cycle counts at the boundaries of every phase of every CTA; ckb200_step_trace copies them out.
constexpr int PS_TRACE_PHASES = 512;
static __device__ long long ps_trace[PS_MAX_CTAS * PS_TRACE_PHASES * 8];
#define PS_TRACE(k, i) do { if (threadIdx.x == 0 && (k) < PS_TRACE_PHASES) ps_trace[((size_t)blockIdx.x * PS_TRACE_PHASES + (k)) * 8 + (i)] = clock64(); } while (0)
#else
#define PS_TRACE(k, i) do { } while (0)
#endif

// ---------------------------------------------------------------- the CTA's state

struct PsShared {
    PsParams p;
    float4 red[PS_NW / 4];
    float part[PS_NW][32], cs[2][PS_MAX_HALF];
    __align__(16) float prob[PS_NW][PS_KEYS * PS_MAX_GROUP + PS_MAX_GROUP];       // attention: a warp's probabilities and corrections
    __align__(16) PsLayer layer[2];
    long long limit;
    int *dev_err;
    float inv_d;
    int pos, dead, last;
    int run, used;                    // attention: keys of a run, runs of the context
    int rank, members;                // this CTA among those that do the step (-1: it came too late)
};
static_assert(sizeof(PsLayer) % 16 == 0, "copied by 16 bytes");
__shared__ PsShared sh;
extern __shared__ __align__(128) uint8_t ps_smem[];   // residual row | quantised input row or attention buffers
__device__ __forceinline__ float *ps_x() { return reinterpret_cast<float *>(ps_smem); }
__device__ __forceinline__ uint8_t *ps_stage() { return ps_smem + (size_t)sh.p.Da * 4; }

__device__ __forceinline__ void ps_arrive()
{
    __syncthreads();                  // every thread's stores come before the release below
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(sh.p.sync + PS_ARRIVALS) : "memory");
}
// `target`: arrivals of all phases so far
__device__ __forceinline__ bool ps_wait(uint32_t target)
{
    asm volatile("cp.async.wait_all;" ::: "memory");      // next layer's entry
    if (threadIdx.x == 0) {
        const unsigned *at = sh.p.sync + PS_ARRIVALS;
        const long long t0 = clock64(), limit = sh.limit;
        for (;;) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(at) : "memory");
            if ((int)(v - target) >= 0) break;
            if (clock64() - t0 > limit) {
                atomicExch(sh.dev_err, DEV_ERR_FULL_WAIT);
                sh.dead = 1;
                break;
            }
        }
    }
    __syncthreads();
    return sh.dead == 0;
}

// One thread per CTA: its place among the CTAs that do this step, and how many those are.  Tickets are handed out until all are taken or the first CTA's patience
// ends; whoever closes the list publishes its length.
__device__ __forceinline__ void ps_enrol(unsigned *sync, int expected, long long limit, int *dev_err, int &rank, int &members)
{
    const uint32_t ticket = atomicAdd(sync + PS_JOINED, 1u);
    rank = -1;
    members = 0;
    if (ticket >= (uint32_t)expected) return;                        // closed, or more CTAs than shares
    const long long t0 = clock64();
    uint32_t n = ticket + 1 == (uint32_t)expected ? (uint32_t)expected : 0;
    if (n) {
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(sync + PS_MEMBERS), "r"(n) : "memory");
    } else {
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(sync + PS_MEMBERS) : "memory");
            if (n) break;
            const long long waited = clock64() - t0;
            if (ticket == 0 && waited > PS_JOIN_CYCLES) {
                n = min(atomicOr(sync + PS_JOINED, PS_CLOSED), (uint32_t)expected);
                asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(sync + PS_MEMBERS), "r"(n) : "memory");
                break;
            }
            if (waited > PS_JOIN_CYCLES + limit) {
                atomicExch(dev_err, DEV_ERR_FULL_WAIT);
                return;
            }
        }
    }
    rank = n == (uint32_t)expected ? (int)blockIdx.x : (int)ticket;      // each its own share, where all are there
    members = (int)n;
}

__device__ __forceinline__ void ps_copy16(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void ps_fetch_layer(int l)
{
    if (l < sh.p.num_layers && threadIdx.x < sizeof(PsLayer) / 16)
        ps_copy16(reinterpret_cast<uint4 *>(&sh.layer[l & 1]) + threadIdx.x, reinterpret_cast<const uint4 *>(sh.p.layers + l) + threadIdx.x);
}
// ---------------------------------------------------------------- products

template <int HD, typename KVT>
__device__ __forceinline__ void ps_epilogue(int epi, void *out, int M, int n0, float s0, float s1)
{
    switch (epi) {
        case PS_EPI_ROPE_Q:
        case PS_EPI_ROPE_K: {
            const int h = n0 / HD, j = (n0 % HD) >> 1;
            const float c = sh.cs[0][j], sn = sh.cs[1][j];
            const float o0 = __fsub_rn(__fmul_rn(s0, c), __fmul_rn(s1, sn)), o1 = __fadd_rn(__fmul_rn(s0, sn), __fmul_rn(s1, c));
            if (epi == PS_EPI_ROPE_Q) {
                float *dst = static_cast<float *>(out) + h * HD;
                dst[j] = o0;
                dst[j + HD / 2] = o1;
            } else {
                KVT *dst = static_cast<KVT *>(out) + ((size_t)h * sh.p.max_seq + sh.pos) * HD;
                dst[j] = (KVT)o0;
                dst[j + HD / 2] = (KVT)o1;
            }
            return;
        }
        case PS_EPI_STORE_V: {          // pairs do not cross a head
            KVT *dst = static_cast<KVT *>(out) + ((size_t)(n0 / HD) * sh.p.max_seq + sh.pos) * HD + n0 % HD;
            dst[0] = (KVT)s0;
            dst[1] = (KVT)s1;
            return;
        }
        case PS_EPI_SWIGLU: {
            const float sgm = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-s0)));
            static_cast<float *>(out)[n0 >> 1] = __fmul_rn(__fmul_rn(s0, sgm), s1);
            return;
        }
        default:
            static_cast<float *>(out)[n0] = s0;
            if (n0 + 1 < M) static_cast<float *>(out)[n0 + 1] = s1;
    }
}

// What a phase multiplies: the matrix (this CTA's), where the results go, the input row, and what is fetched ahead of the wait.
struct PsWork {
    const PsSeg *seg;
    int epi;
    void *out;
    const float *src;       // with norm weights: what is added to the residual row first (NULL: nothing); else the input row itself
    const float *gamma;     // norm weights, or NULL
    int fetch;              // layer whose table entry is fetched (-1: none)
};
struct PsGamma { float4 g[2]; };              // norm weights of the block that this warp quantises first, loaded ahead of the wait

// input row -> quantised, in the layout of format T.  After the barrier wait; ends synchronised.
template <class T>
__device__ __forceinline__ void ps_input(const PsWork &w, PsGamma gm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = w.seg->nb, Da = sh.p.Da, D = sh.p.D;
    const int chunks = T::LPS == 1 ? (nb + 7) / 8 : nb;
    uint8_t *stage = ps_stage();
    if (!w.gamma) {
        const float4 *src = reinterpret_cast<const float4 *>(w.src) + 2 * lane;
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        if (warp < chunks) { lo = __ldcg(src + warp * (QK_K / 4)); hi = __ldcg(src + warp * (QK_K / 4) + 1); }
#pragma unroll 1
        for (int b = warp; b < chunks; b += PS_NW) {                   // the next piece is on its way while this one is quantised
            const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            if (b + PS_NW < chunks) { lo = __ldcg(src + (b + PS_NW) * (QK_K / 4)); hi = __ldcg(src + (b + PS_NW) * (QK_K / 4) + 1); }
            T::put(v, b, nb, lane, stage);
        }
        __syncthreads();
        return;
    }
    float *x = ps_x();
    const float4 *delta = reinterpret_cast<const float4 *>(w.src);
    float ss = 0.0f;
#pragma unroll 1
    for (int i0 = threadIdx.x; i0 < Da >> 2; i0 += 2 * PS_THREADS) {
        float4 dv[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = i0 + k * PS_THREADS;
            dv[k] = delta && i < Da >> 2 ? __ldcg(delta + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = i0 + k * PS_THREADS;
            if (i < Da >> 2) {
                float4 v = reinterpret_cast<float4 *>(x)[i];
                v.x += dv[k].x; v.y += dv[k].y; v.z += dv[k].z; v.w += dv[k].w;
                arq_keep_piece(v, i, D, x, ss);
            }
        }
    }
    ss = group_sum<32>(ss);
    if (lane == 0) reinterpret_cast<float *>(sh.red)[warp] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int k = 0; k < PS_NW / 4; ++k) { const float4 r = sh.red[k]; tot += r.x; tot += r.y; tot += r.z; tot += r.w; }
    const float mean = __fmul_rn(tot, sh.inv_d);
    const float rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, sh.p.eps)));
#pragma unroll 1
    for (int b = warp; b < chunks; b += PS_NW) {
        const int e = b * QK_K + 8 * lane;
        float v[8];
        if (b != warp) {
            gm.g[0] = __ldg(reinterpret_cast<const float4 *>(w.gamma + e));
            gm.g[1] = __ldg(reinterpret_cast<const float4 *>(w.gamma + e + 4));
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float4 r = *reinterpret_cast<const float4 *>(x + e + 4 * k), g = gm.g[k];
            v[4 * k] = e + 4 * k < D ? __fmul_rn(__fmul_rn(r.x, rstd), g.x) : 0.0f;
            v[4 * k + 1] = e + 4 * k + 1 < D ? __fmul_rn(__fmul_rn(r.y, rstd), g.y) : 0.0f;
            v[4 * k + 2] = e + 4 * k + 2 < D ? __fmul_rn(__fmul_rn(r.z, rstd), g.z) : 0.0f;
            v[4 * k + 3] = e + 4 * k + 3 < D ? __fmul_rn(__fmul_rn(r.w, rstd), g.w) : 0.0f;
        }
        T::put(v, b, nb, lane, stage);
    }
    __syncthreads();
}

// Where a product's rows lie: logical rows 2 i and 2 i + 1 are the pair of the epilogue: elements j and j + HD / 2 of a head, gate and up of an output, or neighbours.
template <int HD>
struct PsRows {
    const uint8_t *W;
    size_t rb, pair;
    int M, epi;
    __device__ __forceinline__ PsRows(const PsSeg &s, int epi_) : W(s.W), rb((size_t)s.row_bytes), M(s.M), epi(epi_)
    {
        pair = (epi == PS_EPI_SWIGLU ? M >> 1 : (epi <= PS_EPI_ROPE_K ? HD / 2 : 1)) * rb;
    }
    __device__ __forceinline__ bool neighbours() const { return epi == PS_EPI_STORE_V || epi == PS_EPI_STORE; }
    __device__ __forceinline__ const uint8_t *first(int n) const          // n even
    {
        n = min(n, (M - 1) & ~1);
        return W + (size_t)(epi == PS_EPI_SWIGLU ? n >> 1 : (epi <= PS_EPI_ROPE_K ? (n & ~(HD - 1)) | ((n & (HD - 1)) >> 1) : n)) * rb;
    }
    __device__ __forceinline__ const uint8_t *second(const uint8_t *r0, int n) const { return n + 1 < M ? r0 + pair : r0; }
};

// both sums over G adjacent lanes, in the first of them: the halves of the group take one each after the first exchange
template <int G>
__device__ __forceinline__ void ps_pair_sum(float &a0, float &a1, int lane)
{
    const bool up = (lane & (G / 2)) != 0;
    float v = (up ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up ? a0 : a1, G / 2);
#pragma unroll
    for (int w = G / 4; w > 0; w >>= 1) v += __shfl_xor_sync(0xffffffffu, v, w);
    a1 = __shfl_xor_sync(0xffffffffu, v, G / 2);
    a0 = v;
}

// G lanes per row, T::LPS of them per block.  SPLIT = false: a warp walks the passes of its rows, the next ones on their way.
// SPLIT = true: the passes of a row pair go to different warps and meet in shared memory in a fixed order (one round of loads: the latency form).
template <class T, int G, bool SPLIT, int HD, typename KVT>
__device__ __forceinline__ bool ps_run(const PsWork &w, uint32_t target, int share, bool first)
{
    constexpr int SPP = G / T::LPS, SUB = 32 / G, RPW = SUB * PS_R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int li = lane % G, sub = lane / G, u = li % T::LPS, b0 = li / T::LPS;
    const PsSeg &sg = *w.seg;
    const int nb = sg.nb, M = sg.M, epi = w.epi, ncta = sg.ncta, nitems = sg.items, npass = sg.passes;
    const PsRows<HD> rows(sg, epi);
    const int slot = SPLIT ? warp / npass : warp;               // items side by side in a CTA
    int item = SPLIT && slot >= PS_NW / npass ? nitems : share - sg.cta0 + ncta * slot, pass = SPLIT ? warp - slot * npass : 0;
    const uint8_t *x = ps_stage();

    PsGamma gm = {};
    if (w.gamma && warp < (sh.p.Da >> 8)) {
        gm.g[0] = __ldg(reinterpret_cast<const float4 *>(w.gamma + warp * QK_K + 8 * lane));
        gm.g[1] = __ldg(reinterpret_cast<const float4 *>(w.gamma + warp * QK_K + 8 * lane + 4));
    }
    if (w.fetch >= 0) ps_fetch_layer(w.fetch);

    auto finish = [&](int it, float a0, float a1) {
        const int n0 = it * RPW + sub * PS_R;
        ps_pair_sum<G>(a0, a1, lane);
        if (li == 0 && n0 < M) ps_epilogue<HD, KVT>(epi, w.out, M, n0, a0, a1);
    };
    auto meet = [&](float a0, float a1) {                       // SPLIT: the passes of a pair
        ps_pair_sum<G>(a0, a1, lane);
        if (li == 0) { sh.part[warp][2 * sub] = a0; sh.part[warp][2 * sub + 1] = a1; }
        __syncthreads();
        if (item < nitems && pass == 0 && li == 0) {
            float s0 = 0.0f, s1 = 0.0f;
            for (int q = 0; q < npass; ++q) { s0 += sh.part[warp + q][2 * sub]; s1 += sh.part[warp + q][2 * sub + 1]; }
            const int n0 = item * RPW + sub * PS_R;
            if (n0 < M) ps_epilogue<HD, KVT>(epi, w.out, M, n0, s0, s1);
        }
    };

    float a0 = 0.0f, a1 = 0.0f;
    typename T::W w0 = {}, w1 = {};                             // defined on every path: else they would stay alive through all phases
    const uint8_t *r0 = rows.first(item * RPW + sub * PS_R), *r1 = rows.second(r0, item * RPW + sub * PS_R);
    if (item < nitems) {                                        // weights wait for nothing
        const int b = min(b0 + pass * SPP, nb - 1);
        T::load(w0, r0, nb, b, u);
        T::load(w1, r1, nb, b, u);
    }
    PS_TRACE(target / sh.members, 1);
    if (first) {
        if (!ps_wait(target)) return false;
    } else __syncthreads();                                     // the share before this one has been multiplied
    PS_TRACE(target / sh.members, 2);
    ps_input<T>(w, gm);
    PS_TRACE(target / sh.members, 3);
    if constexpr (SPLIT) {                                      // one round (ckb_step_persistent_plan)
        const int b = b0 + pass * SPP;
        if (item < nitems && b < nb) T::pair(w0, w1, x, nb, b, u, a0, a1);
        meet(a0, a1);
    } else {
#pragma unroll 1
        while (item < nitems) {
            int nitem = item, np = pass + 1;
            if (np == npass) {
                np = 0;
                nitem = item + ncta * PS_NW;
                r0 = rows.first(nitem * RPW + sub * PS_R);
                r1 = rows.second(r0, nitem * RPW + sub * PS_R);
            }
            const int b = b0 + pass * SPP, bn = min(b0 + np * SPP, nb - 1);
            if constexpr (T::DEEP) {
                typename T::W n0 = {}, n1 = {};
                if (nitem < nitems) {
                    T::load(n0, r0, nb, bn, u);
                    T::load(n1, r1, nb, bn, u);
                }
                if (b < nb) T::pair(w0, w1, x, nb, b, u, a0, a1);
                w0 = n0;
                w1 = n1;
            } else {
                if (b < nb) T::pair(w0, w1, x, nb, b, u, a0, a1);
                if (nitem < nitems) {
                    T::load(w0, r0, nb, bn, u);
                    T::load(w1, r1, nb, bn, u);
                }
            }
            if (np == 0) {
                finish(item, a0, a1);
                a0 = a1 = 0.0f;
            }
            item = nitem;
            pass = np;
        }
    }
    return true;
}

template <int HD, typename KVT>
__device__ __forceinline__ bool ps_product(const PsWork &w, uint32_t target, int share, bool first)
{
    const PsSeg &s = *w.seg;
    const int sel = s.fmt * 8 + (s.lanes >> 4) * 2 + s.split;             // lanes 8, 16, 32 -> 0, 1, 2
#define PS_CASE(T, F, G, S) case (F) * 8 + ((G) >> 4) * 2 + (S): return ps_run<T, G, S, HD, KVT>(w, target, share, first);
    switch (sel) {
        PS_CASE(PsQ4, PS_FMT_Q4K, 8, false)
        PS_CASE(PsQ4, PS_FMT_Q4K, 16, false)
        PS_CASE(PsQ4, PS_FMT_Q4K, 32, false)
        PS_CASE(PsQ4, PS_FMT_Q4K, 32, true)
        PS_CASE(PsQ6, PS_FMT_Q6K_PLANAR, 16, false)
        PS_CASE(PsQ6, PS_FMT_Q6K_PLANAR, 32, false)
        PS_CASE(PsQ6, PS_FMT_Q6K_PLANAR, 32, true)
        PS_CASE(PsQ5, PS_FMT_Q50_PLANAR, 32, false)
        PS_CASE(PsQ5, PS_FMT_Q50_PLANAR, 32, true)
        default: return false;
    }
#undef PS_CASE
}

// ---------------------------------------------------------------- attention

__device__ __forceinline__ void ps_widen(const uint4 &r, float (&v)[4])
{
    v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y); v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
}
__device__ __forceinline__ void ps_widen(const uint4 &r, float (&v)[8])
{
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ float ps_warp_max(float v)
{
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, w));
    return v;
}
template <int HD, typename KVT> struct PsRow;                  // a lane's HD / 32 elements of a value row
template <> struct PsRow<128, float> { float4 r; __device__ void ld(const float *q) { r = __ldcg(reinterpret_cast<const float4 *>(q)); }
    __device__ void get(float (&v)[4]) const { v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w; } };
template <> struct PsRow<64, float> { float2 r; __device__ void ld(const float *q) { r = __ldcg(reinterpret_cast<const float2 *>(q)); }
    __device__ void get(float (&v)[2]) const { v[0] = r.x; v[1] = r.y; } };
template <> struct PsRow<128, __half> { uint2 r; __device__ void ld(const __half *q) { r = __ldcg(reinterpret_cast<const uint2 *>(q)); }
    __device__ void get(float (&v)[4]) const
    {
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&r.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&r.y));
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    } };
template <> struct PsRow<64, __half> { uint32_t r; __device__ void ld(const __half *q) { r = __ldcg(reinterpret_cast<const uint32_t *>(q)); }
    __device__ void get(float (&v)[2]) const { const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&r)); v[0] = a.x; v[1] = a.y; } };

// Keys of a run: while the context allows it at most 32 runs, so that the merge is one round of loads, of 32 keys at least; beyond that all CTAs of the kv head.
// (Runs of 64 keys and merges of 16 runs: 673 / 1951 us for the two shapes above where this took 656 / 1829.)
__device__ __forceinline__ int ps_run_keys(int T, int per)
{
    const int few = min(256, (T + PS_MERGE - 1) / PS_MERGE), all = (T + per - 1) / per;
    return (max(PS_MIN_RUN, max(few, all)) + PS_KEYS - 1) / PS_KEYS * PS_KEYS;
}

// A warp scores four keys at a time, eight lanes to a key: eight partial sums a lane are transposed over the eight lanes (7 shuffles), so that lane 8 kk + h ends
// with the score of key kk and head h and takes its exponential; the probabilities go through shared memory to the lanes that hold the value rows, HD / 32
// elements each.  (All 32 lanes to a key and the probabilities by shuffle took 61 shuffles a round: 1000 cycles of the SM's shuffle unit.)
template <int HD, typename KVT>
__device__ __forceinline__ bool ps_attention(const PsLayer &ly, uint32_t target, int share, bool first)
{
    constexpr int E = HD / 32, VE = 16 / sizeof(KVT), NJ = HD / (8 * VE);
    const PsParams &p = sh.p;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kk = lane >> 3, ln = lane & 7;
    const int Hkv = p.Hkv, group = p.H / Hkv, T = sh.pos + 1;
    const int g = share % Hkv, s = share / Hkv, run = sh.run, used = sh.used;
    const bool mine = s < used;
    const int k0 = s * run, k1 = min(k0 + run, T);
    const KVT *kc = static_cast<const KVT *>(ly.kc) + (size_t)g * p.max_seq * HD, *vc = static_cast<const KVT *>(ly.vc) + (size_t)g * p.max_seq * HD;
    uint4 kr[NJ] = {};                                         // defined on every path, as in ps_run
    PsRow<HD, KVT> vr[PS_KEYS] = {};
    int base = k0 + warp * PS_KEYS;
    auto load_k = [&](int at) {
        const KVT *row = kc + (size_t)min(at + kk, k1 - 1) * HD + ln * VE;
#pragma unroll
        for (int j = 0; j < NJ; ++j) kr[j] = __ldcg(reinterpret_cast<const uint4 *>(row + j * 8 * VE));
    };
    auto load_v = [&](int at) {
#pragma unroll
        for (int i = 0; i < PS_KEYS; ++i) vr[i].ld(vc + (size_t)min(at + i, k1 - 1) * HD + lane * E);
    };
    const bool early = mine && base < k1 && base + PS_KEYS <= sh.pos;        // rows of earlier steps
    if (early) { load_k(base); load_v(base); }
    PS_TRACE(target / sh.members, 1);
    if (first) {
        if (!ps_wait(target)) return false;
    } else __syncthreads();                                                  // the share before this one is done with the buffers
    PS_TRACE(target / sh.members, 2);
    if (!mine) return true;                                                  // uniform in the CTA
    float *qs = reinterpret_cast<float *>(ps_stage()), *om = qs + PS_MAX_GROUP * HD, *ms = om + PS_NW * PS_MAX_GROUP * HD, *ls = ms + PS_NW * PS_MAX_GROUP;
    const float scale = __fmul_rn(rsqrtf((float)HD), 1.4426950408889634f);
    for (int i = threadIdx.x; i < PS_MAX_GROUP * HD; i += PS_THREADS) qs[i] = i < group * HD ? __ldcg(p.q + (size_t)g * group * HD + i) * scale : 0.0f;
    if (!early && base < k1) { load_k(base); load_v(base); }
    __syncthreads();
    PS_TRACE(target / sh.members, 3);

    float m = -INFINITY, l = 0.0f, o[PS_MAX_GROUP][E];
    float *prob = sh.prob[warp], *fix = prob + PS_KEYS * PS_MAX_GROUP;
#pragma unroll
    for (int h = 0; h < PS_MAX_GROUP; ++h)
#pragma unroll
        for (int e = 0; e < E; ++e) o[h][e] = 0.0f;
#pragma unroll 1
    for (; base < k1; base += PS_NW * PS_KEYS) {
        const int nbase = base + PS_NW * PS_KEYS;
        float v[PS_MAX_GROUP];
#pragma unroll
        for (int h = 0; h < PS_MAX_GROUP; ++h) v[h] = 0.0f;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            float kf[VE];
            ps_widen(kr[j], kf);
#pragma unroll
            for (int h = 0; h < PS_MAX_GROUP; ++h)
                if (h < group) {
#pragma unroll
                    for (int e = 0; e < VE; e += 4) {
                        const float4 q = *reinterpret_cast<const float4 *>(qs + h * HD + j * 8 * VE + ln * VE + e);
                        v[h] = fmaf(q.x, kf[e], v[h]); v[h] = fmaf(q.y, kf[e + 1], v[h]); v[h] = fmaf(q.z, kf[e + 2], v[h]); v[h] = fmaf(q.w, kf[e + 3], v[h]);
                    }
                }
        }
        if (nbase < k1) load_k(nbase);
#pragma unroll
        for (int w = 4; w > 0; w >>= 1) {
            const bool up = (lane & w) != 0;
#pragma unroll
            for (int i = 0; i < w; ++i) {
                const float send = up ? v[i] : v[i + w], keep = up ? v[i + w] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
            }
        }
        const bool valid = base + kk < k1;                                   // lane 8 kk + h: key kk, head h
        const float sc = valid ? v[0] : -INFINITY;
        float top = fmaxf(sc, __shfl_xor_sync(0xffffffffu, sc, 8));
        top = fmaxf(m, fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16)));
        const float corr = m == top ? 1.0f : exp2f(m - top);
        const float pr = valid ? exp2f(sc - top) : 0.0f;
        l = fmaf(l, corr, pr);
        m = top;
        prob[lane] = pr;
        if (kk == 0) fix[ln] = corr;
        __syncwarp();
        if (__any_sync(0xffffffffu, corr != 1.0f)) {
            float f[PS_MAX_GROUP];
            *reinterpret_cast<float4 *>(f) = *reinterpret_cast<const float4 *>(fix);
            *reinterpret_cast<float4 *>(f + 4) = *reinterpret_cast<const float4 *>(fix + 4);
#pragma unroll
            for (int h = 0; h < PS_MAX_GROUP; ++h)
#pragma unroll
                for (int e = 0; e < E; ++e) o[h][e] *= f[h];
        }
#pragma unroll
        for (int i = 0; i < PS_KEYS; ++i) {
            if (base + i < k1) {                         // a clamped row is another key's: its weight is 0, but 0 x inf is not
                float vf[E], f[PS_MAX_GROUP];
                vr[i].get(vf);
                *reinterpret_cast<float4 *>(f) = *reinterpret_cast<const float4 *>(prob + 8 * i);
                *reinterpret_cast<float4 *>(f + 4) = *reinterpret_cast<const float4 *>(prob + 8 * i + 4);
#pragma unroll
                for (int h = 0; h < PS_MAX_GROUP; ++h)
                    if (h < group) {
#pragma unroll
                        for (int e = 0; e < E; ++e) o[h][e] = fmaf(f[h], vf[e], o[h][e]);
                    }
            }
        }
        __syncwarp();
        if (nbase < k1) load_v(nbase);
    }
    PS_TRACE(target / sh.members, 5);
    l += __shfl_xor_sync(0xffffffffu, l, 8);
    l += __shfl_xor_sync(0xffffffffu, l, 16);
    if (lane < PS_MAX_GROUP) {
        ms[lane * PS_NW + warp] = m;
        ls[lane * PS_NW + warp] = l;
    }
#pragma unroll
    for (int h = 0; h < PS_MAX_GROUP; ++h)
        if (h < group) {
#pragma unroll
            for (int e = 0; e < E; ++e) om[(warp * PS_MAX_GROUP + h) * HD + lane * E + e] = o[h][e];
        }
    __syncthreads();
    // warps of the CTA -> its run's result.  A warp's 32 outputs are of one head: it weighs the partial results for itself, without another barrier.
    float *part = p.part + ((size_t)s * Hkv + g) * PS_MAX_GROUP * (HD + 2);          // [heads][HD], then [heads] of (maximum, sum)
#pragma unroll 1
    for (int i = threadIdx.x; i < group * HD; i += PS_THREADS) {
        const int h = i / HD, e = i % HD;
        const float mk = lane < PS_NW ? ms[h * PS_NW + lane] : -INFINITY, top = ps_warp_max(mk);
        const float f = mk == -INFINITY ? 0.0f : exp2f(mk - top), sum = group_sum<32>(lane < PS_NW ? f * ls[h * PS_NW + lane] : 0.0f);
        float a = 0.0f;
#pragma unroll
        for (int k = 0; k < PS_NW; ++k) a = fmaf(__shfl_sync(0xffffffffu, f, k), om[(k * PS_MAX_GROUP + h) * HD + e], a);
        if (used == 1) p.att[(size_t)g * group * HD + i] = __fdiv_rn(a, sum);
        else {
            part[i] = a;
            if (e == 0) *reinterpret_cast<float2 *>(part + PS_MAX_GROUP * HD + 2 * h) = make_float2(top, sum);
        }
    }
    if (used == 1) return true;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned old;
        asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;" : "=r"(old) : "l"(p.sync + PS_HEADS + g), "r"((unsigned)(used - 1)) : "memory");
        sh.last = old == (unsigned)(used - 1);
    }
    __syncthreads();
    PS_TRACE(target / sh.members, 7);
    if (!sh.last) return true;
    // the last CTA of the kv head: a batch of runs at a time, their values on the way while the warp makes their weights, a lane per run
    const size_t stride = (size_t)Hkv * PS_MAX_GROUP * (HD + 2);
    const float *all = p.part + (size_t)g * PS_MAX_GROUP * (HD + 2);
#pragma unroll 1
    for (int i = threadIdx.x; i < group * HD; i += PS_THREADS) {
        const int h = i / HD;
        float a = 0.0f, top = -INFINITY, sum = 0.0f;
#pragma unroll 1
        for (int j = 0; j < used; j += PS_MERGE) {
            const int n = min(PS_MERGE, used - j);
            const float *at = all + (size_t)j * stride;
            const float2 ml = lane < n ? __ldcg(reinterpret_cast<const float2 *>(at + lane * stride + PS_MAX_GROUP * HD + 2 * h)) : make_float2(-INFINITY, 0.0f);
            float v[PS_MERGE];
#pragma unroll
            for (int k = 0; k < PS_MERGE; ++k) v[k] = k < n ? __ldcg(at + k * stride + i) : 0.0f;
            const float now = fmaxf(top, ps_warp_max(ml.x));
            const float f = top == now ? 1.0f : exp2f(top - now), e = lane < n ? exp2f(ml.x - now) : 0.0f;
            sum = fmaf(sum, f, group_sum<32>(e * ml.y));
            a *= f;
#pragma unroll
            for (int k = 0; k < PS_MERGE; ++k) a = fmaf(__shfl_sync(0xffffffffu, e, k), v[k], a);
            top = now;
        }
        p.att[(size_t)g * group * HD + i] = __fdiv_rn(a, sum);
    }
    return true;
}

// ---------------------------------------------------------------- the step

// All phases of one CTA's shares: its own, or (MANY) every members-th from its own on.  An instantiation of each: with the loop over shares in the way the ordinary
// case took 3 % longer (Qwen2-0.5B shape: 549 us for 533).
template <int HD, typename KVT, bool MANY>
__device__ __forceinline__ void ps_walk(const PsParams &p, int rank, int members)
{
    const int steps = 5 * p.num_layers;
    bool alive = true;
    auto qkv = [&](const PsLayer &ly, int share) { return share >= ly.seg[PS_V].cta0 ? PS_V : (share >= ly.seg[PS_K].cta0 ? PS_K : PS_Q); };
    auto qkv_epi = [](int which) { return which == PS_Q ? PS_EPI_ROPE_Q : (which == PS_K ? PS_EPI_ROPE_K : PS_EPI_STORE_V); };
    // one product in the code for all phases: five times the instructions would not stay in the caches
#pragma unroll 1
    for (int k = 0; k <= steps; ++k) {
        PS_TRACE(k, 0);
        const int l = k / 5, phase = k - 5 * l;
        const PsLayer &ly = sh.layer[l & 1];
        const uint32_t target = (uint32_t)k * members + (k ? p.extra_arrivals : 0);
#pragma unroll 1
        for (int share = rank; share < (MANY ? p.ctas : rank + 1) && alive; share += members) {
            const bool first = !MANY || share == rank;
            if (phase == 1 && k != steps) {
                alive = ps_attention<HD, KVT>(ly, target, share, first);
                continue;
            }
            PsWork w;
            w.gamma = nullptr;
            w.fetch = -1;
            w.epi = PS_EPI_STORE;
            // what is added to the residual row is added once
            if (k == steps) {
                w.seg = &p.head; w.out = p.logits; w.src = l && first ? p.prev : nullptr; w.gamma = p.final_gamma;
            } else if (phase == 0) {
                const int which = qkv(ly, share);
                w.seg = &ly.seg[which]; w.src = l && first ? p.prev : nullptr; w.gamma = ly.ln1; w.fetch = first ? l + 1 : -1;
                w.epi = qkv_epi(which);
                w.out = which == PS_Q ? (void *)p.q : (which == PS_K ? ly.kc : ly.vc);
            } else if (phase == 2) {
                w.seg = &ly.seg[PS_O]; w.out = p.o; w.src = p.att;
            } else if (phase == 3) {
                w.seg = &ly.seg[PS_W1]; w.epi = PS_EPI_SWIGLU; w.out = p.mf; w.src = first ? p.o : nullptr; w.gamma = ly.ln2;
            } else {
                w.seg = &ly.seg[PS_W2]; w.out = p.prev; w.src = p.mf;
            }
            alive = ps_product<HD, KVT>(w, target, share, first);
        }
        PS_TRACE(k, 4);
        if (!alive || k == steps) break;
        ps_arrive();
    }
}

// a function of its own, so that it takes no registers from the ordinary form
template <int HD, typename KVT>
__device__ __noinline__ void ps_walk_shares(const PsParams *p, int rank, int members) { ps_walk<HD, KVT, true>(*p, rank, members); }

template <int HD, typename KVT>
__global__ void __launch_bounds__(PS_THREADS, 1) step_persistent_kernel(const __grid_constant__ PsParams p, const long long limit, int *__restrict__ dev_err)
{
    const int pos = __ldcg(p.pos);
    if (threadIdx.x == 0) {
        sh.p = p;
        sh.limit = limit;
        sh.dev_err = dev_err;
        sh.inv_d = __fdiv_rn(1.0f, (float)p.D);
        sh.pos = pos;
        sh.dead = 0;
        sh.run = ps_run_keys(pos + 1, p.ctas / p.Hkv);
        sh.used = (pos + sh.run) / sh.run;
        ps_enrol(p.sync, p.ctas, limit, dev_err, sh.rank, sh.members);
    }
    for (int i = threadIdx.x; i < p.Da; i += PS_THREADS) ps_x()[i] = __ldcg(p.x + i);
    for (int i = threadIdx.x; i < HD / 2; i += PS_THREADS) {
        sh.cs[0][i] = __ldg(p.cos_cache + (size_t)pos * (HD / 2) + i);
        sh.cs[1][i] = __ldg(p.sin_cache + (size_t)pos * (HD / 2) + i);
    }
    __syncthreads();
    const int rank = sh.rank, members = sh.members;
    if (rank >= 0) {
        ps_fetch_layer(0);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (members == p.ctas) ps_walk<HD, KVT, false>(p, rank, members);
        else ps_walk_shares<HD, KVT>(&p, rank, members);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned old;
        asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;" : "=r"(old) : "l"(p.sync + PS_LEFT), "r"(gridDim.x - 1) : "memory");
        if (old == gridDim.x - 1) {                                  // nobody waits any more
            p.sync[PS_ARRIVALS] = p.sync[PS_JOINED] = p.sync[PS_MEMBERS] = 0;
            for (int g = 0; g < p.Hkv; ++g) p.sync[PS_HEADS + g] = 0;      // zero already, unless a wait ran out
            *p.pos = pos + 1;
        }
    }
}

template <int HD, typename KVT>
static int ps_prepare(size_t smem)
{
    auto kernel = step_persistent_kernel<HD, KVT>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PS_MAX_SMEM) != cudaSuccess) { cudaGetLastError(); return 0; }
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, PS_THREADS, smem) != cudaSuccess) { cudaGetLastError(); return 0; }
    return occ >= 1;
}

template <int HD, typename KVT>
static int ps_launch(const PsParams *p, cudaStream_t st)
{
    PsParams q = *p;
    q.extra_arrivals = ckb_tune_get("step_extra_arrivals", 0);       // test aid: every barrier waits for arrivals that nobody makes
    const int missing = ckb_tune_get("step_missing_ctas", 0);        // test aid: CTAs that the step counts on and that never start
    if (int rc = launch_plain("step_persistent", step_persistent_kernel<HD, KVT>, dim3(missing > 0 && missing < p->ctas ? p->ctas - missing : p->ctas), dim3(PS_THREADS), p->smem, st, q,
                              ckb_wait_limit_cycles(), ckb_device_error_word()))
        return rc;
    return 0;
}

}  // namespace ckb

using namespace ckb;

#ifdef CKB_STEP_TRACE
extern "C" int ckb200_step_trace(long long *out) { return (int)cudaMemcpyFromSymbol(out, ps_trace, sizeof ps_trace); }      // 256 x 512 x 8
#endif

extern "C" size_t ckb_step_persistent_stage_bytes(int fmt, int nb)
{
    return fmt == PS_FMT_Q4K ? (size_t)q4p_smem_bytes(nb) : (size_t)ringx_smem_bytes(fmt == PS_FMT_Q6K_PLANAR ? FMT_Q6K : FMT_Q50, nb);
}

extern "C" size_t ckb_step_persistent_smem(int Da, size_t stage, int head_dim, int kv_f16)
{
    const size_t attn = (size_t)(PS_MAX_GROUP * head_dim + PS_NW * PS_MAX_GROUP * (head_dim + 2)) * sizeof(float);
    const size_t smem = (size_t)Da * 4 + (stage > attn ? stage : attn);
    if (smem > PS_MAX_SMEM || ckb_sm_count() > PS_MAX_CTAS) return 0;
    const int fits = head_dim == 128 ? (kv_f16 ? ps_prepare<128, __half>(smem) : ps_prepare<128, float>(smem))
                                     : (head_dim == 64 ? (kv_f16 ? ps_prepare<64, __half>(smem) : ps_prepare<64, float>(smem)) : 0);
    return fits ? smem : 0;
}

extern "C" size_t ckb_step_persistent_scratch_bytes(int head_dim) { return (size_t)PS_MAX_CTAS * PS_MAX_GROUP * (head_dim + 2) * sizeof(float); }
extern "C" size_t ckb_step_persistent_sync_bytes(void) { return (PS_HEADS + PS_MAX_CTAS) * sizeof(unsigned); }

// Lanes per row: as many as the row has units, 8 (Q4_K) or 16 (Q6_K) at least.  Rows of several passes are split over the warps of a CTA when all
// pieces of the matrix fit its CTAs' warps at once: every warp then has one round of loads instead of a walk.
extern "C" void ckb_step_persistent_plan(PsSeg *s)
{
    const int lps = s->fmt == PS_FMT_Q4K ? 2 : (s->fmt == PS_FMT_Q6K_PLANAR ? 4 : 1);
    s->row_bytes = (int)(s->fmt == PS_FMT_Q4K ? PsQ4::row_bytes(s->nb) : (s->fmt == PS_FMT_Q6K_PLANAR ? PsQ6::row_bytes(s->nb) : PsQ5::row_bytes(s->nb)));
    int g = s->fmt == PS_FMT_Q4K ? 8 : (s->fmt == PS_FMT_Q6K_PLANAR ? 16 : 32);
    while (g < 32 && g < lps * s->nb) g <<= 1;
    s->lanes = g;
    const int spp = g / lps, rows = (32 / g) * PS_R;
    s->passes = (s->nb + spp - 1) / spp;
    s->items = (s->M + rows - 1) / rows;
    s->split = g == 32 && s->passes > 1 && s->passes <= PS_NW && (long long)s->items <= (long long)s->ncta * (PS_NW / s->passes);
}

extern "C" int ckb_launch_step_persistent(const PsParams *p, void *stream)
{
    cudaStream_t st = ckb_stream(stream);
    if (p->head_dim == 128) return p->kv_f16 ? ps_launch<128, __half>(p, st) : ps_launch<128, float>(p, st);
    return p->kv_f16 ? ps_launch<64, __half>(p, st) : ps_launch<64, float>(p, st);
}
