// batched.cu -- many cgemm3m problems of uneven shape and mixed op() in one
// persistent launch (the batching form).
//
// Reference hooks for batched 3M: LaunchCgemm3mOnchipBatches /
// LaunchCgemm3mUnitBatches (blas/gemm/arch35/cgemm_host.cpp:749-782,
// gemm_host_common.h:84-97), used by aclblasCgemm3mStridedBatched
// (cann_ops_blas.h:652).  The reference batches equal shapes only; this form
// takes a heterogeneous list, and like the reference's on-chip batch kernel
// (cgemm_onchip_kernel.h:84 ProducePanel) it deinterleaves inside the GEMM
// instead of through a workspace.
//
// Design.  One persistent kernel (grid = SM count x resident blocks) pulls
// tasks from a device list through an atomic counter; a task is (problem,
// output tile, K partition), and the list is sorted by decreasing work so the
// schedule ends on small tasks.  A task copies op(A) and op(B) element by
// element from the caller's interleaved complex matrices into shared memory
// (8-byte cp.async, zero past the edges, transposed on the way when the matrix
// runs along K), runs the 3M FFMA micro-kernel of the drop-in (one thread per
// output, K in increasing order, fmaf into P0, P1, P2 from +0), and either
// applies alpha/beta and stores, or writes its partition's (Re, Im) partials
// and counts in on a per-tile counter; the last partition to arrive merges all
// partitions in partition order with the merge arithmetic of the drop-in and
// stores.  No block ever waits on another.  Each output is thus a fixed
// function of the inputs and its K split, bit-identical to the drop-in called
// with the same k_partitions.
//
// The micro-kernel works on the interleaved elements as they are: one packed
// FMA multiplies (xr, xi) by (yr, yi) into (P0, P1), a second one two rows'
// sums (xr + xi) by (yr + yi) into P2, and the sums are formed in registers.
// No planes are written to shared memory, the operands of the packed FMAs need
// no moves, and an element costs one 8-byte shared load for three products: at
// 8 x 4 outputs per thread 96 bytes per 96 FMAs, which balances shared-memory
// wavefronts and the FMA pipe.  The loop by itself took 141 cycles a warp and K
// term for 48 packed FMAs and the sums (50 TFLOP/s; what a register file would
// give that serves a packed FMA's three pairs in 2 cycles when one is reused
// from the instruction before and in 3 when not, which no counter shows
// directly), 42-43 TFLOP/s with the copies and epilogues; with planes converted
// into shared memory 31-36.  Over 512 unequal problems the FMA pipe is 60 %
// active, math-pipe throttle the first stall, shared memory at 61 % of its
// wavefronts.  Blocks of 128 threads, three per SM, hide each other's barriers,
// prologues and epilogues.  64 problems of 256 x 192 x 320: 313 -> 185 us in one
// partition, 224 in the two their chain limit asks for; 512 unequal problems
// 2190 -> 1700 us.
//
// Tile (64x64, 128x32, 32x128, 64x32, 32x32) and K split are chosen per problem
// from a policy table; the autotuner times every candidate policy on the device
// with the caller's A and B and a scratch C, keeps the fastest and caches it
// per batch signature (device, ops, shapes).  Execute may replay a captured
// CUDA graph holding the counter reset and the one kernel.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <type_traits>
#include <vector>

#include "cg3m_internal.h"
#include "epilogue.cuh"
#include "ptx.cuh"

namespace cg3m {
namespace {

constexpr int kThreads = 128;  // of the persistent kernels
constexpr int BK = 16;
// K terms unrolled in the FFMA loop.  64 problems of 256 x 192 x 320 in one
// strided launch, one partition: 4 terms 207 us, 8 187, 16 185.  The heterogeneous kernel holds
// five tile shapes' loops and misses the instruction cache at 16: 512 unequal
// problems 4 terms 1766 us, 8 1700, 16 1721.
constexpr int kUnroll = 16, kUnrollMixed = 8;

// Product modes: the standard 3M identity (P0 = Ar.Br, P1 = Ai.Bi,
// P2 = (Ar+Ai).(Br+Bi); Re = P0 - P1, Im = (P2 - P0) - P1) or four real
// products (Re = Ar.Br - Ai.Bi, Im = Ar.Bi + Ai.Br).
constexpr int kMode3M = 0;
constexpr int kMode4M = 1;

struct BProblem {
    int ta, tb, m, n, k;  // k = 0: beta-scale only (k == 0 or alpha == 0)
    EpiParams epi;
    const float2* A;
    const float2* B;
    float2* C;
    int lda, ldb, ldc;
    int tile;    // index into the tile shapes below
    int repair;  // recompute non-finite products with explicit FP32 four-product terms
    int parts, span, tiles_m, tiles_n, ppitch;
    size_t partial_off;  // floats into the partial arena
    size_t counter_off;  // words into the tile counters
};

struct BTask {
    int problem, tile, part, pad;
};

// Tile shapes (BM x BN): 0: 128x64, 1: 64x64, 2: 128x32, 3: 32x128, 4: 64x32, 5: 32x32.
// Tile 0 takes 256 threads in the one-launch kernel (three products only); in
// the persistent kernels a task of tile 0 is two 64x64 tiles, one after the
// other.
constexpr int kTileCount = 6;
__host__ __device__ constexpr int tile_bm(int t)
{
    return (t == 0 || t == 2) ? 128 : (t == 1 || t == 4) ? 64 : 32;
}
__host__ __device__ constexpr int tile_bn(int t)
{
    return t == 3 ? 128 : (t == 0 || t == 1) ? 64 : 32;
}

template <int BM, int BN, int MODE>
struct Cfg {
    static constexpr int AREA = BM * BN;
    static constexpr int MT = AREA >= 4096 ? 8 : 4;                 // outputs per thread along m
    static constexpr int NT = AREA >= 2048 ? 4 : 2;                 // and along n
    static constexpr int TM = BM / MT, TN = BN / NT;                // threads along m, n
    static constexpr int THREADS = TM * TN;
    static constexpr int WX = TM < 8 ? TM : 8, WY = 32 / WX;        // a warp's threads along m, n
    static constexpr int PA = BM + 1, PB = BN + 1;                  // pitch of one K term's elements
    static constexpr int STAGE = BK * (PA + PB);                    // elements of one K-block
    static constexpr int ACC2 = MODE == kMode3M ? MT / 2 : MT;      // packed accumulators besides (P0, P1)
};

// Shared memory: a ring of K-blocks, element (row r, K term kk) of op(A) at
// kk * PA + r, of op(B) after it at kk * PB + r.  The odd pitch spreads the K
// terms a half-warp writes over all banks when the matrix runs along K.
constexpr int kStages = 3;
constexpr size_t kSmemBytes = (size_t)kStages * BK * (128 + 32 + 2) * sizeof(float2);  // the largest 128-thread tile

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 8-byte asynchronous copy global -> shared; src_bytes = 0 writes zeros
// (the source is then not read).
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, int src_bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// One operand's share of a K-block for this thread.  The source's contiguous
// dimension goes to consecutive threads: rows (ROWS: op(A) in {N, R}, op(B) in
// {T, C}; element (row0 + r, k) at X[(row0 + r) + k*ld]) or K (all BK terms of
// a row by 16 consecutive threads; X[k + (row0 + r)*ld]).
template <int R, int THREADS, bool ROWS>
struct Feed {
    static constexpr int PASS = THREADS / (ROWS ? R : BK);  // K terms (rows) one pass of the block covers
    static constexpr int E = R * BK / THREADS;
    static_assert(THREADS % (ROWS ? R : BK) == 0 && R * BK % THREADS == 0, "whole elements per thread");
    static __device__ __forceinline__ int r0() { return ROWS ? threadIdx.x % R : threadIdx.x / BK; }
    static __device__ __forceinline__ int k0() { return ROWS ? threadIdx.x / R : threadIdx.x % BK; }
    // this thread's first element of the tile's first K-block
    static __device__ __forceinline__ const float2* first(const float2* X, int ld, int row0, int kbeg)
    {
        return ROWS ? X + (row0 + r0()) + (long long)(kbeg + k0()) * ld
                    : X + (kbeg + k0()) + (long long)(row0 + r0()) * ld;
    }
    // Issue the copies of the K-block whose first element is src: `rows` valid
    // rows and `kleft` K terms left; everything past them reads as zero (X, the
    // matrix, is then the source of a zero-byte copy).
    static __device__ __forceinline__ void issue(const float2* X, const float2* src, int ld, int rows, int kleft,
                                                 float2* stage)
    {
        const uint32_t dst = smem_u32(stage + k0() * (R + 1) + r0());
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const bool ok = (ROWS ? r0() : r0() + q * PASS) < rows && (ROWS ? k0() + q * PASS : k0()) < kleft;
            cp_async8(dst + (uint32_t)(q * PASS * (ROWS ? R + 1 : 1)) * 8u,
                      ok ? (const void*)(src + (long long)(q * PASS) * ld) : (const void*)X, ok ? 8 : 0);
        }
    }
};

// The copies of one K-block of both operands, and the step to the next.
template <int BM, int BN, int THREADS>
struct Feeds {
    const float2 *sa, *sb;  // this thread's first element of the next K-block
    __device__ __forceinline__ void start(const BProblem& p, int m0, int n0, int kbeg, bool na, bool nb)
    {
        sa = na ? Feed<BM, THREADS, true>::first(p.A, p.lda, m0, kbeg)
                : Feed<BM, THREADS, false>::first(p.A, p.lda, m0, kbeg);
        sb = nb ? Feed<BN, THREADS, false>::first(p.B, p.ldb, n0, kbeg)
                : Feed<BN, THREADS, true>::first(p.B, p.ldb, n0, kbeg);
    }
    __device__ __forceinline__ void issue(const BProblem& p, int m0, int n0, int kleft, bool na, bool nb,
                                          float2* stage)
    {
        if (na) {
            Feed<BM, THREADS, true>::issue(p.A, sa, p.lda, p.m - m0, kleft, stage);
            sa += (long long)BK * p.lda;
        } else {
            Feed<BM, THREADS, false>::issue(p.A, sa, p.lda, p.m - m0, kleft, stage);
            sa += BK;
        }
        stage += BK * (BM + 1);
        if (nb) {
            Feed<BN, THREADS, false>::issue(p.B, sb, p.ldb, p.n - n0, kleft, stage);
            sb += BK;
        } else {
            Feed<BN, THREADS, true>::issue(p.B, sb, p.ldb, p.n - n0, kleft, stage);
            sb += (long long)BK * p.ldb;
        }
    }
};

// C = beta*C for k == 0 or alpha == 0 (beta == 0: zeros, C not read).
__device__ __forceinline__ float2 beta_scaled(const EpiParams& e, const float2* cp)
{
    if (e.beta_zero) {
        return make_float2(0.0f, 0.0f);
    }
    const float2 c = *cp;
    return make_float2(__fsub_rn(__fmul_rn(e.br, c.x), __fmul_rn(e.bi, c.y)),
                       __fadd_rn(__fmul_rn(e.br, c.y), __fmul_rn(e.bi, c.x)));
}

// Non-finite repair of one output (repair_four_product, epilogue.cuh), out of
// line: rare, and inlined once per output it would dwarf the kernels.
__device__ __noinline__ float2 repair_call(const float2* A, int lda, int ta, const float2* B, int ldb, int tb, int k,
                                           int row, int col)
{
    return repair_four_product(A, lda, ta, B, ldb, tb, k, row, col);
}
__device__ __forceinline__ float2 repair_product(const BProblem& p, int row, int col)
{
    return repair_call(p.A, p.lda, p.ta, p.B, p.ldb, p.tb, p.k, row, col);
}

// Partition product (before alpha/beta) of the accumulators of one output.
template <int MODE>
__device__ __forceinline__ float2 part_product(float q0, float q1, float q2, float q3)
{
    if constexpr (MODE == kMode3M) {
        return make_float2(__fsub_rn(q0, q1), __fsub_rn(__fsub_rn(q2, q0), q1));
    } else {
        return make_float2(__fsub_rn(q0, q1), __fadd_rn(q2, q3));
    }
}

__device__ __forceinline__ bool finite2(float2 v) { return isfinite(v.x) && isfinite(v.y); }

// This thread's place in the tile: its outputs are rows tx + TM i, columns
// ty + TN j.  A half-warp's 8-byte loads cover at most 8 consecutive rows and
// 4 columns, so each is one shared-memory wavefront.
template <int BM, int BN, int MODE>
__device__ __forceinline__ int2 thread_xy()
{
    using G = Cfg<BM, BN, MODE>;
    constexpr int WM = G::TM / G::WX;  // warps along m
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    return make_int2((warp % WM) * G::WX + lane % G::WX, (warp / WM) * G::WY + lane / G::WX);
}

// Packed pairs as 64-bit registers.
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// Accumulators.  p[i][j] holds output (i, j)'s (P0, P1) = (sum xr yr, sum xi yi).
// Three products: q[ii][j] holds P2 of outputs (2 ii, j) and (2 ii + 1, j); four
// products: q[i][j] holds (sum xr yi, sum xi yr).  Every packed FMA
// (__ffma2_rn) is two independent round-to-nearest FP32 FMAs, so each sum is
// still one FMA chain in increasing K.
template <int BM, int BN, int MODE>
struct Acc {
    uint64_t p[Cfg<BM, BN, MODE>::MT][Cfg<BM, BN, MODE>::NT];
    uint64_t q[Cfg<BM, BN, MODE>::ACC2][Cfg<BM, BN, MODE>::NT];
};

// Partition product of output (i, j) of this thread.
template <int BM, int BN, int MODE>
__device__ __forceinline__ float2 acc_product(const Acc<BM, BN, MODE>& acc, int i, int j)
{
    const float2 p = unpack2(acc.p[i][j]);
    if constexpr (MODE == kMode3M) {
        const float2 q = unpack2(acc.q[i >> 1][j]);
        return part_product<MODE>(p.x, p.y, (i & 1) ? q.y : q.x, 0.0f);
    } else {
        const float2 q = unpack2(acc.q[i][j]);
        return part_product<MODE>(p.x, p.y, q.x, q.y);
    }
}

// One staged K-block, BK terms in increasing K: a at the block's first term and
// this thread's first row, b at its first column.  Conjugated operands (sa, sb
// = -1) without touching x: y's imaginary part carries sa sb, so xi (sa sb yi)
// is the product of the signed parts, and the sums are xr + sa xi and
// yr + sa (sa sb yi), each one rounding.  Four products sign each operand.
template <int BM, int BN, int MODE, bool CONJ, int UNROLL>
__device__ __forceinline__ void k_block(const float2* a, const float2* b, float sa, float sb, Acc<BM, BN, MODE>& acc)
{
    using G = Cfg<BM, BN, MODE>;
#pragma unroll UNROLL
    for (int kk = 0; kk < BK; ++kk) {
        uint64_t x[G::MT], y[G::NT];
#pragma unroll
        for (int i = 0; i < G::MT; ++i) {
            x[i] = *reinterpret_cast<const uint64_t*>(a + kk * G::PA + i * G::TM);
        }
#pragma unroll
        for (int j = 0; j < G::NT; ++j) {
            y[j] = *reinterpret_cast<const uint64_t*>(b + kk * G::PB + j * G::TN);
            if constexpr (CONJ) {
                y[j] = mul2(y[j], pack2(1.0f, MODE == kMode3M ? sa * sb : sb));
            }
        }
        if constexpr (MODE == kMode3M) {
#pragma unroll
            for (int j = 0; j < G::NT; ++j) {
#pragma unroll
                for (int i = 0; i < G::MT; ++i) {
                    acc.p[i][j] = ffma2(x[i], y[j], acc.p[i][j]);
                }
            }
            uint64_t xs[G::MT / 2];
#pragma unroll
            for (int i = 0; i < G::MT / 2; ++i) {
                const float2 u = unpack2(x[2 * i]), v = unpack2(x[2 * i + 1]);
                xs[i] = CONJ ? pack2(__fmaf_rn(u.y, sa, u.x), __fmaf_rn(v.y, sa, v.x))
                             : pack2(__fadd_rn(u.x, u.y), __fadd_rn(v.x, v.y));
            }
#pragma unroll
            for (int j = 0; j < G::NT; ++j) {
                const float2 u = unpack2(y[j]);
                const float s = CONJ ? __fmaf_rn(u.y, sa, u.x) : __fadd_rn(u.x, u.y);
                const uint64_t ys = pack2(s, s);
#pragma unroll
                for (int i = 0; i < G::MT / 2; ++i) {
                    acc.q[i][j] = ffma2(xs[i], ys, acc.q[i][j]);
                }
            }
        } else {
            if constexpr (CONJ) {
#pragma unroll
                for (int i = 0; i < G::MT; ++i) {
                    x[i] = mul2(x[i], pack2(1.0f, sa));
                }
            }
#pragma unroll
            for (int j = 0; j < G::NT; ++j) {
                const float2 u = unpack2(y[j]);
                const uint64_t swapped = pack2(u.y, u.x);
#pragma unroll
                for (int i = 0; i < G::MT; ++i) {
                    acc.p[i][j] = ffma2(x[i], y[j], acc.p[i][j]);
                    acc.q[i][j] = ffma2(x[i], swapped, acc.q[i][j]);
                }
            }
        }
    }
}

// This thread's outputs of the tile at (m0, n0): repair, alpha/beta, store.
// C is read a column's worth at a time before anything of it is stored.
template <int BM, int BN, int MODE>
__device__ __forceinline__ void store_tile(const BProblem& p, int m0, int n0, int2 t, const Acc<BM, BN, MODE>& acc)
{
    using G = Cfg<BM, BN, MODE>;
    const bool reads_c = !p.epi.unit && !p.epi.beta_zero;
#pragma unroll
    for (int j = 0; j < G::NT; ++j) {
        const int col = n0 + t.y + G::TN * j;
        if (col >= p.n) {
            break;
        }
        float2* cp = p.C + (size_t)col * p.ldc + m0 + t.x;
        float2 old[G::MT];
#pragma unroll
        for (int i = 0; i < G::MT; ++i) {
            old[i] = reads_c && m0 + t.x + G::TM * i < p.m ? cp[G::TM * i] : make_float2(0.0f, 0.0f);
        }
#pragma unroll
        for (int i = 0; i < G::MT; ++i) {
            const int row = m0 + t.x + G::TM * i;
            if (row < p.m) {
                float2 v = acc_product<BM, BN, MODE>(acc, i, j);
                if (p.repair && !finite2(v)) {
                    v = repair_product(p, row, col);
                }
                cp[G::TM * i] = epilogue_with(v.x, v.y, p.epi, old[i]);
            }
        }
    }
}

// The products of K terms [kbeg, kbeg + klen) of the BM x BN tile at (m0, n0),
// accumulated from zero into acc, through a ring of STAGES K-blocks.  Every
// thread is past its last shared-memory read when the next barrier completes.
template <int BM, int BN, int MODE, int STAGES, int UNROLL>
__device__ __forceinline__ void accumulate(const BProblem& p, int m0, int n0, int kbeg, int klen, float2* ring,
                                           Acc<BM, BN, MODE>& acc)
{
    using G = Cfg<BM, BN, MODE>;
    const int nk = (klen + BK - 1) / BK;
    const int2 t = thread_xy<BM, BN, MODE>();
    const bool na = p.ta == CG3M_OP_N || p.ta == CG3M_OP_R;
    const bool nb = p.tb == CG3M_OP_N || p.tb == CG3M_OP_R;
    const bool ca = p.ta == CG3M_OP_C || p.ta == CG3M_OP_R;
    const bool cb = p.tb == CG3M_OP_C || p.tb == CG3M_OP_R;
    const float sa = ca ? -1.0f : 1.0f, sb = cb ? -1.0f : 1.0f;
    const bool conj = MODE == kMode3M ? ca != cb || ca : ca || cb;
    Feeds<BM, BN, G::THREADS> feeds;
    feeds.start(p, m0, n0, kbeg, na, nb);
#pragma unroll
    for (int j = 0; j < G::NT; ++j) {
#pragma unroll
        for (int i = 0; i < G::MT; ++i) {
            acc.p[i][j] = 0;
        }
#pragma unroll
        for (int i = 0; i < G::ACC2; ++i) {
            acc.q[i][j] = 0;
        }
    }
    // Prologue: K-blocks 0 .. STAGES-2 in flight (one commit group each, empty
    // groups past the end keep the counting uniform).
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < nk) {
            feeds.issue(p, m0, n0, klen - s * BK, na, nb, ring + s * G::STAGE);
        }
        cp_async_commit();
    }
    int slot = 0, refill = STAGES - 1;
    for (int kb = 0; kb < nk; ++kb) {
        cp_async_wait<STAGES - 2>();  // this thread's copies of K-block kb have landed
        // Everyone's have, and everyone is done with K-block kb - 1, whose
        // stage takes K-block kb + STAGES - 1.
        __syncthreads();
        const int nxt = kb + STAGES - 1;
        if (nxt < nk) {
            feeds.issue(p, m0, n0, klen - nxt * BK, na, nb, ring + refill * G::STAGE);
        }
        cp_async_commit();
        const float2* stage = ring + slot * G::STAGE;
        if (conj) {
            k_block<BM, BN, MODE, true, UNROLL>(stage + t.x, stage + BK * G::PA + t.y, sa, sb, acc);
        } else {
            k_block<BM, BN, MODE, false, UNROLL>(stage + t.x, stage + BK * G::PA + t.y, 1.0f, 1.0f, acc);
        }
        slot = slot + 1 == STAGES ? 0 : slot + 1;
        refill = refill + 1 == STAGES ? 0 : refill + 1;
    }
    cp_async_wait<0>();  // only empty groups can remain; keep the count at zero between tasks
}

template <int BM, int BN, int MODE, int UNROLL>
__device__ __forceinline__ void run_task(const BProblem& p, int m0, int n0, int tile, int part, float2* ring,
                                         float* partials, uint32_t* counters, int* last_flag)
{
    using G = Cfg<BM, BN, MODE>;
    const int kbeg = part * p.span;
    const int kend = min(p.k, kbeg + p.span);
    const int klen = kend > kbeg ? kend - kbeg : 0;
    const int2 t = thread_xy<BM, BN, MODE>();
    Acc<BM, BN, MODE> acc;
    accumulate<BM, BN, MODE, kStages, UNROLL>(p, m0, n0, kbeg, klen, ring, acc);

    if (p.parts == 1) {
        if (p.k == 0) {
            for (int e = threadIdx.x; e < BM * BN; e += G::THREADS) {
                const int row = m0 + e % BM, col = n0 + e / BM;
                if (row < p.m && col < p.n) {
                    float2* cp = p.C + (size_t)col * p.ldc + row;
                    *cp = beta_scaled(p.epi, cp);
                }
            }
        } else {
            store_tile<BM, BN, MODE>(p, m0, n0, t, acc);
        }
        return;
    }

    // K split: store this partition's (Re, Im), count in; the last to arrive merges.
    float* base = partials + p.partial_off;
    const size_t plane = (size_t)p.ppitch * p.n;
#pragma unroll
    for (int j = 0; j < G::NT; ++j) {
        const int col = n0 + t.y + G::TN * j;
#pragma unroll
        for (int i = 0; i < G::MT; ++i) {
            const int row = m0 + t.x + G::TM * i;
            if (row < p.m && col < p.n) {
                const size_t o = (size_t)col * p.ppitch + row;
                const float2 v = acc_product<BM, BN, MODE>(acc, i, j);
                __stcg(base + (size_t)(2 * part) * plane + o, v.x);
                __stcg(base + (size_t)(2 * part + 1) * plane + o, v.y);
            }
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t* ctr = counters + p.counter_off + tile;
        const uint32_t prev = atomicAdd(ctr, 1u);
        const int last = prev == (uint32_t)(p.parts - 1);
        if (last) {
            *ctr = 0;  // ready for the next execution of the plan
        }
        *last_flag = last;
    }
    __syncthreads();
    if (!*last_flag) {
        return;
    }
    __threadfence();
    // Three outputs per step (the most that fits the kernel's registers) so
    // the loads of one partition for all three are in flight together; each
    // output still adds its partitions in order.
    constexpr int U = 3;
    for (int e0 = threadIdx.x; e0 < BM * BN; e0 += U * kThreads) {
        size_t o[U];
        bool ok[U];
        float re[U], im[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = e0 + u * kThreads;
            const int row = m0 + e % BM, col = n0 + e / BM;
            ok[u] = e < BM * BN && row < p.m && col < p.n;
            o[u] = ok[u] ? (size_t)col * p.ppitch + row : 0;
            re[u] = ok[u] ? __ldcg(base + o[u]) : 0.0f;
            im[u] = ok[u] ? __ldcg(base + plane + o[u]) : 0.0f;
        }
        for (int q = 1; q < p.parts; ++q) {
            float tr[U], ti[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                tr[u] = ok[u] ? __ldcg(base + (size_t)(2 * q) * plane + o[u]) : 0.0f;
                ti[u] = ok[u] ? __ldcg(base + (size_t)(2 * q + 1) * plane + o[u]) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                re[u] = __fadd_rn(re[u], tr[u]);
                im[u] = __fadd_rn(im[u], ti[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (ok[u]) {
                const int e = e0 + u * kThreads;
                const int row = m0 + e % BM, col = n0 + e / BM;
                float2 v = make_float2(re[u], im[u]);
                if (p.repair && !finite2(v)) {
                    v = repair_product(p, row, col);
                }
                float2* cp = p.C + (size_t)col * p.ldc + row;
                *cp = epilogue_value(v.x, v.y, p.epi, cp);
            }
        }
    }
}

// One task of the tile shape: tile 0 walks its 64x64 tiles (unsplit along K, so
// without counters), the others are one tile.
template <int TILE, int MODE, int UNROLL>
__device__ __forceinline__ void tile_task(const BProblem& p, int tile, int part, float2* ring, float* partials,
                                          uint32_t* counters, int* last_flag)
{
    constexpr int BM = TILE == 0 ? 64 : tile_bm(TILE), BN = tile_bn(TILE);
    const int m0 = (tile % p.tiles_m) * tile_bm(TILE), n0 = (tile / p.tiles_m) * BN;
    for (int m = m0; m < min(p.m, m0 + tile_bm(TILE)); m += BM) {
        if (TILE == 0 && m != m0) {
            __syncthreads();  // the previous tile's shared-memory reads are done
        }
        run_task<BM, BN, MODE, UNROLL>(p, m, n0, tile, part, ring, partials, counters, last_flag);
    }
}

// Out of line in the heterogeneous kernel, so that each tile shape's loop gets
// the registers to itself; the strided kernel is instantiated per tile (all
// shapes inlined side by side spilled: 200 us instead of 185 on 64 problems of
// 256 x 192 x 320).
template <int TILE>
__device__ __noinline__ void tile_task_call(const BProblem& p, int tile, int part, float2* ring, float* partials,
                                            uint32_t* counters, int* last_flag)
{
    tile_task<TILE, kMode3M, kUnrollMixed>(p, tile, part, ring, partials, counters, last_flag);
}

// Heterogeneous batch: tasks from a device list (problem, tile, partition).
__global__ void __launch_bounds__(kThreads, 3) batched_kernel(const BProblem* __restrict__ problems,
                                                              const BTask* __restrict__ tasks, int ntasks,
                                                              int* __restrict__ next, float* partials,
                                                              uint32_t* counters)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* ring = reinterpret_cast<float2*>(smem_raw);
    __shared__ int task_id;
    __shared__ int last_flag;
    __shared__ BProblem cur;  // the task's problem: its fields are read where they are used
    static_assert(sizeof(BProblem) % 4 == 0 && sizeof(BProblem) / 4 <= kThreads, "one word per thread");
    // A block's first task is its own (gridDim.x <= ntasks): blocks are placed one
    // on every SM before any takes a second, so the longest tasks, first in the
    // list, start on SMs of their own.  Drawn from the counter, as the later ones
    // are, they met on one SM by chance: 11 problems 74 -> 133 us.
    for (int t = blockIdx.x; t < ntasks; t = task_id) {
        const BTask tk = tasks[t];
        if (threadIdx.x < sizeof(BProblem) / 4) {
            reinterpret_cast<uint32_t*>(&cur)[threadIdx.x] =
                reinterpret_cast<const uint32_t*>(problems + tk.problem)[threadIdx.x];
        }
        __syncthreads();
        switch (cur.tile) {
            case 1: tile_task_call<1>(cur, tk.tile, tk.part, ring, partials, counters, &last_flag); break;
            case 2: tile_task_call<2>(cur, tk.tile, tk.part, ring, partials, counters, &last_flag); break;
            case 3: tile_task_call<3>(cur, tk.tile, tk.part, ring, partials, counters, &last_flag); break;
            case 4: tile_task_call<4>(cur, tk.tile, tk.part, ring, partials, counters, &last_flag); break;
            default: tile_task_call<5>(cur, tk.tile, tk.part, ring, partials, counters, &last_flag); break;
        }
        __syncthreads();  // the task's shared-memory reads are done
        if (threadIdx.x == 0) {
            task_id = (int)gridDim.x + atomicAdd(next, 1);
        }
        __syncthreads();
    }
}

// Strided batch (and single problems): batch b's problem is `proto` with
// A + b*sA, B + b*sB, C + b*sC and its own partial / counter ranges; task t
// is (b, tile, part) = (t / per_batch, (t % per_batch) / parts, t % parts).
// counters[0] is the task counter; tile counters follow.
// Geometry of the strided kernel's tile (tile 0 walks 64 x 64 tiles).
template <int MODE, int TILE>
using StridedCfg = Cfg<TILE == 0 ? 64 : tile_bm(TILE), tile_bn(TILE), MODE>;
// Blocks per SM the registers allow: 96 accumulators a thread leave room for
// three, the four-product mode's 128 for two.
template <int MODE, int TILE>
constexpr int kStridedBlocks = StridedCfg<MODE, TILE>::AREA >= 4096   ? (MODE == kMode3M ? 3 : 2)
                               : StridedCfg<MODE, TILE>::AREA >= 2048 ? 4
                                                                      : 5;
template <int MODE, int TILE>
constexpr size_t kStridedSmem = (size_t)kStages * StridedCfg<MODE, TILE>::STAGE * sizeof(float2);

template <int MODE, int TILE>
__global__ void __launch_bounds__(kThreads, (kStridedBlocks<MODE, TILE>))
    strided_kernel(const __grid_constant__ BProblem proto, long long sA, long long sB, long long sC, int batch,
                   size_t partial_stride, float* partials, uint32_t* counters)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* ring = reinterpret_cast<float2*>(smem_raw);
    __shared__ int task_id;
    __shared__ int last_flag;
    __shared__ BProblem cur;  // the task's problem: its fields are read where they are used
    const int tiles = proto.tiles_m * proto.tiles_n;
    const int per_batch = tiles * proto.parts;
    const long long ntasks = (long long)per_batch * batch;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            task_id = (int)atomicAdd(counters, 1u);
        }
        __syncthreads();
        const int t = task_id;
        if (t >= ntasks) {
            return;
        }
        const int b = t / per_batch, r = t - b * per_batch;
        if (threadIdx.x == 0) {
            cur = proto;
            cur.A = proto.A + (long long)b * sA;
            cur.B = proto.B + (long long)b * sB;
            cur.C = proto.C + (long long)b * sC;
            cur.partial_off = (size_t)b * partial_stride;
            cur.counter_off = 1 + (size_t)b * tiles;
        }
        __syncthreads();
        tile_task<TILE, MODE, kUnroll>(cur, r / proto.parts, r % proto.parts, ring, partials, counters, &last_flag);
    }
}

// ---- one problem, one launch: K partitions merged through the cluster -------
//
// Block (tile, part) of grid (tiles, parts) computes partition `part` of output
// tile `tile` with the same K loop as the persistent kernels; the partitions
// of a tile form one thread-block cluster (cluster dims 1 x parts).  Each block
// leaves its partition's (Re, Im) in its own shared memory; after a cluster
// barrier, block q merges the q-th slice of the tile's outputs, reading every
// partition's value through distributed shared memory and adding them in
// partition order with the merge arithmetic of the drop-in, then applies
// alpha/beta and stores.  A second cluster barrier keeps every block's shared
// memory in place until all reads are done.  Nothing goes through global
// memory but A, B and C: no workspace, no counters, no second launch.  Both
// barriers are reached by every thread of every block (no early exits).
// Shared memory of an SM, and what each block takes besides its own.
constexpr size_t kSmSmem = 228 * 1024, kBlockSmem = 1024;
template <int BM, int BN, int MODE>
struct SingleCfg {
    using G = Cfg<BM, BN, MODE>;
    // blocks per SM the registers allow (65536 / threads / registers of the micro-kernel)
    static constexpr int BLOCKS = G::THREADS == 256 ? 1 : G::AREA >= 4096 ? (MODE == kMode3M ? 3 : 2)
                                                      : G::AREA >= 2048   ? 4
                                                                          : 5;
    // Four stages, or three where only those leave room for BLOCKS blocks on an
    // SM (128 x 32 and 32 x 128, three products: 1.06 times as fast as four
    // stages and two blocks over 70 shapes, 0.9 to 1.3).
    static constexpr size_t stage_bytes = (size_t)G::STAGE * sizeof(float2);
    static constexpr int STAGES = BLOCKS * (4 * stage_bytes + kBlockSmem) <= kSmSmem ? 4 : 3;
    static constexpr size_t SMEM = STAGES * stage_bytes;
    static_assert(BLOCKS * (SMEM + kBlockSmem) <= kSmSmem, "the blocks that registers allow fit shared memory");
    static_assert((size_t)2 * BM * BN * sizeof(float) <= SMEM, "partials exceed the ring");
};

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

constexpr int kMaxClusterParts = 8;  // portable cluster size
// Outputs whose remote partials a thread loads together in the cluster merge:
// a thread merges up to 32 / parts outputs, each a round trip to the other
// blocks' shared memory.  Graph replay of 1208 x 23 x 25 in two partitions: one
// at a time 4.00 us, two 3.64, four 4.08 (registers); of 256^3: 6.98, 6.75, 7.71.
constexpr int kMergeAhead = 2;

template <int BM, int BN, int MODE>
__global__ void __launch_bounds__(Cfg<BM, BN, MODE>::THREADS, SingleCfg<BM, BN, MODE>::BLOCKS)
    single_kernel(const BProblem p)
{
    using G = Cfg<BM, BN, MODE>;
    using S = SingleCfg<BM, BN, MODE>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* ring = reinterpret_cast<float2*>(smem_raw);
    const int tile = blockIdx.x, part = blockIdx.y;
    const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
    const int m0 = tm * BM, n0 = tn * BN;
    const int kbeg = part * p.span;
    const int kend = min(p.k, kbeg + p.span);
    const int klen = kend > kbeg ? kend - kbeg : 0;
    const int2 t = thread_xy<BM, BN, MODE>();
    Acc<BM, BN, MODE> acc;
    accumulate<BM, BN, MODE, S::STAGES, kUnroll>(p, m0, n0, kbeg, klen, ring, acc);

    if (p.parts == 1) {
        store_tile<BM, BN, MODE>(p, m0, n0, t, acc);
        return;
    }

    // This partition's (Re, Im) at part_re[e], part_im[e], e = c*BM + r (tile
    // coordinates), over the ring: every copy has landed, and the barrier puts
    // every thread past its last read.
    __syncthreads();
    float* part_re = reinterpret_cast<float*>(ring);
    float* part_im = part_re + BM * BN;
#pragma unroll
    for (int j = 0; j < G::NT; ++j) {
        const int c = t.y + G::TN * j;
#pragma unroll
        for (int i = 0; i < G::MT; ++i) {
            const int r = t.x + G::TM * i;
            const float2 v = acc_product<BM, BN, MODE>(acc, i, j);
            part_re[c * BM + r] = v.x;
            part_im[c * BM + r] = v.y;
        }
    }
    const uint32_t re_local = static_cast<uint32_t>(__cvta_generic_to_shared(part_re));
    const uint32_t im_local = static_cast<uint32_t>(__cvta_generic_to_shared(part_im));
    const int per = (BM * BN + p.parts - 1) / p.parts;  // outputs merged by each block
    const int begin = part * per + (int)threadIdx.x, e_end = min(BM * BN, (part + 1) * per);
    const bool reads_c = !p.epi.unit && !p.epi.beta_zero;
    float2 old[kMergeAhead] = {};
    auto load_c = [&](int first) {
#pragma unroll
        for (int u = 0; u < kMergeAhead; ++u) {
            const int e = first + u * G::THREADS, row = m0 + e % BM, col = n0 + e / BM;
            old[u] = e < e_end && row < p.m && col < p.n ? p.C[(size_t)col * p.ldc + row]
                                                                     : make_float2(0.0f, 0.0f);
        }
    };
    if (reads_c) {
        load_c(begin);
    }   // C on the way while the cluster meets
    cluster_sync();  // every partition's values are in place and visible to the cluster
    // kMergeAhead outputs' remote loads are in flight together.
    for (int first = begin; first < e_end; first += kMergeAhead * G::THREADS) {
        if (reads_c && first != begin) {
            load_c(first);
        }
        float tr[kMergeAhead][kMaxClusterParts], ti[kMergeAhead][kMaxClusterParts];
#pragma unroll
        for (int u = 0; u < kMergeAhead; ++u) {
            const int e = first + u * G::THREADS;
#pragma unroll
            for (int q = 0; q < kMaxClusterParts; ++q) {
                if (q < p.parts && e < e_end) {
                    tr[u][q] = ld_cluster_f32(mapa_shared(re_local + 4u * e, q));
                    ti[u][q] = ld_cluster_f32(mapa_shared(im_local + 4u * e, q));
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kMergeAhead; ++u) {
            const int e = first + u * G::THREADS;
            const int row = m0 + e % BM, col = n0 + e / BM;
            if (e >= e_end || row >= p.m || col >= p.n) {
                continue;
            }
            float re = tr[u][0], im = ti[u][0];
#pragma unroll
            for (int q = 1; q < kMaxClusterParts; ++q) {
                if (q < p.parts) {
                    re = __fadd_rn(re, tr[u][q]);
                    im = __fadd_rn(im, ti[u][q]);
                }
            }
            float2 v = make_float2(re, im);
            if (p.repair && !finite2(v)) {
                v = repair_product(p, row, col);
            }
            p.C[(size_t)col * p.ldc + row] = epilogue_with(v.x, v.y, p.epi, old[u]);
        }
    }
    cluster_sync();  // no block leaves while others may still read its shared memory
}

template <int MODE>
cudaError_t launch_single_tile(cudaStream_t s, const BProblem& bp, int tile)
{
    auto run = [&](auto kernel, int threads, size_t smem) -> cudaError_t {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) {
            return e;
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(bp.tiles_m * bp.tiles_n), (unsigned)bp.parts, 1);
        cfg.blockDim = dim3((unsigned)threads, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = (unsigned)bp.parts;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, kernel, bp);
    };
    auto launch_tile = [&](auto bm, auto bn) -> cudaError_t {
        constexpr int BM = decltype(bm)::value, BN = decltype(bn)::value;
        return run(single_kernel<BM, BN, MODE>, Cfg<BM, BN, MODE>::THREADS, SingleCfg<BM, BN, MODE>::SMEM);
    };
    using std::integral_constant;
    switch (tile) {
        case 0:
            if constexpr (MODE == kMode3M) {
                return launch_tile(integral_constant<int, 128>{}, integral_constant<int, 64>{});
            }
            return cudaErrorInvalidValue;
        case 1: return launch_tile(integral_constant<int, 64>{}, integral_constant<int, 64>{});
        case 2: return launch_tile(integral_constant<int, 128>{}, integral_constant<int, 32>{});
        case 3: return launch_tile(integral_constant<int, 32>{}, integral_constant<int, 128>{});
        case 4: return launch_tile(integral_constant<int, 64>{}, integral_constant<int, 32>{});
        default: return launch_tile(integral_constant<int, 32>{}, integral_constant<int, 32>{});
    }
}

}  // namespace
}  // namespace cg3m

using namespace cg3m;

struct cg3mBatchPlan {
    int device = -1;
    int count = 0;
    int sm_count = 148;
    int blocks_per_sm = 1;
    std::vector<int> index;  // caller's problem i -> host[] position, -1 for quick returns
    std::vector<BProblem> host;
    std::vector<BTask> tasks;
    BProblem* d_problems = nullptr;
    BTask* d_tasks = nullptr;
    float* d_partials = nullptr;
    uint32_t* d_counters = nullptr;
    int* d_next = nullptr;
    cudaStream_t capture_stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    ~cg3mBatchPlan()
    {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (capture_stream) cudaStreamDestroy(capture_stream);
        cudaFree(d_problems);
        cudaFree(d_tasks);
        cudaFree(d_partials);
        cudaFree(d_counters);
        cudaFree(d_next);
    }
};

namespace {

// One candidate table: the largest tile area allowed and the cap on K
// partitions.  Each problem takes the allowed tile with the least estimated
// time -- padded work (tiles x BM x BN x (k + 16)) over the tile's relative
// FFMA efficiency -- and is split along K as far as BatchChains asks: where a
// large tile's task would exceed a quarter of the batch's average work per SM
// (the longest task bounds the persistent schedule), keeping >= 128 K terms per
// partition, whatever the tile.
struct Policy {
    int max_area;
    int split_cap;
};

constexpr Policy kPolicies[] = {{4096, 1}, {4096, 2}, {4096, 4}, {4096, 8}, {2048, 1},
                                {2048, 4}, {2048, 8}, {1024, 1}, {1024, 4}, {1024, 8}};

// Relative FFMA efficiency of each tile shape (per output-element-term), from
// the per-term cost of blocks sharing an SM (kSingleCost below): the narrower
// tiles load more shared memory per FMA.
constexpr double kTileEfficiency[kTileCount] = {1.0, 1.0, 0.93, 0.88, 0.87, 0.75};

int span_for(int k, int parts) { return ceil_div(ceil_div(k, 16), parts) * 16; }

// The allowed tile with the least estimated time for p (padded work over
// efficiency).
void choose_tile(BProblem& p, int max_area)
{
    int best = kTileCount - 1;
    double best_cost = 1e300;
    for (int t = 1; t < kTileCount; ++t) {
        if (tile_bm(t) * tile_bn(t) > max_area) {
            continue;
        }
        const double work =
            (double)ceil_div(p.m, tile_bm(t)) * ceil_div(p.n, tile_bn(t)) * tile_bm(t) * tile_bn(t) * (p.k + 16);
        const double cost = work / kTileEfficiency[t];
        if (cost < best_cost) {
            best_cost = cost;
            best = t;
        }
    }
    p.tile = best;
    p.tiles_m = ceil_div(p.m, tile_bm(best));
    p.tiles_n = ceil_div(p.n, tile_bn(best));
}

void apply_policy(std::vector<BProblem>& ps, const Policy& pol, int sm_count)
{
    BatchChains chains(kMode3M, sm_count);
    for (const auto& p : ps) {
        chains.add(p.m, p.n, p.k, 1);
    }
    for (auto& p : ps) {
        choose_tile(p, pol.max_area);
        p.parts = chains.parts(p.m, p.n, p.k, pol.split_cap);
        p.span = p.parts > 1 ? span_for(p.k, p.parts) : p.k;
    }
}

// Lays out partials and counters, and lists the tasks by decreasing work.
void build_tasks(std::vector<BProblem>& ps, std::vector<BTask>& tasks, size_t* partial_floats,
                 size_t* counter_words)
{
    std::vector<std::pair<double, BTask>> v;
    size_t pf = 0, cw = 0;
    for (size_t i = 0; i < ps.size(); ++i) {
        BProblem& p = ps[i];
        p.ppitch = (int)align_up((size_t)p.m, 32);
        p.partial_off = pf;
        p.counter_off = cw;
        if (p.parts > 1) {
            pf += (size_t)p.ppitch * p.n * 2 * p.parts;
            cw += (size_t)p.tiles_m * p.tiles_n;
        }
        const double cost =
            (double)tile_bm(p.tile) * tile_bn(p.tile) * ((p.parts > 1 ? p.span : p.k) + 16) / kTileEfficiency[p.tile];
        for (int t = 0; t < p.tiles_m * p.tiles_n; ++t) {
            for (int q = 0; q < p.parts; ++q) {
                v.push_back({cost, BTask{(int)i, t, q, 0}});
            }
        }
    }
    std::stable_sort(v.begin(), v.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
    tasks.clear();
    tasks.reserve(v.size());
    for (auto& x : v) {
        tasks.push_back(x.second);
    }
    *partial_floats = pf;
    *counter_words = cw;
}

void release_device(cg3mBatchPlan* plan)
{
    if (plan->exec) {
        cudaGraphExecDestroy(plan->exec);
        plan->exec = nullptr;
    }
    if (plan->graph) {
        cudaGraphDestroy(plan->graph);
        plan->graph = nullptr;
    }
    cudaFree(plan->d_problems);
    cudaFree(plan->d_tasks);
    cudaFree(plan->d_partials);
    cudaFree(plan->d_counters);
    plan->d_problems = nullptr;
    plan->d_tasks = nullptr;
    plan->d_partials = nullptr;
    plan->d_counters = nullptr;
}

// (Re)builds the task list of `ps` under `pol` and uploads it with zeroed
// tile counters.
cudaError_t materialise(cg3mBatchPlan* plan, std::vector<BProblem>& ps, const Policy& pol)
{
    release_device(plan);
    apply_policy(ps, pol, plan->sm_count);
    size_t pf = 0, cw = 0;
    build_tasks(ps, plan->tasks, &pf, &cw);
    cudaError_t e = cudaMalloc(&plan->d_problems, sizeof(BProblem) * std::max<size_t>(1, ps.size()));
    if (e == cudaSuccess) e = cudaMalloc(&plan->d_tasks, sizeof(BTask) * std::max<size_t>(1, plan->tasks.size()));
    if (e == cudaSuccess) e = cudaMalloc(&plan->d_partials, sizeof(float) * std::max<size_t>(1, pf));
    if (e == cudaSuccess) e = cudaMalloc(&plan->d_counters, sizeof(uint32_t) * std::max<size_t>(1, cw));
    if (e == cudaSuccess && plan->d_next == nullptr) e = cudaMalloc(&plan->d_next, sizeof(int));
    if (e == cudaSuccess && !ps.empty())
        e = cudaMemcpy(plan->d_problems, ps.data(), sizeof(BProblem) * ps.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !plan->tasks.empty())
        e = cudaMemcpy(plan->d_tasks, plan->tasks.data(), sizeof(BTask) * plan->tasks.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(plan->d_counters, 0, sizeof(uint32_t) * std::max<size_t>(1, cw));
    // Pageable uploads may still be in flight on the legacy stream when
    // cudaMemcpy returns; the plan's launches go to other streams.
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    return e;
}

cudaError_t launch(cg3mBatchPlan* plan, cudaStream_t s)
{
    if (plan->tasks.empty()) {
        return cudaSuccess;
    }
    cudaError_t e = cudaMemsetAsync(plan->d_next, 0, sizeof(int), s);
    if (e != cudaSuccess) {
        return e;
    }
    const int grid = (int)std::min<size_t>(plan->tasks.size(), (size_t)plan->sm_count * plan->blocks_per_sm);
    batched_kernel<<<grid, kThreads, kSmemBytes, s>>>(plan->d_problems, plan->d_tasks, (int)plan->tasks.size(),
                                                      plan->d_next, plan->d_partials, plan->d_counters);
    return cudaGetLastError();
}

std::mutex g_tune_mutex;
std::map<std::string, Policy> g_tuned;  // batch signature -> chosen policy

std::string signature(int device, const std::vector<BProblem>& ps)
{
    std::string s = std::to_string(device) + ":";
    s.reserve(ps.size() * 24);
    char b[80];
    for (const auto& p : ps) {
        std::snprintf(b, sizeof b, "%d%d,%d,%d,%d,%d;", p.ta, p.tb, p.m, p.n, p.k, p.epi.beta_zero);
        s += b;
    }
    return s;
}

// Times every candidate policy (median of 3 launches after one warm-up) with
// the caller's A and B and a scratch C, and returns the fastest.  The
// caller's C is never written.  `untuned` where nothing can be timed.
Policy autotune(cg3mBatchPlan* plan, cudaStream_t s, const Policy& untuned)
{
    size_t celems = 0;
    for (const auto& p : plan->host) {
        celems += (size_t)p.ldc * p.n;
    }
    float2* scratch = nullptr;
    if (cudaMalloc(&scratch, sizeof(float2) * std::max<size_t>(1, celems)) != cudaSuccess) {
        cudaGetLastError();
        return untuned;
    }
    cudaMemsetAsync(scratch, 0, sizeof(float2) * std::max<size_t>(1, celems), s);
    std::vector<BProblem> trial = plan->host;
    size_t off = 0;
    for (auto& p : trial) {
        p.C = scratch + off;
        off += (size_t)p.ldc * p.n;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    Policy best = untuned;
    float best_ms = 1e30f;
    for (const Policy& pol : kPolicies) {
        if (materialise(plan, trial, pol) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        float times[3] = {0, 0, 0};
        bool ok = true;
        for (int r = 0; r < 4 && ok; ++r) {
            ok = cudaEventRecord(e0, s) == cudaSuccess && launch(plan, s) == cudaSuccess &&
                 cudaEventRecord(e1, s) == cudaSuccess && cudaEventSynchronize(e1) == cudaSuccess;
            if (ok && r > 0) {
                cudaEventElapsedTime(&times[r - 1], e0, e1);
            }
        }
        if (!ok) {
            cudaGetLastError();
            continue;
        }
        std::sort(times, times + 3);
        if (times[1] < best_ms) {
            best_ms = times[1];
            best = pol;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaStreamSynchronize(s);
    cudaFree(scratch);
    return best;
}

}  // namespace

namespace cg3m {

int single_tile_bm(int tile) { return tile_bm(tile); }
int single_tile_bn(int tile) { return tile_bn(tile); }

// Time model of the one-launch kernel (three-product mode), in microseconds,
// fitted on B200 to 2500 timed (shape, tile, partitions) launches (median
// error 2-4 % per tile then, 3-8 % since the merge loads two outputs at a time,
// the small tiles' launches being the faster; what the planner picks costs a
// mean 1.1 % over the best within the chain limit, 210 shapes).  Clusters of `parts` blocks run in waves of as many
// clusters as fit at once; a wave costs a fixed part and span x the per-term
// time a block needs by itself.  Blocks that share an SM add a per-term cost
// for every layer of clusters: one layer holds as many as fit with one block
// per SM, which is fewer than sm_count / parts (GPC boundaries), so a split
// of 7 or 8 starts its second layer at 105 or 120 blocks.  Beyond kShortChain
// terms the layers are those that the clusters need at several blocks per SM.
namespace {
struct SingleCost {
    double base_us, fixed_us, term_ns, shared_term_ns, merge_us;
};
constexpr SingleCost kSingleCost[kTileCount] = {{3.396, 3.006, 0.0, 167.65, 0.031},  {6.203, 0.0, 25.64, 70.90, 0.0},
                                                {4.231, 2.119, 18.57, 76.50, 0.0},   {3.417, 2.711, 16.39, 80.99, 0.135},
                                                {3.483, 0.0, 17.18, 40.77, 0.131},   {1.719, 0.927, 13.61, 23.63, 0.150}};
// Blocks per SM of each tile, three and four products (tile 0: three only).
template <int MODE>
constexpr int single_occ(int t)
{
    constexpr int occ[kTileCount] = {SingleCfg<128, 64, kMode3M>::BLOCKS, SingleCfg<64, 64, MODE>::BLOCKS,
                                     SingleCfg<128, 32, MODE>::BLOCKS,    SingleCfg<32, 128, MODE>::BLOCKS,
                                     SingleCfg<64, 32, MODE>::BLOCKS,     SingleCfg<32, 32, MODE>::BLOCKS};
    return occ[t];
}
int single_occ(int mode, int t) { return mode == kMode4M ? single_occ<kMode4M>(t) : single_occ<kMode3M>(t); }
}  // namespace

// The policy of a batch that is not timed: four partitions at most, and the
// tiles with the least bound on the schedule, the longest task on an SM of its
// own plus an SM's share of the work (the model above).  A few problems need
// small tiles to reach every SM; with 64 x 64 wherever they fit, 80 batches of 1
// to 48 problems took 1.9 times as long (2 problems 68 us, now 40).
static Policy untuned_policy(const std::vector<BProblem>& ps, int sm_count)
{
    Policy best{};
    double least = 1e300;
    for (const int area : {4096, 2048, 1024}) {
        const Policy pol{area, 4};
        std::vector<BProblem> trial = ps;
        apply_policy(trial, pol, sm_count);
        double longest = 0.0, total = 0.0;
        for (const auto& p : trial) {
            const SingleCost& c = kSingleCost[p.tile];
            const double terms = 1e-3 * (p.parts > 1 ? p.span : p.k);
            longest = std::max(longest, c.fixed_us + terms * (c.term_ns + c.shared_term_ns));
            total += (double)p.tiles_m * p.tiles_n * p.parts * (c.fixed_us + terms * c.shared_term_ns);
        }
        const double us = longest + total / std::max(sm_count, 1);
        if (us < least) {
            least = us;
            best = pol;
        }
    }
    return best;
}

// A K split in the strided kernel: its last block's merge, and per output of a
// task the partials written and read.
constexpr double kSplitLaunchUs = 3.0, kSplitUsPerOutput = 0.6e-3;

namespace {

// Floats of one problem's partials.
size_t strided_partials(const Problem& p, int parts)
{
    return parts > 1 ? align_up((size_t)p.m, 32) * p.n * 2 * parts : 0;
}

// Where the partials start: after the task counter and the tile counters.
size_t strided_partial_off(int batch, int tiles) { return align_up((1 + (size_t)batch * tiles) * sizeof(uint32_t), 256); }

}  // namespace

bool make_strided_plan(const Problem& p, int mode, int batch, int sm_count, StridedPlan* out)
{
    if (batch <= 0 || p.m <= 0 || p.n <= 0 || p.k <= 0 || (mode != kMode3M && mode != kMode4M)) {
        return false;
    }
    BatchChains chains(mode, sm_count);
    chains.add(p.m, p.n, p.k, batch);
    const int parts = chains.parts(p.m, p.n, p.k, 4);
    // 32 x 32 tiles have the most counters
    const size_t bytes = strided_partial_off(batch, ceil_div(p.m, 32) * ceil_div(p.n, 32)) +
                         (size_t)batch * strided_partials(p, parts) * sizeof(float);
    return make_strided_plan(p, mode, batch, sm_count, parts > 1 ? span_for(p.k, parts) : p.k,
                             std::max(kPlanWorkspace, bytes), out);
}

bool make_strided_plan(const Problem& p, int mode, int batch, int sm_count, int max_span, size_t max_bytes,
                       StridedPlan* out)
{
    if (batch <= 0 || p.m <= 0 || p.n <= 0 || p.k <= 0 || (mode != kMode3M && mode != kMode4M)) {
        return false;
    }
    // The tile and K split with the least estimated time: the one-launch
    // kernel's model (kSingleCost) without clusters -- a task is a block of its
    // own -- plus the partials a split leaves in L2 and its last block merges.
    BProblem bp{};
    bp.m = p.m;
    bp.n = p.n;
    bp.k = p.k;
    const long long sms = std::max(sm_count, 1);
    const int most = std::max(8, ceil_div(p.k, std::max(max_span / 16 * 16, 16)));
    double best = 1e300;
    for (int t = 1; t < kTileCount; ++t) {
        const int tm = ceil_div(p.m, tile_bm(t)), tn = ceil_div(p.n, tile_bn(t));
        const int occ = single_occ(mode, t);
        const SingleCost& c = kSingleCost[t];
        for (int q = 1; q <= most; ++q) {
            const int span = q == 1 ? p.k : span_for(p.k, q);
            const int coarser = q > 2 ? span_for(p.k, q - 1) : p.k;
            if (span > max_span || (q > 1 && ((span < 48 && coarser <= max_span) || (q - 1) * span >= p.k))) {
                continue;
            }
            if (q > 1 && strided_partial_off(batch, tm * tn) + (size_t)batch * strided_partials(p, q) * sizeof(float) >
                             max_bytes) {
                continue;
            }
            const long long tasks = (long long)tm * tn * batch * q;
            const long long waves = (tasks + sms * occ - 1) / (sms * occ), load = (tasks + sms - 1) / sms;
            const double fma = (mode == kMode4M ? 4.0 / 3.0 : 1.0) * (load > 1 ? 1.07 : 1.0);
            double us = c.base_us + (double)waves * c.fixed_us +
                        span * 1e-3 * fma * ((double)waves * c.term_ns + (double)load * c.shared_term_ns);
            if (q > 1) {
                us += kSplitLaunchUs + (double)load * tile_bm(t) * tile_bn(t) * kSplitUsPerOutput;
            }
            if (us < best) {
                best = us;
                bp.tile = t;
                bp.tiles_m = tm;
                bp.tiles_n = tn;
                bp.parts = q;
                bp.span = span;
            }
        }
    }
    if (best == 1e300) {
        return false;
    }
    // Two tiles per task once every block has many of them: half the trips to
    // the task counter, and the pair shares op(B)'s columns.
    const long long rounds =
        (long long)bp.tiles_m * bp.tiles_n * batch / (3LL * std::max(sm_count, 1));
    if (mode == kMode3M && bp.tile == 1 && bp.parts == 1 && rounds >= 16) {
        bp.tile = 0;
        bp.tiles_m = ceil_div(p.m, tile_bm(0));
    }
    StridedPlan pl{};
    pl.tile = bp.tile;
    pl.tile_m = tile_bm(bp.tile);
    pl.tile_n = tile_bn(bp.tile);
    pl.est_us = best;
    pl.parts = bp.parts;
    pl.span = bp.span;
    pl.tiles = bp.tiles_m * bp.tiles_n;
    pl.ppitch = (int)align_up((size_t)p.m, 32);
    pl.partial_stride = bp.parts > 1 ? (size_t)pl.ppitch * p.n * 2 * bp.parts : 0;
    pl.counters = 1 + (size_t)batch * pl.tiles;
    pl.partial_off = align_up(pl.counters * sizeof(uint32_t), 256);
    pl.bytes = pl.partial_off + (size_t)batch * pl.partial_stride * sizeof(float);
    *out = pl;
    return true;
}

double plan_single(int m, int n, int k, int mode, int sm_count, int forced_tile, int forced_parts, int max_span,
                   int* tile, int* parts)
{
    sm_count = std::max(sm_count, 1);
    double best[kMaxClusterParts + 1];
    int best_tile[kMaxClusterParts + 1];
    for (int q = 0; q <= kMaxClusterParts; ++q) {
        best[q] = 1e300;
        best_tile[q] = kTileCount - 1;
    }
    int bp = 1;
    for (int t = 0; t < kTileCount; ++t) {
        if ((forced_tile >= 0 && t != forced_tile) || (mode == kMode4M && t == 0)) {
            continue;
        }
        const long long tiles = (long long)ceil_div(m, tile_bm(t)) * ceil_div(n, tile_bn(t));
        const int most = std::min(kMaxClusterParts, ceil_div(k, 16));  // partitions of 16 terms or more
        for (int q = 1; q <= most; ++q) {
            if (forced_parts > 0 && q != forced_parts) {
                continue;
            }
            const int span = q == 1 ? k : span_for(k, q);
            if ((q > 1 && (q - 1) * span >= k) || (forced_parts <= 0 && span > max_span)) {
                continue;
            }
            const int occ = single_occ(mode, t);
            const long long cap = std::max<long long>(1, (long long)kClusterCap[occ - 1][q - 1] * sm_count / 148);
            const long long layer = std::max<long long>(1, (long long)kClusterCap[0][q - 1] * sm_count / 148);
            const long long waves = (tiles + cap - 1) / cap;
            long long load = (tiles + layer - 1) / layer;
            if (k > kShortChain) {
                // Long chains outlast the placement: full waves, then the fewest
                // blocks per SM that hold the remaining clusters (25 x 1025 x
                // 59274: 33 clusters of 8 are two layers, not three; 8 partitions
                // took 438 us, 4, the least by whole layers, 549).
                load = tiles / cap * occ;
                if (const long long rest = tiles % cap) {
                    int o = 1;
                    while (o < occ && (long long)kClusterCap[o - 1][q - 1] * sm_count / 148 < rest) {
                        ++o;
                    }
                    load += o;
                }
            }
            const SingleCost& c = kSingleCost[t];
            // Four-product mode: four FFMA per output and K term instead of
            // three (the per-term costs scaled by that ratio, not fitted).
            // Shared SMs run 7 % above the linear fit, which single layers dominate.
            const double fma = (mode == kMode4M ? 4.0 / 3.0 : 1.0) * (load > 1 ? 1.07 : 1.0);
            double us = c.base_us + (double)waves * c.fixed_us +
                        span * 1e-3 * fma * ((double)waves * c.term_ns + (double)load * c.shared_term_ns);
            if (q > 1) {
                us += c.merge_us * q;
            }
            if (us < best[q]) {
                best[q] = us;
                best_tile[q] = t;
                bp = us < best[bp] || best[bp] == 1e300 ? q : bp;
            }
        }
    }
    // A chain's rounding error grows with the square root of its terms: beyond
    // kShortChain terms the finest split within 20 % of the least time.
    if (k > kShortChain) {
        const double least = best[bp];
        for (int q = kMaxClusterParts; q > bp && span_for(k, bp) > kShortChain; --q) {
            if (best[q] <= 1.2 * least) {
                bp = q;
            }
        }
    }
    if (tile != nullptr) {
        *tile = best_tile[bp];
    }
    if (parts != nullptr) {
        *parts = bp;
    }
    return best[bp];
}

cudaError_t launch_single(cudaStream_t s, const Problem& p, int mode, int repair, int tile, int parts)
{
    if (p.m <= 0 || p.n <= 0 || p.k <= 0 || parts < 1 || parts > kMaxClusterParts || tile < 0 ||
        tile >= kTileCount || (mode != kMode3M && mode != kMode4M) || (mode == kMode4M && tile == 0)) {
        return cudaErrorInvalidValue;
    }
    BProblem bp{};
    bp.ta = p.transa;
    bp.tb = p.transb;
    bp.m = p.m;
    bp.n = p.n;
    bp.k = p.k;
    const bool beta_zero = p.br == 0.0f && p.bi == 0.0f;
    const bool unit = p.ar == 1.0f && p.ai == 0.0f && beta_zero;
    bp.epi = EpiParams{p.ar, p.ai, p.br, p.bi, unit ? 1 : 0, beta_zero ? 1 : 0};
    bp.A = static_cast<const float2*>(p.A);
    bp.B = static_cast<const float2*>(p.B);
    bp.C = static_cast<float2*>(p.C);
    bp.lda = p.lda;
    bp.ldb = p.ldb;
    bp.ldc = p.ldc;
    bp.tile = tile;
    bp.repair = repair;
    bp.parts = parts;
    bp.span = span_for(p.k, parts);
    if ((parts - 1) * bp.span >= p.k) {
        return cudaErrorInvalidValue;  // the caller passes a partition count whose last part is non-empty
    }
    if (parts == 1) {
        bp.span = p.k;
    }
    bp.tiles_m = ceil_div(p.m, tile_bm(tile));
    bp.tiles_n = ceil_div(p.n, tile_bn(tile));
    const cudaError_t e =
        mode == kMode3M ? launch_single_tile<kMode3M>(s, bp, tile) : launch_single_tile<kMode4M>(s, bp, tile);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_strided(cudaStream_t s, const Problem& p, int mode, int repair, long long sA, long long sB,
                           long long sC, int batch, const StridedPlan& plan, void* ws, int sm_count)
{
    BProblem proto{};
    proto.ta = p.transa;
    proto.tb = p.transb;
    proto.m = p.m;
    proto.n = p.n;
    proto.k = p.k;
    const bool beta_zero = p.br == 0.0f && p.bi == 0.0f;
    const bool unit = p.ar == 1.0f && p.ai == 0.0f && beta_zero;
    proto.epi = EpiParams{p.ar, p.ai, p.br, p.bi, unit ? 1 : 0, beta_zero ? 1 : 0};
    proto.A = static_cast<const float2*>(p.A);
    proto.B = static_cast<const float2*>(p.B);
    proto.C = static_cast<float2*>(p.C);
    proto.lda = p.lda;
    proto.ldb = p.ldb;
    proto.ldc = p.ldc;
    proto.tile = plan.tile;
    proto.repair = repair;
    proto.parts = plan.parts;
    proto.span = plan.span;
    proto.tiles_m = ceil_div(p.m, plan.tile_m);
    proto.tiles_n = ceil_div(p.n, plan.tile_n);
    proto.ppitch = plan.ppitch;
    uint32_t* counters = static_cast<uint32_t*>(ws);
    float* partials = reinterpret_cast<float*>(static_cast<char*>(ws) + plan.partial_off);
    cudaError_t e = cudaMemsetAsync(counters, 0, plan.counters * sizeof(uint32_t), s);
    if (e != cudaSuccess) {
        return e;
    }
    const long long ntasks = (long long)plan.tiles * plan.parts * batch;
    auto run = [&](auto mode_c, auto tile_c) -> cudaError_t {
        constexpr int M = decltype(mode_c)::value, T = decltype(tile_c)::value;
        auto kernel = strided_kernel<M, T>;
        const size_t smem = kStridedSmem<M, T>;
        const int grid = (int)std::min<long long>(ntasks, (long long)std::max(sm_count, 1) * kStridedBlocks<M, T>);
        const cudaError_t attr = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (attr == cudaSuccess) {
            kernel<<<grid, kThreads, smem, s>>>(proto, sA, sB, sC, batch, plan.partial_stride, partials, counters);
        }
        return attr;
    };
    using std::integral_constant;
    auto run_mode = [&](auto mode_c) -> cudaError_t {
        switch (plan.tile) {
            case 0:
                if constexpr (decltype(mode_c)::value == kMode3M) {
                    return run(mode_c, integral_constant<int, 0>{});
                }
                return cudaErrorInvalidValue;
            case 1: return run(mode_c, integral_constant<int, 1>{});
            case 2: return run(mode_c, integral_constant<int, 2>{});
            case 3: return run(mode_c, integral_constant<int, 3>{});
            case 4: return run(mode_c, integral_constant<int, 4>{});
            default: return run(mode_c, integral_constant<int, 5>{});
        }
    };
    e = mode == kMode3M ? run_mode(integral_constant<int, kMode3M>{}) : run_mode(integral_constant<int, kMode4M>{});
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace cg3m

extern "C" {

cg3mStatus_t cg3mBatchPlanCreate(cg3mHandle_t handle, const cg3mProblem* problems, int count, int tune,
                                 cg3mBatchPlan_t* out, int* bad_index)
{
    if (handle == nullptr) {
        return CG3M_STATUS_HANDLE_IS_NULLPTR;
    }
    if (out == nullptr || count < 0 || (count > 0 && problems == nullptr)) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    *out = nullptr;
    std::vector<BProblem> ps;
    std::vector<int> index((size_t)count, -1);
    for (int i = 0; i < count; ++i) {
        const cg3mProblem& q = problems[i];
        int action = 0;
        const cg3mStatus_t st = validate(q.transa, q.transb, q.m, q.n, q.k, &q.alpha, q.A, q.lda, q.B, q.ldb, &q.beta,
                                         q.C, q.ldc, true, &action);
        if (st != CG3M_STATUS_SUCCESS) {
            if (bad_index != nullptr) {
                *bad_index = i;
            }
            return st;
        }
        if (action == 0) {
            continue;  // quick return: C unchanged
        }
        BProblem p{};
        p.ta = q.transa;
        p.tb = q.transb;
        p.m = q.m;
        p.n = q.n;
        p.k = action == 1 ? 0 : q.k;
        const bool beta_zero = q.beta.real == 0.0f && q.beta.imag == 0.0f;
        const bool unit = q.alpha.real == 1.0f && q.alpha.imag == 0.0f && beta_zero;
        p.epi = EpiParams{q.alpha.real, q.alpha.imag, q.beta.real, q.beta.imag, unit ? 1 : 0, beta_zero ? 1 : 0};
        p.A = reinterpret_cast<const float2*>(q.A);
        p.B = reinterpret_cast<const float2*>(q.B);
        p.C = reinterpret_cast<float2*>(q.C);
        p.lda = q.lda;
        p.ldb = q.ldb;
        p.ldc = q.ldc;
        index[(size_t)i] = (int)ps.size();
        ps.push_back(p);
    }
    cg3mBatchPlan* plan = new (std::nothrow) cg3mBatchPlan();
    if (plan == nullptr) {
        return CG3M_STATUS_ALLOC_FAILED;
    }
    plan->count = count;
    plan->index = std::move(index);
    plan->host = std::move(ps);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&plan->sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&plan->blocks_per_sm, batched_kernel, kThreads, kSmemBytes) !=
            cudaSuccess) {
        cudaGetLastError();
        delete plan;
        return CG3M_STATUS_INTERNAL_ERROR;
    }
    plan->device = dev;
    plan->blocks_per_sm = std::max(1, plan->blocks_per_sm);
    Policy pol = untuned_policy(plan->host, plan->sm_count);
    const std::string sig = signature(dev, plan->host);
    bool cached = false;
    {
        std::lock_guard<std::mutex> lock(g_tune_mutex);
        auto it = g_tuned.find(sig);
        if (it != g_tuned.end()) {
            pol = it->second;
            cached = true;
        }
    }
    if (tune && !cached && !plan->host.empty()) {
        pol = autotune(plan, handle->stream, pol);
        std::lock_guard<std::mutex> lock(g_tune_mutex);
        g_tuned[sig] = pol;
    }
    if (materialise(plan, plan->host, pol) != cudaSuccess) {
        cudaGetLastError();
        delete plan;
        return CG3M_STATUS_ALLOC_FAILED;
    }
    *out = plan;
    return CG3M_STATUS_SUCCESS;
}

cg3mStatus_t cg3mBatchPlanExecute(cg3mHandle_t handle, cg3mBatchPlan_t plan, int use_graph)
{
    if (handle == nullptr) {
        return CG3M_STATUS_HANDLE_IS_NULLPTR;
    }
    if (plan == nullptr) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    if (!use_graph || plan->tasks.empty()) {
        return launch(plan, handle->stream) == cudaSuccess ? CG3M_STATUS_SUCCESS : CG3M_STATUS_EXECUTION_FAILED;
    }
    if (plan->exec == nullptr) {
        if (plan->capture_stream == nullptr &&
            cudaStreamCreateWithFlags(&plan->capture_stream, cudaStreamNonBlocking) != cudaSuccess) {
            return CG3M_STATUS_INTERNAL_ERROR;
        }
        if (cudaStreamBeginCapture(plan->capture_stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            return CG3M_STATUS_EXECUTION_FAILED;
        }
        const cudaError_t le = launch(plan, plan->capture_stream);
        cudaGraph_t g = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(plan->capture_stream, &g);
        if (le != cudaSuccess || ce != cudaSuccess || g == nullptr) {
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            return CG3M_STATUS_EXECUTION_FAILED;
        }
        plan->graph = g;
        if (cudaGraphInstantiate(&plan->exec, g, 0) != cudaSuccess) {
            cudaGetLastError();
            plan->exec = nullptr;
            return CG3M_STATUS_EXECUTION_FAILED;
        }
    }
    return cudaGraphLaunch(plan->exec, handle->stream) == cudaSuccess ? CG3M_STATUS_SUCCESS
                                                                      : CG3M_STATUS_EXECUTION_FAILED;
}

cg3mStatus_t cg3mBatchPlanDestroy(cg3mBatchPlan_t plan)
{
    if (plan == nullptr) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    // Work enqueued with the plan may still read its task list.
    if (plan->device >= 0) {
        int cur = 0;
        cudaGetDevice(&cur);
        cudaSetDevice(plan->device);
        cudaDeviceSynchronize();
        cudaSetDevice(cur);
    }
    delete plan;
    return CG3M_STATUS_SUCCESS;
}

cg3mStatus_t cg3mBatchPlanDescribe(cg3mBatchPlan_t plan, int* tile_m, int* tile_n, int* k_partitions)
{
    if (plan == nullptr) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    for (int i = 0; i < plan->count; ++i) {
        const int h = plan->index[(size_t)i];
        const BProblem* p = h >= 0 ? &plan->host[(size_t)h] : nullptr;
        if (tile_m) tile_m[i] = p ? tile_bm(p->tile) : 0;
        if (tile_n) tile_n[i] = p ? tile_bn(p->tile) : 0;
        if (k_partitions) k_partitions[i] = p ? (p->k > 0 ? p->parts : 0) : 0;
    }
    return CG3M_STATUS_SUCCESS;
}

}  // extern "C"
