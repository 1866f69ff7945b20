// ozaki.cu -- FP64-accurate recompute of the flagged outputs of dense tiles on
// the tensor cores: the rounding-correction pass of the tensor-core forms.
//
// The reference recomputes flagged outputs with its segmented FP32 replay
// (cgemm3m_rounding_kernel.cpp:192-404); the tensor-core forms of this library
// promise instead that every flagged output is within one FP32 rounding of the
// exact product.  Recomputing ~3/4 of a 4096^3 product in FP64 on the CUDA
// cores takes ~24 ms at this GPU's FP64 rate, so the products run on the int8
// tensor cores as exact integer products modulo small coprime moduli, put
// back together by the Chinese remainder theorem (the modular form of the
// Ozaki scheme: Ozaki, Uchino and Imamura, "Ozaki Scheme II: A GEMM-oriented
// emulation of floating-point matrix multiplication using an integer modular
// technique", 2025):
//
//   1. ozaki_split_kernel: every op(A) row i and op(B) column j gets a power
//      of two 2^E > max |x| over the row (real and imaginary parts together;
//      the energy kernel finds it); each part becomes the integer
//      a = rn(x 2^(beta - E)), |a| <= 2^beta, beta = 47, and the row counts its
//      parts for which a != x 2^(beta - E) (cA_i; cB_j for the columns).  Every prime factor of the kOzMods = 15
//      moduli p_m <= 241 (pairwise coprime, product M ~ 2^111.1) is 1 mod 4, so
//      -1 has a square root r_m mod p_m and z -> (Re z + r_m Im z,
//      Re z - r_m Im z) turns a complex product mod p_m into two independent
//      real ones (quadratic residue numbers: Krogmeier and Jenkins, "Error
//      detection and correction in quadratic residue number systems", 1983).
//      The planes hold both images of every element as int8.
//   2. ozaki_pair_kernel: for each modulus the two products
//        P+ = sum A+ B+,  P- = sum A- B-
//      are exact in the int32 TMEM accumulators (|sum| <= 4096 * 125^2 < 2^26);
//      the epilogue stores a byte y in [0, 255) congruent to the sum mod p_m
//      per output and product.
//   3. ozaki_crt_kernel: mod p_m, Re = (P+ + P-) / 2 and Im = (P+ - P-) / (2 r_m).
//      So x = sum_m (y+ + y-) w_m - k M for the real part, with
//      w_m = u_m (M / p_m), u_m = (2 M / p_m)^-1 mod p_m (w_m = 1/2 mod p_m, 0
//      mod the other moduli), the imaginary part with (y+ - y-) and
//      u_m = (2 r_m M / p_m)^-1, and k the nearest integer to the sum / M (from
//      the exact limb sums)
//      (|x| <= 2 n 2^(2 beta) <= 2^107 < M / 8, so k is never in doubt),
//      evaluated exactly in three 40-bit limbs of FP64.  Rounding a part moves
//      each real product by at most 2^(beta - 1), so
//        |error| <= (cA_i + cB_j) 2^(beta - 1)   (units of 2^(E_i + F_j - 2 beta)),
//      zero for rows and columns that scaled exactly.  Every output of a tile
//      that ran is written (flagged or not: the form's own products skip
//      these tiles) when the bound is zero or both parts exceed 2^25 times it
//      (so the result, rounded to FP32, is within one FP32 rounding of the
//      exact product); otherwise it is marked for the FP64 per-output kernel,
//      as are outputs whose row or column holds a non-finite value.
//
// Two products per modulus instead of the four of Re = Ar Br - Ai Bi,
// Im = Ar Bi + Ai Br: 30 int8 products of n^3 against 56 with 14 moduli that
// need no square root of -1.  At 4096^3 with every tile dense: products 2.57 ->
// 1.28 ms, residues 0.34 -> 0.29, reconstruction 0.21 -> 0.23.  A work unit is
// 256 rows x 512 columns of one product, so 768 operand rows feed 256 x 512
// outputs (12.1 GB from L2 in all, 9.4 TB/s) and both TMEM accumulators
// (2 x 256 columns) share the op(A) stage.  Loads alone took 0.91 ms and the
// MMAs need 0.87 ms at the tensor pipe's rate; 64-byte instead of 128-byte K
// rows took 1.6x as long, and MMAs issued from a lane-0 branch instead of a
// warp that stays together 1.4x.
//
// B200 design: a persistent cluster of two CTAs per SM pair
// (tcgen05.mma.cta_group::2.kind::i8, M = 256, N = 256, K = 32) walks the
// units (product plane, taken tiles).  The units of one plane are consecutive,
// so all pairs stream the same few planes and find them in L2.  CTA r stages
// rows [128r, 128r + 128) of op(A) and columns [128r, 128r + 128) of each of
// the unit's two 256-column tiles, 128-byte K rows with the 128-byte swizzle,
// 48 KB per stage in a 4-stage ring.  Warp 0 of both CTAs issues the TMA
// copies (completion on the even CTA's barrier), one lane of the even CTA's
// warp 1 issues every MMA, warps 2..9 of both CTAs drain the accumulators.
// kOzGroup stages at a time run all of one half's MMAs before the other's, so
// at a unit's ends each half drains while the tensor core works on the other
// half (1.34 ms with one stage at a time, 1.28 with two or three).  Every wait
// is bounded.
#include "cg3m_internal.h"
#include "ptx.cuh"

namespace cg3m {

namespace {

constexpr int kOzMods = 15;                    // moduli; two product planes each
constexpr int kOzPlanes = 2 * kOzMods;         // planes per operand, and product residue planes
constexpr int kOzBeta = 47;                    // bits of the scaled integer parts
constexpr int kOzMaxN = 4096;                  // 2 n 2^(2 beta) <= M / 8 up to this order
constexpr int OZ_TILE_M = kOzakiTile;          // output rows of a tile (M of the pair MMA)
constexpr int OZ_TN = kOzakiTile;              // output columns of a tile (N of the pair MMA)
constexpr int OZ_ROWS = 128;                   // rows of each operand tile staged by one CTA
constexpr int OZ_BK = 128;                     // K bytes per staged row (128-byte swizzle)
constexpr int OZ_PLANE = OZ_ROWS * OZ_BK;      // 16 KB
constexpr int OZ_STAGE = 3 * OZ_PLANE;         // op(A) and two op(B) tiles
constexpr int OZ_STAGES = 4;
constexpr size_t OZ_SMEM = (size_t)OZ_STAGES * OZ_STAGE + 1024 + 256;
constexpr int kOzGroup = 2;                    // stages run on one half, then on the other
constexpr int kOzEpiWarps = 8;
constexpr int OZ_PIECE = OZ_TN / (kOzEpiWarps / 4);  // columns of a half one epilogue warp drains
constexpr int kOzThreads = (2 + kOzEpiWarps) * 32;
constexpr int kOzMaxTiles = kOzMaxN / kOzakiTile;                      // tiles per side
constexpr int kOzMaxUnits = kOzMaxTiles * ((kOzMaxTiles + 1) / 2);     // tile pairs of one plane
constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: x + kMagic rounds x to an integer
constexpr float kMagicF = 12582912.0f;         // 1.5 * 2^23
static_assert(kOzGroup < OZ_STAGES, "a group holds its stages until both halves have read them");

// Moduli, largest first: pairwise coprime, every prime factor 1 mod 4
// (221 = 13 17, 205 = 5 41, the rest prime), and a square root of -1 mod each.
constexpr int kOzModuli[kOzMods] = {241, 233, 229, 221, 205, 197, 193, 181, 173, 157, 149, 137, 113, 109, 101};
constexpr int kOzRoots[kOzMods] = {64, 89, 107, 21, 32, 14, 81, 19, 80, 28, 44, 37, 15, 33, 10};

constexpr int balanced_mod(long long v, int p)
{
    const int r = (int)(((v % p) + p) % p);
    return r <= p / 2 ? r : r - p;
}
constexpr int abs_int(int v) { return v < 0 ? -v : v; }

// The images' constants: an element with 16-bit limbs (real a2 a1 a0,
// imaginary b2 b1 b0, |limb| <= 2^15) has the images
// (a2 c2 + a1 c1 + a0) +- (b2 d2 + b1 d1 + b0 d0) mod p; c1 = 2^16, c2 = 2^32,
// d0 = r, d1 = 2^16 r, d2 = 2^32 r, each balanced mod p.
struct OzSplitMod {
    float c1, c2, d0, d1, d2, pf, inv_pf;
};
constexpr OzSplitMod split_mod(int mi)
{
    const int p = kOzModuli[mi], r = kOzRoots[mi];
    return OzSplitMod{(float)balanced_mod(1LL << 16, p),       (float)balanced_mod(1LL << 32, p),
                      (float)balanced_mod(r, p),               (float)balanced_mod((1LL << 16) * r, p),
                      (float)balanced_mod((1LL << 32) * r, p), (float)p, 1.0f / (float)p};
}
// Every image's limb sum is an exact FP32 integer: 2^15 (1 + sum |c|) < 2^24,
// and r_m^2 = -1 mod p_m.
constexpr bool split_constants_ok()
{
    for (int mi = 0; mi < kOzMods; ++mi) {
        const int p = kOzModuli[mi], r = kOzRoots[mi];
        const int sum = 1 + abs_int(balanced_mod(1LL << 16, p)) + abs_int(balanced_mod(1LL << 32, p)) +
                        abs_int(balanced_mod(r, p)) + abs_int(balanced_mod((1LL << 16) * r, p)) +
                        abs_int(balanced_mod((1LL << 32) * r, p));
        if (sum >= 512 || (r * r + 1) % p != 0) {
            return false;
        }
    }
    return true;
}
static_assert(split_constants_ok(), "limb sums of the images must be exact in FP32");

// Constants of the reconstruction (host-computed once, passed by value).
struct OzCrt {
    double w[kOzMods][2][3];  // w_m of the real, imaginary part in 40-bit limbs, low first
    double m[3];              // M in 40-bit limbs, low first
    double k2, k1;            // rn(2^80 / M), rn(2^40 / M): k from the limb sums
};

struct OzParams {
    int kblocks;             // 128-byte K blocks
    int tiles;               // tiles per side
    int tn0, tn1;            // tile columns of this launch
    const uint8_t* tile_ran; // per tile (tn * tiles + tm): 1 when the exact products run there
    uint8_t* residues;       // [kOzPlanes][y_pad / 16][y_pad][16]
    int y_pad;
    size_t y_plane;
    int p[kOzMods];
    int inv[kOzMods];        // floor(2^32 / p)
    int bias[kOzMods];       // the multiple of p at or above 2^26
    int* status;
};

struct OzFinish {
    int n;
    int tiles;
    int strip0;              // first 16-column strip of this launch
    const int* E;            // op(A) row exponents
    const int* F;            // op(B) column exponents
    const int* CA;           // rounded parts per op(A) row
    const int* CB;           // rounded parts per op(B) column
    const uint8_t* tile_ran;
    const uint8_t* residues;
    int y_pad;
    size_t y_plane;
    uint32_t* stats;
    uint32_t* fallback_bits;
    float2* C;
    OzCrt crt;
};

// ---- 1. residues -------------------------------------------------------------------

// The three signed 16-bit limbs of an integer-valued t (|t| <= 2^47, given
// tm = t + 1.5 * 2^52, whose low 51 bits hold t in two's complement):
// t = l[2] 2^32 + l[1] 2^16 + l[0], l[0] and l[1] in [-2^15, 2^15).
__device__ __forceinline__ void limbs16(double tm, float* l)
{
    const int lo = __double2loint(tm), hi = __double2hiint(tm) - 0x43380000;
    const int l0 = (int)(short)lo;
    // exact: lo - l0 is a multiple of 2^16, and hi takes both carries below
    const int m1 = (int)(((unsigned)lo >> 16) + (l0 < 0 ? 1u : 0u));  // 0 .. 2^16
    const int l1 = m1 >= 32768 ? m1 - 65536 : m1;
    const int l2 = hi + (m1 >= 32768 ? 1 : 0);
    l[0] = __fsub_rn(__int_as_float(0x4B400000 + l0), kMagicF);
    l[1] = __fsub_rn(__int_as_float(0x4B400000 + l1), kMagicF);
    l[2] = __fsub_rn(__int_as_float(0x4B400000 + l2), kMagicF);
}

// s mod p as an integer of magnitude <= 125, in the low byte of the result's
// bits: q = rint(s rn(1/p)) is off s / p by at most 1/2 + 2^-6 (|s| < 2^24,
// p >= 101), and s - q p is exact.
__device__ __forceinline__ float2 mod_bits2(float2 s, float2 neg_p, float2 inv_p)
{
    const float2 magic = make_float2(kMagicF, kMagicF), neg_magic = make_float2(-kMagicF, -kMagicF);
    const float2 q = __fadd2_rn(__ffma2_rn(s, inv_p, magic), neg_magic);
    return __fadd2_rn(__ffma2_rn(q, neg_p, s), magic);
}

// Low bytes of four packed pairs' bits as eight consecutive bytes.
__device__ __forceinline__ uint2 low_bytes8(const float2* v)
{
    uint32_t w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t a = __byte_perm(__float_as_uint(v[2 * h].x), __float_as_uint(v[2 * h].y), 0x0040);
        const uint32_t b = __byte_perm(__float_as_uint(v[2 * h + 1].x), __float_as_uint(v[2 * h + 1].y), 0x0040);
        w[h] = __byte_perm(a, b, 0x5410);
    }
    return make_uint2(w[0], w[1]);
}

// Both images of eight consecutive terms for modulus MI and the ones after it.
template <int MI>
__device__ __forceinline__ void store_images(const float2 (*re)[3], const float2 (*im)[3], int8_t* dst,
                                             size_t plane_bytes)
{
    if constexpr (MI < kOzMods) {
        constexpr OzSplitMod k = split_mod(MI);
        const float2 c1 = make_float2(k.c1, k.c1), c2 = make_float2(k.c2, k.c2);
        const float2 d0 = make_float2(k.d0, k.d0), d1 = make_float2(k.d1, k.d1), d2 = make_float2(k.d2, k.d2);
        const float2 neg_p = make_float2(-k.pf, -k.pf), inv_p = make_float2(k.inv_pf, k.inv_pf);
        const float2 zero = make_float2(0.0f, 0.0f), minus = make_float2(-1.0f, -1.0f);
        float2 plus_bits[4], minus_bits[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float2 a = __ffma2_rn(re[u][2], c2, __ffma2_rn(re[u][1], c1, re[u][0]));
            const float2 b = __ffma2_rn(im[u][2], d2, __ffma2_rn(im[u][1], d1, __ffma2_rn(im[u][0], d0, zero)));
            plus_bits[u] = mod_bits2(__fadd2_rn(a, b), neg_p, inv_p);
            minus_bits[u] = mod_bits2(__ffma2_rn(b, minus, a), neg_p, inv_p);
        }
        *reinterpret_cast<uint2*>(dst) = low_bytes8(plus_bits);
        *reinterpret_cast<uint2*>(dst + plane_bytes) = low_bytes8(minus_bits);
        store_images<MI + 1>(re, im, dst + 2 * plane_bytes, plane_bytes);
    }
}

// One block per op(A) row (the first nrows_a) or op(B) column of the panel.
// Plane layout: [2m + {0 plus, 1 minus}][row][kpitch] int8 for both operands.
//
// All FP32: the 47-bit parts go through 16-bit limbs, so a residue is a few
// exact FP32 products (15 FP32 operations per element and modulus for both
// images, two elements per instruction) instead of FP64 ones.  Scalar FMAs with
// immediate constants took 0.355 ms at 4096^3, packed ones 0.287.  The row's
// exponent comes from the energy kernel, which reads the same rows: finding the
// largest part here took a second read and a barrier before any arithmetic.
__global__ void __launch_bounds__(256)
    ozaki_split_kernel(int n, int pitch, const float2* __restrict__ rows_a, const float2* __restrict__ rows_b,
                       int8_t* __restrict__ pa, int8_t* __restrict__ pb, int kpitch, size_t plane_bytes,
                       const int* __restrict__ E, const int* __restrict__ F, int* __restrict__ CA,
                       int* __restrict__ CB, int nrows_a, int j0, const uint8_t* __restrict__ band_a, const uint8_t* __restrict__ band_b)
{
    __shared__ int wcnt[8];
    const int r = panel_row(blockIdx.x, nrows_a, n, j0);
    const bool is_a = r < n;
    const int row = is_a ? r : r - n;
    if (!(is_a ? band_a : band_b)[row / kOzakiTile]) {
        return;  // no tile of this band runs, or an earlier panel's residues stand
    }
    const float2* src = (is_a ? rows_a : rows_b) + (size_t)row * pitch;
    const int tid = threadIdx.x;
    // Every part scaled by 2^(beta - e) lies in (-2^beta, 2^beta).
    const int e = (is_a ? E : F)[row];
    const bool usable = e != kOzNonFinite && e != kOzZero;
    const double scale = usable ? ldexp(1.0, kOzBeta - e) : 0.0;
    int8_t* dst = (is_a ? pa : pb) + (size_t)row * kpitch;
    int rounded = 0;
    // Eight consecutive K terms per thread: 8-byte stores into every plane.
#pragma unroll 1
    for (int k0 = tid * 8; k0 < n; k0 += 256 * 8) {
        float2 re[4][3], im[4][3];  // [pair of terms][limb]
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k0 + u;
            const float2 x = (k < n && usable) ? src[k] : make_float2(0.0f, 0.0f);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const double sx = __dmul_rn((double)(part == 0 ? x.x : x.y), scale);  // exact: a power of two
                const double tm = __dadd_rn(sx, kMagic);  // rounds to an integer: |sx| < 2^51
                rounded += __dsub_rn(tm, kMagic) != sx;   // the nearest integer, |t| <= 2^beta
                float l[3];
                limbs16(tm, l);
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    float2& pair = part == 0 ? re[u >> 1][b] : im[u >> 1][b];
                    ((u & 1) ? pair.y : pair.x) = l[b];
                }
            }
        }
        // K beyond n is never read (the tensor maps stop at n), so whole
        // 8-byte groups may be stored while k0 < n <= kpitch.
        store_images<0>(re, im, dst + k0, plane_bytes);
    }
    rounded = __reduce_add_sync(0xffffffffu, rounded);
    if ((tid & 31) == 0) {
        wcnt[tid >> 5] = rounded;
    }
    __syncthreads();
    if (tid == 0) {
        int total = 0;
        for (int w = 0; w < 8; ++w) {
            total += wcnt[w];
        }
        (is_a ? CA : CB)[row] = total;
    }
}

// ---- 2. residue products --------------------------------------------------------------

// Shared-memory matrix descriptor: K-major, 128-byte swizzle (layout type 2),
// 8-row groups 8 x 128 = 1024 bytes apart (SBO), leading offset unused (1),
// descriptor version 1.  Each plane tile starts on a 1024-byte boundary; the
// 32-byte K steps of a row advance the start address by 32 bytes.
__device__ __forceinline__ uint64_t oz_desc(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)((8 * OZ_BK) >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

__device__ __forceinline__ void umma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 16 accumulator values (int32 bits, |x| < 2^26) -> 16 bytes congruent mod p:
// with X = x + bias in [0, 2^27 + p) and inv = floor(2^32 / p),
// q = floor(X inv / 2^32) is floor(X / p) or one less when X / p lies within
// 2^-5 above an integer, so X - q p is in [0, p + p / 32], below 256.
__device__ __forceinline__ uint4 residue_bytes16(const float* v, int neg_p, int inv, int bias)
{
    uint32_t w[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        uint32_t r[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int x = __float_as_int(v[4 * g + b]) + bias;
            r[b] = (uint32_t)(__mulhi(x, inv) * neg_p + x);
        }
        w[g] = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// One work unit's tiles: tile row tm and one or two taken tile columns.
struct OzUnit {
    uint8_t tm, tn[2], halves;
};

__global__ void __launch_bounds__(kOzThreads, 1)
    ozaki_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ OzParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = align_shared<1024>(smem_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(ring + OZ_STAGES * OZ_STAGE);
    uint64_t* empty = full + OZ_STAGES;
    uint64_t* acc_full = empty + OZ_STAGES;  // [2] MMA -> epilogue: half h's sums are in TMEM
    uint64_t* acc_free = acc_full + 2;       // [2] epilogue -> MMA (even CTA): half h drained
    uint64_t* mma_done = acc_free + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    __shared__ OzUnit units[kOzMaxUnits];
    __shared__ int unit_count;

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank() & 1u;
    const bool leader = rank == 0;
    const uint16_t pair_mask = 0x3u;
    const int pid = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    // The units of one plane, the same list in every CTA: each tile row's taken
    // tile columns in twos (lane r of warp 0 lists row r).
    if (warp == 0) {
        uint32_t mask = 0;
        if (lane < p.tiles) {
            for (int tn = p.tn0; tn < p.tn1; ++tn) {
                mask |= (p.tile_ran[(size_t)tn * p.tiles + lane] ? 1u : 0u) << tn;
            }
        }
        const int mine = (__popc(mask) + 1) / 2;
        int at = mine;
#pragma unroll
        for (int off = 1; off < 32; off *= 2) {
            const int up = __shfl_up_sync(0xffffffffu, at, off);
            at += lane >= off ? up : 0;
        }
        if (lane == 31) {
            unit_count = at;
        }
        at -= mine;
        while (mask != 0) {
            OzUnit u{(uint8_t)lane, {0, 0}, 0};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (mask != 0) {
                    u.tn[h] = (uint8_t)(__ffs(mask) - 1);
                    mask &= mask - 1;
                    u.halves = (uint8_t)(h + 1);
                }
            }
            units[at++] = u;
        }
    }
    __syncthreads();
    const int per_plane = unit_count, total = per_plane * kOzPlanes;
    if (pid >= total) {
        return;  // both CTAs of the pair, before any barrier or TMEM is touched
    }
    if (tid == 0) {
        for (int s = 0; s < OZ_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int h = 0; h < 2; ++h) {
            mbar_init(&acc_full[h], 1);
            mbar_init(&acc_free[h], 2 * kOzEpiWarps);
        }
        mbar_init(mma_done, 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer (both CTAs) ----------------
        if (lane == 0) {
            tma_prefetch_desc(&tmA);
            tma_prefetch_desc(&tmB);
            const uint32_t full0 = mapa_shared(smem_u32(full), 0);  // the even CTA's barriers
            int it = 0;
            bool stop = false;
            for (int g = pid; g < total && !stop; g += pairs) {
                const int plane = g / per_plane;
                const OzUnit u = units[g - plane * per_plane];
                const int m0 = u.tm * OZ_TILE_M + (int)rank * OZ_ROWS;
                for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
                    const int slot = it % OZ_STAGES;
                    if ((it >= OZ_STAGES && !mbar_wait(&empty[slot], ((it / OZ_STAGES) - 1) & 1, p.status)) ||
                        *abort_flag) {
                        *abort_flag = 1;
                        stop = true;
                        break;
                    }
                    uint8_t* st = ring + slot * OZ_STAGE;
                    const uint32_t bar = full0 + (uint32_t)slot * 8u;
                    if (leader) {
                        mbar_arrive_expect_tx(&full[slot], 2 * (1 + u.halves) * OZ_PLANE);
                    }
                    tma_load_3d_pair(st, &tmA, bar, kb * OZ_BK, m0, plane);
                    for (int h = 0; h < u.halves; ++h) {
                        tma_load_3d_pair(st + (1 + h) * OZ_PLANE, &tmB, bar, kb * OZ_BK,
                                         u.tn[h] * OZ_TN + (int)rank * OZ_ROWS, plane);
                    }
                }
            }
            if (leader) {
                for (int j = it > OZ_STAGES ? it - OZ_STAGES : 0; j < it; ++j) {
                    mbar_wait(&full[j % OZ_STAGES], (j / OZ_STAGES) & 1, p.status);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (even CTA) ----------------
        // The whole warp walks the loop, one elected lane issues.
        if (leader) {
            const bool issuer = elect_one();
            // descriptor of the ring's start; the address field counts 16 bytes
            const uint64_t desc0 = oz_desc(smem_u32(ring));
            // S32 accumulate, signed 8-bit A and B, both K-major, N = 256, M = 256.
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_TN >> 3) << 17) |
                                   ((uint32_t)(OZ_TILE_M >> 4) << 24);
            int it = 0;
            uint32_t phase = 0;  // bit h: parity of the units that used half h
            bool stop = false;
            for (int g = pid; g < total && !stop; g += pairs) {
                const int halves = units[g % per_plane].halves;
                for (int kb = 0; kb < p.kblocks && !stop;) {
                    const bool first = kb == 0;
                    const bool last = kb + kOzGroup >= p.kblocks;
                    const int group = last ? p.kblocks - kb : kOzGroup;
                    for (int h = 0; h < halves && !stop; ++h) {
                        if (first) {
                            // passes at once for the half's first unit
                            if (!warp_all(mbar_wait_cluster(&acc_free[h], ((phase >> h) & 1u) ^ 1u, p.status))) {
                                *abort_flag = 1;
                                stop = true;
                                break;
                            }
                            tc_fence_after();
                        }
                        const uint32_t d = tmem + (uint32_t)(h * OZ_TN);
                        for (int j = 0; j < group; ++j) {
                            const int slot = (it + j) % OZ_STAGES;
                            if (h == 0) {
                                if (!warp_all(mbar_wait(&full[slot], ((it + j) / OZ_STAGES) & 1, p.status))) {
                                    *abort_flag = 1;
                                    stop = true;
                                    break;
                                }
                                tc_fence_after();
                            }
                            const uint64_t a = desc0 + (uint32_t)(slot * (OZ_STAGE >> 4));
                            const uint64_t b = a + (uint32_t)((1 + h) * (OZ_PLANE >> 4));
                            if (issuer) {
#pragma unroll
                                for (int kk = 0; kk < OZ_BK / 32; ++kk) {
                                    umma_i8_pair(d, a + 2 * kk, b + 2 * kk, idesc, (kb + j > 0 || kk > 0) ? 1u : 0u);
                                }
                                if (h == halves - 1) {
                                    umma_commit_pair(&empty[slot], pair_mask);
                                }
                            }
                        }
                        if (last && !stop) {
                            if (issuer) {
                                umma_commit_pair(&acc_full[h], pair_mask);
                            }
                            phase ^= 1u << h;
                        }
                    }
                    kb += group;
                    it += group;
                }
            }
            if (issuer) {
                umma_commit_pair(mma_done, pair_mask);
            }
            mbar_wait(mma_done, 0, p.status);  // nothing may still write TMEM when it is freed
        }
    } else {
        // ---------------- epilogue warps 2..9 (both CTAs) ----------------
        // TMEM lane quadrant = warp % 4 (the warp's 32 rows); of each half's
        // 256 columns the two warps of a
        // quadrant take 128 each.  Every
        // row and column of a tile lies inside the padded residue planes, so
        // the stores need no bounds (rows and columns past n hold zeros).
        const int quad = warp & 3;
        const int piece = (warp - 2) >> 2;
        const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(piece * OZ_PIECE);
        const size_t strip = (size_t)p.y_pad * 16;  // bytes of one 16-column strip of a plane
        uint32_t phase = 0;
        bool ok = true;
        for (int g = pid; g < total && ok; g += pairs) {
            const int plane = g / per_plane;
            const OzUnit u = units[g - plane * per_plane];
            const int mi = plane >> 1;
            const int neg_p = -p.p[mi], inv = p.inv[mi], bias = p.bias[mi];
            const int row = u.tm * OZ_TILE_M + (int)rank * OZ_ROWS + quad * 32 + lane;
            for (int h = 0; h < u.halves; ++h) {
                const bool ready = mbar_wait(&acc_full[h], (phase >> h) & 1u, p.status);
                phase ^= 1u << h;
                tc_fence_after();
                ok = __all_sync(0xffffffffu, ready && !*abort_flag);
                if (!ok) {
                    break;
                }
                uint8_t* out = p.residues + (size_t)plane * p.y_plane +
                               (size_t)((u.tn[h] * OZ_TN + piece * OZ_PIECE) >> 4) * strip + (size_t)row * 16;
                const uint32_t src = lane_addr + (uint32_t)(h * OZ_TN);
#pragma unroll 1
                for (int cb = 0; cb < OZ_PIECE; cb += 32) {
                    float v[32];
                    tmem_ld16x2(src + (uint32_t)cb, src + (uint32_t)(cb + 16), v, v + 16);
                    __stcg(reinterpret_cast<uint4*>(out), residue_bytes16(v, neg_p, inv, bias));
                    __stcg(reinterpret_cast<uint4*>(out + strip), residue_bytes16(v + 16, neg_p, inv, bias));
                    out += 2 * strip;
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(mapa_shared(smem_u32(&acc_free[h]), 0));
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the even CTA's MMAs are complete; neither CTA's memory is used any more
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem, 512);
    }
}

// ---- 3. reconstruction ---------------------------------------------------------------

// 2^e as a double for -1022 <= e <= 1023.
__device__ __forceinline__ double pow2d(int e)
{
    return __hiloint2double((e + 1023) << 20, 0);
}

// 2^52 + v for an integer v in [0, 2^32), minus `off`: exact.
__device__ __forceinline__ double small_int_d(int v, double off)
{
    return __dsub_rn(__hiloint2double(0x43300000, v), off);
}

// One part's exact integer product from its limb sums.
__device__ __forceinline__ double crt_value(const OzCrt& crt, const double* s)
{
    // S / M = k + x / M with |x / M| < 1/8, S = (s2 2^40 + s1) 2^40 + s0;
    // s2 rn(2^80 / M) + s1 rn(2^40 / M) is off S / M by < 2^-38 (|S / M| < 7700)
    const double k = rint(__fma_rn(s[2], crt.k2, __dmul_rn(s[1], crt.k1)));
    const double d0 = __fma_rn(-k, crt.m[0], s[0]);  // exact integers of magnitude <= 2^53
    const double d1 = __fma_rn(-k, crt.m[1], s[1]);
    const double d2 = __fma_rn(-k, crt.m[2], s[2]);
    // x = (d2 2^40 + d1) 2^40 + d0: two roundings, relative error < 2^-52
    return __fma_rn(__fma_rn(d2, 1099511627776.0, d1), 1099511627776.0, d0);
}

// One thread per op(A) row and two consecutive op(B) columns; a block holds 32
// rows x 16 columns inside one exact tile, and a warp (4 rows x 8 column
// pairs) reads 64 consecutive residue bytes per plane and writes whole 32-byte
// sectors of C.  Two outputs per thread keep it near 64 registers, for twice
// the resident warps of four.  Writes every output of the tile whose bound
// certifies it and marks the rest in fallback_bits.
constexpr int kCrtRows = 32;

__global__ void __launch_bounds__(256, 4) ozaki_crt_kernel(const __grid_constant__ OzFinish f)
{
    const int pair = threadIdx.x & 7;
    const int row = blockIdx.y * kCrtRows + (threadIdx.x >> 3);
    const int strip = f.strip0 + blockIdx.x;
    const int col0 = strip * 16 + pair * 2;
    const int n = f.n;
    const int tm = (blockIdx.y * kCrtRows) / OZ_TILE_M, tn = (strip * 16) / OZ_TN;
    if (!f.tile_ran[(size_t)tn * f.tiles + tm] || row >= n || col0 >= n) {
        return;
    }
    // Every output of a tile that ran is written here, flagged or not: the
    // form's own products skipped these tiles.
    const uint8_t* src = f.residues + ((size_t)strip * f.y_pad + row) * 16 + pair * 2;
    double xr[2], xi[2];
    {
        double s[2][2][3];  // [part][output][limb]
#pragma unroll
        for (int part = 0; part < 2; ++part) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                s[part][c][0] = s[part][c][1] = s[part][c][2] = 0.0;
            }
        }
        uint32_t yp[kOzMods], ym[kOzMods];
#pragma unroll
        for (int mi = 0; mi < kOzMods; ++mi) {
            yp[mi] = __ldcs(reinterpret_cast<const unsigned short*>(src + (size_t)(2 * mi) * f.y_plane));
            ym[mi] = __ldcs(reinterpret_cast<const unsigned short*>(src + (size_t)(2 * mi + 1) * f.y_plane));
        }
#pragma unroll
        for (int mi = 0; mi < kOzMods; ++mi) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int a = (int)((yp[mi] >> (8 * c)) & 0xFFu), b = (int)((ym[mi] >> (8 * c)) & 0xFFu);
                const double v[2] = {small_int_d(a + b, 4503599627370496.0),
                                     small_int_d(a - b + 256, 4503599627370496.0 + 256.0)};
                // |v| < 512, 40-bit limbs, 15 terms: every product and partial
                // sum stays below 2^53: exact
#pragma unroll
                for (int part = 0; part < 2; ++part) {
#pragma unroll
                    for (int l = 0; l < 3; ++l) {
                        s[part][c][l] = __fma_rn(v[part], f.crt.w[mi][part][l], s[part][c][l]);
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            xr[c] = crt_value(f.crt, s[0][c]);
            xi[c] = crt_value(f.crt, s[1][c]);
        }
    }
    const int ei = f.E[row];
    const int ca = f.CA[row];
    uint32_t fallbacks = 0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int col = col0 + c;
        if (col >= n) {
            break;
        }
        const size_t idx = (size_t)col * n + row;
        const int fj = f.F[col];
        bool ok = ei != kOzNonFinite && fj != kOzNonFinite;
        float2 out = make_float2(0.0f, 0.0f);  // a zero row or column: the exact product is zero
        if (ok && ei != kOzZero && fj != kOzZero) {
            const int cnt = ca + f.CB[col];
            if (cnt != 0) {
                // |error| <= cnt 2^(beta - 1): both parts must exceed 2^25 (1 + 2^-20) times that
                const double lim = (double)cnt * 0x1.00001p+71;
                ok = fabs(xr[c]) >= lim && fabs(xi[c]) >= lim;
            }
            const double sc = pow2d(ei + fj - 2 * kOzBeta);  // exact: x is an integer, |x| >= 1 or x = 0
            out = make_float2((float)(xr[c] * sc), (float)(xi[c] * sc));
        }
        if (ok) {
            f.C[idx] = out;
        } else {
            atomicOr(&f.fallback_bits[idx >> 5], 1u << (idx & 31));
            ++fallbacks;
        }
    }
    if (fallbacks != 0) {
        atomicAdd(&f.stats[kStatFallback], fallbacks);
    }
}

// The constants of the moduli, exact in 128-bit integers.
OzCrt make_crt()
{
    OzCrt c{};
    unsigned __int128 M = 1;
    for (int mi = 0; mi < kOzMods; ++mi) {
        M *= (unsigned)kOzModuli[mi];
    }
    const unsigned __int128 mask40 = ((unsigned __int128)1 << 40) - 1;
    auto limbs = [&](unsigned __int128 v, double* out) {
        for (int l = 0; l < 3; ++l) {
            out[l] = (double)(uint64_t)((v >> (40 * l)) & mask40);
        }
    };
    auto inverse = [](int v, int p) {
        for (int u = 1; u < p; ++u) {
            if ((v * u) % p == 1) {
                return u;
            }
        }
        return 0;
    };
    for (int mi = 0; mi < kOzMods; ++mi) {
        const int p = kOzModuli[mi];
        const unsigned __int128 W = M / (unsigned)p;
        const int w2 = (int)((2 * W) % (unsigned)p);
        // W u < M: no reduction
        limbs(W * (unsigned)inverse(w2, p), c.w[mi][0]);
        limbs(W * (unsigned)inverse(w2 * kOzRoots[mi] % p, p), c.w[mi][1]);
    }
    limbs(M, c.m);
    c.k2 = (double)((long double)((unsigned __int128)1 << 80) / (long double)M);
    c.k1 = (double)((long double)((unsigned __int128)1 << 40) / (long double)M);
    return c;
}

// Whether every exact product of order <= kOzMaxN lies within M / 8 (the
// reconstruction's margin).
bool crt_range_ok()
{
    unsigned __int128 M = 1;
    for (int mi = 0; mi < kOzMods; ++mi) {
        M *= (unsigned)kOzModuli[mi];
    }
    const unsigned __int128 bound = (unsigned __int128)(2 * kOzMaxN) << (2 * kOzBeta);
    return bound <= M / 8;
}

}  // namespace

OzLayout oz_layout(int n, uint8_t* base, std::vector<size_t>* guards)
{
    OzLayout L;
    L.kpitch = (n + 63) / 64 * 64;
    L.plane_bytes = (size_t)n * L.kpitch;
    L.y_pad = (n + kOzakiTile - 1) / kOzakiTile * kOzakiTile;
    L.y_plane = (size_t)L.y_pad * L.y_pad;
    const int tiles = L.y_pad / kOzakiTile;
    size_t off = 0;
    const size_t e_off = off;
    off = next_region(off, (size_t)n * 4, guards);
    const size_t f_off = off;
    off = next_region(off, (size_t)n * 4, guards);
    const size_t ca_off = off;
    off = next_region(off, (size_t)n * 4, guards);
    const size_t cb_off = off;
    off = next_region(off, (size_t)n * 4, guards);
    const size_t t_off = off;
    off = next_region(off, (size_t)tiles * tiles, guards);
    const size_t a_off = off;
    off = next_region(off, kOzPlanes * L.plane_bytes, guards);
    const size_t b_off = off;
    off = next_region(off, kOzPlanes * L.plane_bytes, guards);
    const size_t y_off = off;
    off = next_region(off, kOzPlanes * L.y_plane, guards);
    L.bytes = off;
    if (base != nullptr) {
        L.E = reinterpret_cast<int*>(base + e_off);
        L.F = reinterpret_cast<int*>(base + f_off);
        L.CA = reinterpret_cast<int*>(base + ca_off);
        L.CB = reinterpret_cast<int*>(base + cb_off);
        L.tile_ran = base + t_off;
        L.planes_a = reinterpret_cast<int8_t*>(base + a_off);
        L.planes_b = reinterpret_cast<int8_t*>(base + b_off);
        L.residues = base + y_off;
    }
    return L;
}

static const OzCrt& crt_constants()
{
    static const OzCrt crt = make_crt();
    return crt;
}

cudaError_t launch_ozaki_split(cudaStream_t s, int n, int pitch, const ColPanel& panel, const float2* rows_a,
                               const float2* rows_b, const OzLayout& L, const uint8_t* band_a, const uint8_t* band_b)
{
    static const bool range_ok = crt_range_ok();
    if (n > kOzMaxN || !range_ok) {
        return cudaErrorInvalidValue;  // the moduli cover the exact products up to order kOzMaxN
    }
    const int nrows_a = n;  // a later panel may be the first to take a tile of a row band
    ozaki_split_kernel<<<nrows_a + panel.j1 - panel.j0, 256, 0, s>>>(
        n, pitch, rows_a, rows_b, L.planes_a, L.planes_b, L.kpitch, L.plane_bytes, L.E, L.F, L.CA, L.CB, nrows_a,
        panel.j0, band_a, band_b);
    return cudaGetLastError();
}

cudaError_t launch_ozaki_tiles(cudaStream_t s, int n, const ColPanel& panel, const OzLayout& L, uint32_t* stats,
                               uint32_t* fallback_bits, float2* C, int* status, int* launched,
                               const std::function<void(int)>& mark)
{
    const OzCrt& crt = crt_constants();
    int count = 0;
    if (launched != nullptr) {
        *launched = 0;
    }
    if (n > kOzMaxN) {
        return cudaErrorInvalidValue;
    }
    cudaError_t err = cudaSuccess;
    const int tiles = L.y_pad / kOzakiTile;
    {
        CUtensorMap ta, tb;
        const uint64_t dims[3] = {(uint64_t)n, (uint64_t)n, (uint64_t)kOzPlanes};
        const uint64_t strides[2] = {(uint64_t)L.kpitch, (uint64_t)L.plane_bytes};
        const uint32_t box[3] = {(uint32_t)OZ_BK, (uint32_t)OZ_ROWS, 1u};
        if (!encode_tensor_map(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                               L.planes_a) ||
            !encode_tensor_map(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                               L.planes_b)) {
            err = cudaErrorInvalidValue;
        }
        OzParams p{};
        p.kblocks = (n + OZ_BK - 1) / OZ_BK;
        p.tiles = tiles;
        p.tn0 = panel.j0 / OZ_TN;
        p.tn1 = ceil_div(panel.j1, OZ_TN);
        p.tile_ran = L.tile_ran;
        p.residues = L.residues;
        p.y_pad = L.y_pad;
        p.y_plane = L.y_plane;
        for (int mi = 0; mi < kOzMods; ++mi) {
            const int m = kOzModuli[mi];
            p.p[mi] = m;
            p.inv[mi] = (int)((1ULL << 32) / (unsigned)m);
            p.bias[mi] = ((1 << 26) + m - 1) / m * m;
        }
        p.status = status;
        int device = 0, sms = 0;
        if (err == cudaSuccess) {
            err = cudaGetDevice(&device);
        }
        if (err == cudaSuccess) {
            err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        }
        if (err == cudaSuccess) {
            err = cudaFuncSetAttribute(ozaki_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OZ_SMEM);
        }
        if (err == cudaSuccess) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((unsigned)(sms / 2 * 2));  // one pair per two SMs
            cfg.blockDim = dim3(kOzThreads);
            cfg.dynamicSmemBytes = OZ_SMEM;
            cfg.stream = s;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            err = cudaLaunchKernelEx(&cfg, ozaki_pair_kernel, ta, tb, p);
            if (err == cudaSuccess) {
                err = cudaGetLastError();
            }
        }
        mark(++count);
    }
    if (err == cudaSuccess) {
        OzFinish f{};
        f.n = n;
        f.tiles = tiles;
        f.strip0 = panel.j0 / 16;
        f.E = L.E;
        f.F = L.F;
        f.CA = L.CA;
        f.CB = L.CB;
        f.tile_ran = L.tile_ran;
        f.residues = L.residues;
        f.y_pad = L.y_pad;
        f.y_plane = L.y_plane;
        f.stats = stats;
        f.fallback_bits = fallback_bits;
        f.C = C;
        f.crt = crt;
        const int strips = ceil_div(panel.j1, 16) - f.strip0;
        ozaki_crt_kernel<<<dim3((unsigned)strips, (unsigned)(L.y_pad / kCrtRows)), 256, 0, s>>>(f);
        err = cudaGetLastError();
        mark(++count);
    }
    if (launched != nullptr) {
        *launched = count;
    }
    return err;
}

}  // namespace cg3m
