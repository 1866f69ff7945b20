// planner.cpp -- argument validation and path / tile / K-split selection.
//
// Reference: ValidateCgemmParams and ValidateCgemmPointers
// (blas/gemm/arch35/cgemm_host.cpp:589-634,687-699), LaunchComplexGemm
// (:701-730), CalculateCgemmWorkspaceSizes (:228-285) with
// SelectCgemmAccumulationTile (:130), EstimateCgemmCoreWork (:145),
// SelectCgemmProductTile (:157), SelectCgemm3mDecomposition (:174) and the
// rounding gate (:234-238), AllocateCgemmWorkspace (:326-360).
//
// The validation order, statuses and quick returns are the reference's.  The
// tile/K-split policy keeps the reference's structure -- a joint search over
// output tile x K partitions that minimises the busiest core's work times
// (span + 16), with a forced deeper split for narrow long-K outputs -- but its
// capacities are the B200's: the "cores" are SM slots (148 SMs x resident CTAs
// of the tile), the tiles are this kernel's, and the partition bound scales
// with how few tiles there are, since a 148-SM part needs far more
// independent tasks than a 1-4-way split of a handful of tiles provides.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>

#include <vector>

#include "cg3m_internal.h"

namespace cg3m {

static bool is_op(int op, bool allow_conj_only)
{
    return op == CG3M_OP_N || op == CG3M_OP_T || op == CG3M_OP_C || (allow_conj_only && op == CG3M_OP_R);
}

cg3mStatus_t validate(int transa, int transb, int m, int n, int k, const cg3mComplex* alpha, const void* A, int lda,
                      const void* B, int ldb, const cg3mComplex* beta, const void* C, int ldc, bool allow_conj_only,
                      int* action)
{
    *action = 0;
    // Enum errors are reported as INVALID_VALUE by the 3m entry (cgemm_host.cpp:713).
    if (!is_op(transa, allow_conj_only) || !is_op(transb, allow_conj_only)) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    if (m < 0 || n < 0 || k < 0) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    const bool normal_a = transa == CG3M_OP_N || transa == CG3M_OP_R;
    const bool normal_b = transb == CG3M_OP_N || transb == CG3M_OP_R;
    if (lda < std::max(1, normal_a ? m : k)) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    if (ldb < std::max(1, normal_b ? k : n)) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    if (ldc < std::max(1, m)) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    if (alpha == nullptr || beta == nullptr) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    if (m == 0 || n == 0) {
        return CG3M_STATUS_SUCCESS;  // quick return after validation (cgemm_host.cpp:715)
    }
    const bool alpha_zero = alpha->real == 0.0f && alpha->imag == 0.0f;
    if (C == nullptr) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    if (!alpha_zero && k > 0 && (A == nullptr || B == nullptr)) {
        return CG3M_STATUS_INVALID_VALUE;
    }
    if (k == 0 || alpha_zero) {
        const bool beta_one = beta->real == 1.0f && beta->imag == 0.0f;
        *action = beta_one ? 0 : 1;  // cgemm_host.cpp:639
        return CG3M_STATUS_SUCCESS;
    }
    *action = 2;
    return CG3M_STATUS_SUCCESS;
}

namespace {

struct TileChoice {
    int bm, bn;
    int slots_per_sm;  // resident CTAs per SM of this tile's kernel
};

// FP32 FFMA kernel tile (gemm_fp32.cu).  The kernel also instantiates 64 x 64,
// 64 x 32 and 32 x 32 tiles, but measured on B200 they run at about a third of
// the 128 x 64 tile's per-SM FFMA rate (short pipelines, few warps), so the
// planner splits K over 128 x 64 tiles instead (512^3: 64 x 32 x 3 parts
// 62.9 us, 128 x 64 x 4 parts 38.8 us; 1024^3: 306 vs 174 us).
const TileChoice kFp32Tiles[] = {{128, 64, 1}};
// Cost of one wave of 128 x 64 FP32 tiles in K terms of that tile (0.111 us
// per term): a fixed part (pipeline fill, epilogue, wave launch; 56 terms in the
// microsecond model below) plus the span; the split-K merge costs about 30 terms
// plus the partial planes it reads.  Beyond kShortChain terms splits are chosen
// with a fixed part of 38 terms: as fast (75 timed shapes, 0.1 %), and finer
// where the two differ (756 x 344 x 3425: 12 partitions 135.6 us, 3 149.8), which
// keeps chains short: a chain's relative error grows as 2.6e-8 sqrt(terms)
// (uniform data: 8.3e-7 at 1024 terms, 1.03e-6 at 1646, 1.43e-6 at 3125).
constexpr uint64_t kFp32WaveFixed = 56, kLongWaveFixed = 38;
constexpr uint64_t kMergeFixed = 30;
constexpr uint64_t kMergeFloatsPerTerm = 41500;
// With 2..8 partitions the partitions of a tile form one thread-block cluster
// and merge through distributed shared memory inside the GEMM (no merge
// kernel, no partial planes): waves then hold as many clusters as fit at once
// (kClusterCap, one block per SM), and the merge costs about one K term per
// partition.
constexpr int kClusterMergeMax = 8;

uint64_t fp32_waves(uint64_t tiles, int parts, int sm_count)
{
    if (parts > 1 && parts <= kClusterMergeMax) {
        const uint64_t cap = std::max<uint64_t>(1, (uint64_t)kClusterCap[0][parts - 1] * sm_count / 148);
        return (tiles + cap - 1) / cap;
    }
    return (tiles * parts + sm_count - 1) / sm_count;
}
// The same costs in microseconds for the whole packed call (pack kernel over
// op(A) and op(B) -- 8 bytes read, 12 written per element -- GEMM waves, merge),
// fitted on B200 to 460 timed (shape, partitions) calls (median error 1.5 %).
constexpr double kPackedFixedUs = 2.91;
constexpr double kPackedUsPerMB = 0.1323;
constexpr double kPackedUsPerTerm = 0.1113;
constexpr double kPackedUsPerPart = 0.0857;
constexpr double kMergeLaunchUs = 2.5;
// The one-launch engine has to look faster by this much: its model errs by up
// to 10 % where the two engines meet, the packed one's by 3 %.
constexpr double kSingleMargin = 1.06;
constexpr double kSingleGain = 0.7;
// Tensor-core kernel tile (gemm_tc.cu): 128 x 128, one CTA per SM (TMEM).
const TileChoice kTcTiles[] = {{128, 128, 1}};

// kSpan = ceil(ceil(k/g)/parts)*g (cgemm_host.cpp:274-275 with g = 16).  The
// granule g is the GEMM kernel's K-tile so that only the last partition has a
// ragged tail: 16 for the FP32 kernel, 64 elements (one 128-byte row of the
// widest split plane) for the tensor-core kernel.
int k_span(int k, int parts, int g = 16)
{
    return ceil_div(ceil_div(k, g), parts) * g;
}

double packed_time_us(const Problem& p, int parts, int span, uint64_t tiles, int sm_count)
{
    const uint64_t waves = fp32_waves(tiles, parts, sm_count);
    const double bytes = ((double)p.m * p.k + (double)p.k * p.n) * 20.0;
    double us = kPackedFixedUs + kPackedUsPerMB * bytes * 1e-6 + kPackedUsPerTerm * (double)waves * (span + kFp32WaveFixed);
    if (parts > kClusterMergeMax) {
        us += kMergeLaunchUs;
    } else if (parts > 1) {
        us += kPackedUsPerPart * parts;
    }
    return us;
}

// Tensor-core call in microseconds, fitted on B200 to 600 timed (shape, form,
// K split) calls of up to 3000 x 3000 x 4000 (median error 2 %; the split it
// picks, or plain FP32, costs a mean 0.1 % over the best of each shape): the
// pack per 5.5 MB it moves, waves of CTA-pair tiles (256 x 128 on two SMs; 128 x
// 128 on one for a single row tile) at a fixed part and a time per K term that
// depends on the accumulation segment, and the merge, in the tile's cluster or
// per 10 MB of partials and output.
struct TcCost {
    double base_us, pack_us, wave_us, cluster_us, merge_us, term_us[3];  // segments of >= 128, 64, 32 terms
};
constexpr TcCost kTcCost[3] = {{3.85, 1.131, 5.81, 2.96, 0.929, {0.0409, 0.0521, 0.0711}},   // 3xTF32
                               {3.57, 1.132, 6.82, 2.24, 0.947, {0.0394, 0.0523, 0.0523}},   // split-BF16 x6
                               {4.32, 1.162, 6.40, 2.16, 0.990, {0.0563, 0.0632, 0.0632}}};  // split-BF16 x9

uint64_t tc_tiles(const Problem& p)
{
    return p.m > 128 ? (uint64_t)ceil_div(p.m, 256) * ceil_div(p.n, 128) : (uint64_t)ceil_div(p.n, 128);
}

// K splits merged on chip: only when every cluster of 2 x parts CTAs is
// resident at once.  A grid that one wave holds as loose CTAs but not as
// clusters runs a second wave, which costs more than the merge launch it saves
// (1.3-1.6x on 128..144-CTA grids).
bool tc_cluster_merge(const Problem& p, int parts, int sm_count)
{
    if (p.m <= 128 || parts < 2 || parts > 4) {
        return false;
    }
    const uint64_t cap = std::max<uint64_t>(1, (uint64_t)kClusterCap[0][2 * parts - 1] * sm_count / 148);
    return tc_tiles(p) <= cap;
}

double tc_time_us(const Problem& p, int form, int segment, int parts, int span, int sm_count, int count = 1)
{
    const TcCost& c = kTcCost[form - CG3M_FORM_TF32X3];
    const uint64_t slots = std::max(1, p.m > 128 ? sm_count / 2 : sm_count);
    const bool merged = tc_cluster_merge(p, parts, sm_count) && count == 1;
    const double waves = merged ? 1.0 : (double)((tc_tiles(p) * parts * count + slots - 1) / slots);
    const double mb = ((double)p.m * p.k + (double)p.k * p.n) * count * (form == CG3M_FORM_TF32X3 ? 32e-6 : 26e-6);
    const double terms = (double)align_up((size_t)span, 64);
    double us = c.base_us + c.pack_us * mb / 5.5 +
                waves * (c.wave_us + terms * c.term_us[segment >= 128 ? 0 : segment >= 64 ? 1 : 2]);
    if (merged) {
        us += c.cluster_us;
    } else if (parts > 1) {
        us += c.merge_us * (double)(16 * parts + 16) * p.m * p.n * 1e-7;
    }
    return us;
}

// K terms accumulated in TMEM between round-to-nearest merges.
int tc_segment(const cg3mOptions& opts, int k)
{
    return opts.tc_segment > 0 ? opts.tc_segment : (k >= 2048 ? 128 : k > 1024 ? 64 : 32);
}

}  // namespace

double batch_tc_time_us(const Problem& p, const cg3mOptions& opts, int sm_count, int count)
{
    return tc_time_us(p, opts.form, tc_segment(opts, p.k), 1, p.k, sm_count, count);
}

bool batch_tc_plan(const Problem& p, const cg3mOptions& opts, int sm_count, int count, Plan* plan)
{
    cg3mOptions o = opts;
    o.engine = 1;
    o.k_partitions = 1;
    o.rounding = CG3M_ROUNDING_OFF;
    if (p.m <= 128 || opts.form == CG3M_FORM_FP32 || !make_plan(p, o, sm_count, plan)) {
        return false;
    }
    const size_t elem = opts.form == CG3M_FORM_TF32X3 ? 4 : 2;
    plan->planes_a_off = 0;
    plan->planes_b_off = align_up(plan->plane_a_elems * elem * plan->planes * count, kRegionAlign);
    plan->total = align_up(plan->planes_b_off + plan->plane_b_elems * elem * plan->planes * count, kRegionAlign);
    plan->guards = 0;
    return true;
}

bool make_plan(const Problem& p, const cg3mOptions& opts, int sm_count, Plan* plan, int max_chain)
{
    Plan out{};
    out.action = 2;
    out.form = opts.form;
    out.unit = p.ar == 1.0f && p.ai == 0.0f && p.br == 0.0f && p.bi == 0.0f;
    // Tensor-core forms restart their TMEM accumulators every `tc_segment` K
    // terms and merge segments with round-to-nearest FP32 adds.  The truncation
    // error of one segment grows with its length, while the plain FP32 form's
    // error grows with sqrt(K); these lengths keep the tensor-core error at or
    // below the plain form's (measured on data with a 2^16 dynamic range in the
    // imaginary parts), at the cost of more merges for short K.
    out.tc_segment = tc_segment(opts, p.k);
    out.beta_zero = p.br == 0.0f && p.bi == 0.0f;
    if (sm_count <= 0) {
        sm_count = 148;
    }
    const bool tc = opts.form != CG3M_FORM_FP32;
    if (opts.form < CG3M_FORM_FP32 || opts.form > CG3M_FORM_BF16X9) {
        return false;  // the host-buffer entry point plans before any call checks its options
    }
    if (opts.engine < 0 || opts.engine > 2 || opts.onchip_tile < 0 || opts.onchip_tile > 6) {
        return false;
    }

    // Rounding-correction gate (cgemm_host.cpp:234-238).
    out.rounding = opts.rounding == CG3M_ROUNDING_AUTO && out.unit && p.m == p.n && p.n == p.k && p.k >= 2048 &&
                   p.k <= 4096 && p.lda == p.m && p.ldb == p.m && p.ldc == p.m;

    // ---- engine 2: one launch, K partitions merged in a cluster -----------------
    if (opts.engine == 2) {
        if (tc || out.rounding || opts.k_partitions > 8) {
            return false;
        }
        int parts = opts.k_partitions;
        while (parts > 1 && (parts - 1) * k_span(p.k, parts) >= p.k) {
            --parts;
        }
        int tile = 0;
        const int longest =
            parts > 0 ? p.k : chain_limit(p, opts.form, 2, opts.onchip_tile - 1, sm_count).span;
        out.est_us = plan_single(p.m, p.n, p.k, 0, sm_count, opts.onchip_tile - 1, parts, longest, &tile, &parts);
        out.engine = 2;
        out.onchip_tile = tile;
        out.tile_m = single_tile_bm(tile);
        out.tile_n = single_tile_bn(tile);
        out.parts = parts;
        out.span = parts > 1 ? k_span(p.k, parts) : p.k;
        out.total = 0;
        *plan = out;
        return true;
    }

    // The chains the planner may choose; a tensor-core call whose form the rule
    // rules out runs as plain FP32.
    ChainLimit limit;
    int longest = p.k;
    if (!out.rounding && opts.k_partitions <= 0) {
        if (max_chain > 0) {
            longest = max_chain;
        } else if (!tc || opts.engine == 0) {
            limit = chain_limit(p, opts.form, opts.engine, -1, sm_count);
            longest = limit.span;
        }
        if (tc && opts.engine == 0 && !limit.tensor) {
            cg3mOptions fo = opts;
            fo.form = CG3M_FORM_FP32;
            fo.rounding = CG3M_ROUNDING_OFF;
            return make_plan(p, fo, sm_count, plan);
        }
    }

    // ---- tile x K-partition search -------------------------------------------
    const TileChoice* tiles = tc ? kTcTiles : kFp32Tiles;
    const int granule = tc ? 64 : 16;
    const uint64_t default_tiles = (uint64_t)ceil_div(p.m, tiles[0].bm) * ceil_div(p.n, tiles[0].bn);
    TileChoice best_tile = tiles[0];
    int best_parts = 1;
    bool packed = true;
    if (opts.k_partitions > 0) {
        best_parts = std::min(opts.k_partitions, 64);
    } else if (!tc && !out.rounding) {
        // FP32: waves of 128 x 64 tiles at (span + fixed) each, plus the merge
        // (EstimateCgemmCoreWork's busiest-core work with measured B200 costs).
        const size_t rows = align_up((size_t)p.m, 32), cols = align_up((size_t)p.n, 32);
        const size_t planes = 12 * (rows + cols) * (size_t)p.k, partial = 8 * rows * (size_t)p.n;
        // Workspace: no call takes more than a default workspace that did with less
        // by the rule's split; splits finer than a larger one's may add an eighth.
        const auto bytes = [&](int parts) { return planes + (parts > kClusterMergeMax ? parts * partial : 0); };
        size_t room = std::numeric_limits<size_t>::max();
        if (max_chain <= 0) {
            const size_t rule = limit.onchip ? 0 : bytes(limit.parts);
            room = std::max(kPlanWorkspace, rule + (rule > kDefaultWorkspaceBytes ? rule / 8 : 0));
        }
        const uint64_t fixed = p.k > kShortChain ? kLongWaveFixed : kFp32WaveFixed;
        uint64_t best = std::numeric_limits<uint64_t>::max();
        for (int parts = 1; parts <= 64; ++parts) {
            const int span = k_span(p.k, parts, granule);
            if (parts > 1 && span < 64) {
                break;
            }
            if ((parts - 1) * span >= p.k || (parts > 1 ? span : p.k) > longest || bytes(parts) > room) {
                continue;
            }
            const uint64_t waves = fp32_waves(default_tiles, parts, sm_count);
            const uint64_t gemm = waves * ((uint64_t)span + fixed);
            const uint64_t merge =
                parts > kClusterMergeMax ? kMergeFixed + (uint64_t)(2 * parts + 2) * p.m * p.n / kMergeFloatsPerTerm
                : parts > 1              ? (uint64_t)parts
                                         : 0;
            // Beyond 32 partitions for a clear gain only (54 x 460 x 42520: 18
            // partitions 372 us, 36 381; 128 x 128 x 65536: 32 295, 64 186).
            const uint64_t cost = (gemm + merge) * (parts > 32 ? 21 : 20);
            if (cost < best) {
                best = cost;
                best_parts = parts;
            }
        }
        packed = best != std::numeric_limits<uint64_t>::max();
    } else if (!out.rounding) {
        // Tensor-core forms: the split with the least estimated time
        // (SelectCgemm3mDecomposition's joint search, :174-200, over one tile).
        // Partitions keep >= 64 K terms, one K-block of the split planes (546 x 739 x
        // 204, 3xTF32: four of 64 20.0 us, two of 128 23.9), >= 256 beyond the
        // reference's four.
        double best = std::numeric_limits<double>::max();
        for (int parts = 1; parts <= 64; ++parts) {
            const int span = k_span(p.k, parts, granule);
            if (parts > 1 && ((parts - 1) * span >= p.k || span < (parts > 4 ? 256 : 64))) {
                continue;
            }
            const double us =
                tc_time_us(p, opts.form, out.tc_segment, parts, parts > 1 ? span : p.k, sm_count);
            if (us < best) {
                best = us;
                best_parts = parts;
            }
        }
    }
    // Narrow long-K outputs force >= 8 partitions (cgemm_host.cpp:269-273).
    if (opts.k_partitions <= 0 && !tc && p.k >= 1024 && std::min(p.m, p.n) <= 16 && std::max(p.m, p.n) <= 32) {
        best_parts = std::max(best_parts, 8);
    }
    // The tensor-core forms' rounding pass runs its products over the whole K:
    // the risk plane needs the whole chain and the form's products on the
    // tiles the exact recompute does not take run unsplit.
    if (tc && out.rounding) {
        best_parts = 1;
    }
    out.tile_m = best_tile.bm;
    out.tile_n = best_tile.bn;
    out.parts = best_parts;
    out.span = k_span(p.k, best_parts, granule);
    while (out.parts > 1 && (out.parts - 1) * out.span >= p.k) {
        --out.parts;
        out.span = k_span(p.k, out.parts, granule);
    }
    if (out.parts == 1) {
        out.span = p.k;
    }

    // ---- engine (FP32 form without the rounding pass) ---------------------------
    // The one-launch engine skips the pack kernel and the merge kernel; it
    // wins on small and latency-bound shapes, the packed engine's faster FFMA
    // tile on large ones.  Both time models are fitted on B200.
    if (!tc && !out.rounding && opts.engine == 0 && (opts.k_partitions <= 0 || out.parts <= 8)) {
        const bool narrow = p.k >= 1024 && std::min(p.m, p.n) <= 16 && std::max(p.m, p.n) <= 32;
        const int forced = opts.k_partitions > 0 ? out.parts : narrow ? 8 : 0;
        int tile = 0, parts = 0;
        double single = plan_single(p.m, p.n, p.k, 0, sm_count, -1, forced, longest, &tile, &parts);
        const int single_span = parts > 1 ? k_span(p.k, parts) : p.k;
        if (single_span > longest) {
            single = 1e300;
        }
        out.est_us = packed ? packed_time_us(p, out.parts, out.span, default_tiles, sm_count) : 1e300;
        // Within the limit, chains up to twice as long as the packed split's (1.4
        // times the error) or short, or a clear gain: narrow outputs pad the packed
        // tile several times over (25 x 1025 x 59274: 8 partitions in one launch
        // 438 us, 26 packed 1078).
        const bool chains = !packed || opts.k_partitions > 0 || single_span <= std::max(kShortChain, 2 * out.span) ||
                            single < kSingleGain * out.est_us;
        if (single < 1e300 && chains && (!packed || single * kSingleMargin < out.est_us)) {
            out.est_us = single;
            out.engine = 2;
            out.onchip_tile = tile;
            out.tile_m = single_tile_bm(tile);
            out.tile_n = single_tile_bn(tile);
            out.parts = parts;
            out.span = parts > 1 ? k_span(p.k, parts) : p.k;
            out.total = 0;
            *plan = out;
            return true;
        }
    }

    if (!packed) {
        return false;  // max_chain below every split's chains
    }

    // ---- tensor-core forms on small shapes ---------------------------------------
    // A tensor-core call carries a fixed cost of 10-11 us (pack, TMEM set-up,
    // pipeline fill; kTcCost) that the FP32 engines do not.  Where an FP32 plan is
    // faster by more than the tensor-core model errs, the call runs that plan in
    // plain FP32 and reports form FP32: one whose chains are no longer than the
    // segments the form accumulates, which leaves an error no larger than the
    // form's (256 terms, segments of 32, uniform: FP32 chains of 32 1.62e-7,
    // 3xTF32 2.67e-7, split-BF16 4.27e-7).  engine 1 (or a forced K split) keeps
    // the tensor-core path.
    if (tc) {
        out.est_us = tc_time_us(p, opts.form, out.tc_segment, out.parts, out.span, sm_count);
    }
    if (tc && !out.rounding && opts.engine == 0 && opts.k_partitions <= 0) {
        cg3mOptions fo = opts;
        fo.form = CG3M_FORM_FP32;
        fo.rounding = CG3M_ROUNDING_OFF;
        Plan fp;
        if (make_plan(p, fo, sm_count, &fp, out.tc_segment) && fp.est_us * 1.05 < out.est_us) {
            *plan = fp;
            return true;
        }
    }

    // ---- workspace layout -----------------------------------------------------
    const bool kmajor = tc;
    int splits = 1;
    size_t elem = 4;
    if (opts.form == CG3M_FORM_TF32X3) {
        splits = 2;
    } else if (opts.form == CG3M_FORM_BF16X6 || opts.form == CG3M_FORM_BF16X9) {
        splits = 3;
        elem = 2;
    }
    out.planes = 3 * splits;
    if (kmajor) {
        // [mn][k] planes: K padded so every row starts on a 128-byte boundary.
        const int kp = (int)align_up((size_t)p.k, 128 / elem);
        out.pitch_a = kp;
        out.pitch_b = kp;
        out.plane_a_elems = (size_t)p.m * kp;
        out.plane_b_elems = (size_t)p.n * kp;
    } else {
        out.pitch_a = (int)align_up((size_t)p.m, 32);
        out.pitch_b = (int)align_up((size_t)p.n, 32);
        out.plane_a_elems = (size_t)out.pitch_a * p.k;
        out.plane_b_elems = (size_t)out.pitch_b * p.k;
    }
    size_t off = 0;
    std::vector<size_t> guards;
    out.planes_a_off = off;
    off = next_region(off, out.plane_a_elems * elem * out.planes, &guards);
    out.planes_b_off = off;
    off = next_region(off, out.plane_b_elems * elem * out.planes, &guards);
    out.partial_pitch = (int)align_up((size_t)p.m, 32);
    out.partial_plane_elems = (size_t)out.partial_pitch * p.n;
    // K splits merged on chip through the tile's cluster: the FP32 GEMM (up to 8
    // partitions) and the tensor-core CTA-pair kernel (up to 4, two CTAs each).
    out.cluster_merge = !out.rounding && out.parts > 1 &&
                        (tc ? tc_cluster_merge(p, out.parts, sm_count)
                            : (out.parts <= kClusterMergeMax && out.tile_m == 128 && out.tile_n == 64));
    out.partial_off = off;
    if (out.parts > 1 && !out.cluster_merge) {
        off = next_region(off, out.partial_plane_elems * 4 * 2 * out.parts, &guards);
    }
    out.round_off = off;
    if (out.rounding) {
        std::vector<size_t> inner;
        off = next_region(off, rounding_bytes(p.n, out.form, &inner), &guards);  // layout in rounding.cu
        for (size_t g : inner) {
            guards.push_back(out.round_off + g);
        }
    }
    out.total = off;
    if (guards.size() > (size_t)Plan::kMaxGuards) {
        return false;
    }
    out.guards = (int)guards.size();
    for (size_t i = 0; i < guards.size(); ++i) {
        out.guard_off[i] = guards[i];
    }
    *plan = out;
    return true;
}

}  // namespace cg3m
