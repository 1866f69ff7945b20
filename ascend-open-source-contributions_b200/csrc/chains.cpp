// chains.cpp -- how long the FP32 chains of a product may be.
//
// A K split is chosen for speed, but it also sets the length of every output's
// FP32 chain, whose rounding error grows with it: as sqrt(terms) on data of
// both signs (uniform: 2.6e-8 sqrt(terms)), as the terms on data of one sign.
// So no time model decides that length alone: the planners take the fastest
// split whose chains are no longer than those of the split found here.  The
// rule is the search of EstimateCgemmCoreWork / SelectCgemm3mDecomposition
// (cgemm_host.cpp:145-200) with fixed costs of its own: it defines a chain
// length, it does not estimate a time, and refitting the planners' time models
// leaves it as it is.
//
// The tensor-core forms accumulate segments of 32, 64 or 128 terms and add the
// segments' sums, so their error does not depend on the K split (384 x 320,
// uniform: split-BF16 x6 4.34e-7 at 1024 terms in one partition, 4.31e-7 in
// eight; 3xTF32 2.90e-7 and 2.79e-7) and is above that of a finely split FP32
// product (2.98e-7 in eight partitions).  Which of the two runs is therefore
// part of the rule as well.
#include <algorithm>
#include <cmath>
#include <limits>

#include "cg3m_internal.h"

namespace cg3m {
namespace {

int k_span(int k, int parts, int g = 16) { return ceil_div(ceil_div(k, g), parts) * g; }

struct Split {
    double cost = 1e300;
    int parts = 1, span = 0;
};

// Outputs a few rows and columns wide over a long K always take eight
// partitions (cgemm_host.cpp:269-273).
bool narrow(int m, int n, int k) { return k >= 1024 && std::min(m, n) <= 16 && std::max(m, n) <= 32; }

// One launch, partitions merged in a cluster: a fixed cost per wave, one per K
// term of a wave and one per K term of every block of the busiest SM.
struct TileCost {
    double fixed, term, shared;
    int blocks;  // per SM
};
constexpr TileCost kOnchip[6] = {{4.96, 183.8, 0.0, 1}, {3.55, 129.2, 0.0, 1}, {3.31, 176.6, 0.0, 1},
                                 {3.29, 118.7, 0.0, 1}, {2.99, 51.4, 59.7, 2}, {2.26, 15.3, 43.7, 3}};

Split onchip_split(int m, int n, int k, bool four_products, int sms, int only_tile, int only_parts)
{
    Split best;
    best.span = k;
    for (int t = four_products ? 1 : 0; t < 6; ++t) {
        if (only_tile >= 0 && t != only_tile) {
            continue;
        }
        const TileCost& c = kOnchip[t];
        const long long tiles = (long long)ceil_div(m, single_tile_bm(t)) * ceil_div(n, single_tile_bn(t));
        const int most = std::min(8, ceil_div(k, 16));  // partitions of 16 terms or more
        for (int q = 1; q <= most; ++q) {
            const int span = q == 1 ? k : k_span(k, q);
            if ((only_parts > 0 && q != only_parts) || (q > 1 && (q - 1) * span >= k)) {
                continue;
            }
            const long long fit = std::max<long long>(1, (long long)kClusterCap[c.blocks - 1][q - 1] * sms / 148);
            const double waves = (double)((tiles + fit - 1) / fit), load = (double)((tiles * q + sms - 1) / sms);
            const double cost = waves * c.fixed +
                                span * 1e-3 * (four_products ? 4.0 / 3.0 : 1.0) * (waves * c.term + load * c.shared) +
                                (q > 1 ? 0.146 * q : 0.0);
            if (cost < best.cost) {
                best = {cost, q, span};
            }
        }
    }
    return best;
}

// Packed planes, 128 x 64 tiles: waves of span + 38 terms and the merge, up to
// eight partitions in a cluster.  The cost in K terms picks the split, the one
// in microseconds meets the other engine's.
Split packed_split(int m, int n, int k, int sms)
{
    const uint64_t tiles = (uint64_t)ceil_div(m, 128) * ceil_div(n, 64);
    auto waves = [&](int parts) {
        if (parts > 1 && parts <= 8) {
            const uint64_t fit = std::max<uint64_t>(1, (uint64_t)kClusterCap[0][parts - 1] * sms / 148);
            return (tiles + fit - 1) / fit;
        }
        return (tiles * parts + sms - 1) / sms;
    };
    uint64_t least = std::numeric_limits<uint64_t>::max();
    Split best;
    for (int parts = 1; parts <= 32; ++parts) {
        const int span = k_span(k, parts);
        if (parts > 1 && span < 64) {
            break;
        }
        if ((parts - 1) * span >= k) {
            continue;
        }
        const uint64_t merge = parts > 8   ? 30 + (uint64_t)(2 * parts + 2) * m * n / 41500
                               : parts > 1 ? (uint64_t)parts
                                           : 0;
        const uint64_t cost = waves(parts) * ((uint64_t)span + 38) + merge;
        if (cost < least) {
            least = cost;
            best.parts = parts;
        }
    }
    if (narrow(m, n, k)) {
        best.parts = std::max(best.parts, 8);
    }
    best.span = k_span(k, best.parts);
    while (best.parts > 1 && (best.parts - 1) * best.span >= k) {
        --best.parts;
        best.span = k_span(k, best.parts);
    }
    if (best.parts == 1) {
        best.span = k;
    }
    best.cost = 1.64 + 0.199e-6 * 20.0 * ((double)m * k + (double)k * n) +
                0.1205 * (double)waves(best.parts) * (best.span + 38) +
                (best.parts > 8 ? 3.53 : best.parts > 1 ? 0.1205 * best.parts : 0.0);
    return best;
}

// Cost of the tensor-core call the rule compares with plain FP32: the split
// over 128 x 128 tiles first, then pack and waves in microseconds.
double tensor_cost(int m, int n, int k, int form, int sms)
{
    const uint64_t tiles = (uint64_t)ceil_div(m, 128) * ceil_div(n, 128);
    int parts = 1;
    if (tiles < (uint64_t)sms) {
        uint64_t least = std::numeric_limits<uint64_t>::max();
        const int most = std::min(64, (int)std::max<uint64_t>(4, 2 * (uint64_t)sms / std::max<uint64_t>(tiles, 1)));
        for (int q = 1; q <= most; ++q) {
            const int span = k_span(k, q, 64);
            if ((q - 1) * span >= k || (q > 4 && span < 256)) {
                continue;
            }
            const uint64_t waves = (tiles * q + sms - 1) / sms;
            const uint64_t cost = waves * std::min(m, 128) * std::min(n, 128) * (uint64_t)(span + 16) +
                                  (q > 1 ? (uint64_t)q * m * n / sms : 0);
            if (cost < least) {
                least = cost;
                parts = q;
            }
        }
    }
    int span = k_span(k, parts, 64);
    while (parts > 1 && (parts - 1) * span >= k) {
        --parts;
        span = k_span(k, parts, 64);
    }
    if (parts == 1) {
        span = k;
    }
    const uint64_t pairs = m > 128 ? (uint64_t)ceil_div(m, 256) * ceil_div(n, 128) : (uint64_t)ceil_div(n, 128);
    const double waves = (double)((pairs * parts + sms - 1) / sms), elems = (double)m * k + (double)k * n;
    if (form == CG3M_FORM_TF32X3) {
        return 11.80 + 0.1374 * elems * 32e-6 + 0.11003 * waves * span + (parts > 1 ? 1.25 : 0.0);
    }
    return 13.27 + 0.1055 * elems * 44e-6 + 0.08315 * (form == CG3M_FORM_BF16X9 ? 1.5 : 1.0) * waves * span;
}

// The on-chip family's batches: tiles by padded work, larger ones preferred,
// and partitions for tasks above a quarter of an SM's work.
constexpr double kTilePreference[6] = {1.0, 0.85, 0.8, 0.8, 0.65, 0.45};

}  // namespace

ChainLimit chain_limit(const Problem& p, int form, int engine, int tile, int sm_count)
{
    const int sms = sm_count > 0 ? sm_count : 148;
    const Split packed = packed_split(p.m, p.n, p.k, sms);
    const Split onchip = onchip_split(p.m, p.n, p.k, false, sms, engine == 2 ? tile : -1,
                                      engine != 2 && narrow(p.m, p.n, p.k) ? 8 : 0);
    ChainLimit out;
    out.onchip = engine == 2 || (engine == 0 && onchip.cost < packed.cost);
    out.span = out.onchip ? onchip.span : packed.span;
    out.parts = out.onchip ? onchip.parts : packed.parts;
    out.tensor = form != CG3M_FORM_FP32 &&
                 !(std::min(onchip.cost, packed.cost) * 1.1 < tensor_cost(p.m, p.n, p.k, form, sms));
    return out;
}

int onchip_chain_limit(int m, int n, int k, int mode, int sm_count)
{
    return onchip_split(m, n, k, mode != 0, sm_count > 0 ? sm_count : 148, -1, 0).span;
}

BatchChains::BatchChains(int mode, int sm_count) : first_tile(mode != 0 ? 1 : 0), sms(std::max(sm_count, 1)) {}

double BatchChains::task_work(int m, int n, int k, long long* tiles) const
{
    double best = 1e300, task = 0.0;
    for (int t = first_tile; t < 6; ++t) {
        const double one = (double)single_tile_bm(t) * single_tile_bn(t) * (k + 16) / kTilePreference[t];
        const long long count = (long long)ceil_div(m, single_tile_bm(t)) * ceil_div(n, single_tile_bn(t));
        if (one * count < best) {
            best = one * count;
            task = one;
            *tiles = count;
        }
    }
    return task;
}

void BatchChains::add(int m, int n, int k, int count)
{
    long long tiles = 0;
    const double task = task_work(m, n, k, &tiles);
    total += task * tiles * count;
}

int BatchChains::parts(int m, int n, int k, int most) const
{
    if (most <= 1 || k < 256) {
        return 1;
    }
    long long tiles = 0;
    const int want = (int)std::min(1e6, std::ceil(task_work(m, n, k, &tiles) / (0.25 * (total / sms))));
    int q = std::max(1, std::min({want, most, k / 128}));
    while (q > 1 && (q - 1) * k_span(k, q) >= k) {
        --q;
    }
    return q;
}

}  // namespace cg3m
