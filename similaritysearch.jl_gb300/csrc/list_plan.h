// How a list scan (tc_list.cu) is split over the database, the queries and the
// memory of its lists (host code, no CUDA).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <numeric>

#ifdef __CUDACC__
#define SSG_PLAN_HD __host__ __device__
#else
#define SSG_PLAN_HD
#endif

namespace ssg {

constexpr int kListMaxCap = 1024;  // entries of one list at most
constexpr int kListSlack = 160;    // entries beyond kk that every list has room for at least
constexpr int kListSegs = 2;       // lists of a query per split
// What a pass over a chunk of the queries may take: lists, minima, bounds, counts.
constexpr size_t kListBudget = size_t(1) << 30;
// Minima per query at most: those of the smallest chunk (256 queries) stay
// within half the budget.  Reached from 4e8 rows on.
constexpr int64_t kListMaxGroups = int64_t(kListBudget / 2 / (256 * 4));

// Database splits per query tile for a kernel with `cap` resident CTAs on the
// device: qctas * s CTAs run in ceil(qctas * s / cap) waves, each CTA scanning
// 1/s of the database, so the scan takes ~ waves(s) / s.  Minimise that, with
// a 1% charge per extra split for the wider merge, over s <= max_s.
inline double split_charge(int64_t s) { return 1.0 + 0.01 * double(s - 1); }
inline int64_t wave_splits(int64_t qctas, int64_t cap, int64_t max_s) {
    qctas = std::max<int64_t>(1, qctas);
    const int64_t hi = std::max<int64_t>(1, std::min<int64_t>(max_s, 4 * ((cap + qctas - 1) / qctas)));
    int64_t best = 1;
    double best_cost = 1e300;
    for (int64_t sp = 1; sp <= hi; ++sp) {
        const double waves = double((qctas * sp + cap - 1) / cap);
        const double cost = waves / double(sp) * split_charge(sp);
        if (cost < best_cost * (1.0 - 1e-9)) { best_cost = cost; best = sp; }
    }
    return best;
}

// Which rows the seed's sample holds: units of one tile's height, put together
// from atoms of 8 rows of as many tiles as a tile has atoms, q tiles apart
// over the whole database.  Neighbouring rows are often alike (stored cluster
// by cluster, duplicates): a sample of whole tiles of 128 rows misses most
// clusters, and the bound is then the distance of many others (2,048 queries x
// 1e6 BF16 rows of 96 stored in clusters of 100, k = 10: 1,659 us, in units
// 1,017; allknn of 40,000 split rows of 64, likewise: 4.9 ms and 2.3).
// A group of columns whose minimum the seed keeps is the rows at two of the
// eight places of their atoms, of atoms far apart: alike rows count as several,
// and not as the one that is nearest, though they lie together.  So wide tiles
// are visited a golden section of the sample apart, one's two units half of it
// (groups of whole chunks of columns: allknn of 37,705 rows of 11, Cosine, in
// clusters of 37, k = 11, 3,491 us, so 1,140; of 24,481 BF16 rows of 22 in
// clusters of 139 923 and 423; rows in random order the same).
struct SampleRows {
    int64_t q = 0;      // tiles between the atoms of a unit
    uint64_t step = 0;  // units per sampled unit, 32 fractional bits
    int samples = 1, stride = 1;  // wide tiles; wide tile w's first unit is w * stride mod samples
};
inline SampleRows sample_rows(int64_t n, int tile_rows, int64_t samples) {
    const int atoms = tile_rows / 8;
    SampleRows s;
    s.q = n / tile_rows / atoms;
    s.step = (uint64_t(s.q * atoms) << 32) / uint64_t(2 * samples);
    s.samples = int(samples);
    s.stride = std::max(1, int(0.618034 * double(samples)));
    while (std::gcd(s.stride, s.samples) != 1) ++s.stride;
    return s;
}
// The first of the two units of wide tile w; the other one is s.samples further on.
SSG_PLAN_HD inline int sample_first(const SampleRows &s, int64_t w) {
    return int(uint64_t(w) * uint64_t(s.stride) % uint64_t(s.samples));
}
SSG_PLAN_HD inline int sample_next(const SampleRows &s, int v) {
    v += s.stride;
    return v >= s.samples ? v - s.samples : v;
}
// The v-th of the sample's units: its first tile and its line of atoms.
SSG_PLAN_HD inline void sample_unit(const SampleRows &s, int atoms, int64_t v, int64_t *tile, int *line) {
    const int64_t e = int64_t((uint64_t(v) * s.step) >> 32);
    *tile = e / atoms;
    *line = int(e % atoms);
}
// The row at place c of a unit.
SSG_PLAN_HD inline int64_t sample_row(const SampleRows &s, int tile_rows, int64_t tile, int line, int c) {
    return (tile + c / 8 * s.q) * tile_rows + line * 8 + c % 8;
}

// One call: m queries, kk candidates each, over n rows in wide tiles of `wide`
// rows, on a device that holds `pairs` CTA pairs.
struct ListCall {
    int64_t n = 0, m = 0;
    int kk = 0;
    int64_t wide = 256;
    bool streamed = false;  // rows in 128-byte K-blocks
    int64_t splits = 0;     // splits asked for (0: chosen here)
    int64_t pairs = 1;
};

struct ListPlan {
    int splits = 0, cap = 0, groups = 0, per_tile = 0, keys = 0;
    int64_t samples = 0;
    int64_t chunk = 0;  // queries per pass
};

// Device bytes per query of a chunk.
inline size_t list_query_bytes(const ListPlan &p) {
    const size_t segs = size_t(kListSegs) * size_t(p.splits);
    return segs * (size_t(p.cap) * 8 + 4) + size_t(p.groups) * 4 + 4;
}

// False when the scan does not apply: too few whole wide tiles for a bound
// (four groups of columns per candidate from at most a quarter of the
// database), or lists longer than a list's room.
inline bool list_plan(const ListCall &c, ListPlan *p) {
    const int kk = c.kk;
    const int64_t n_full = c.n / c.wide, n_wide = (c.n + c.wide - 1) / c.wide;
    if (kk > (kListMaxCap - 64) / 2 || n_full < 8) return false;
    // The sample costs its share of a scan, and a bound from one row in f
    // lets about 1.2 kk f candidates per query through.  Where the scan waits
    // for its epilogue (sketches, rows in 64-byte K-blocks) a sixth: 10,000
    // queries x 2e6 sketches 6.87 ms (an eighth 7.26, a quarter 6.85), 2,048 x
    // 1e6 BF16 rows of 96 460 us (476, 460), 1,000 x 1e5 split rows of 128 164
    // (178, 164).  Long rows' MMAs hide more of the appends: an eighth, 4,096 x
    // 2e6 FP8 rows of 768 4.71 ms (a sixth 4.84, a twelfth 4.77).  With few
    // queries the scan reads memory and hardly appends: a twelfth, 64 queries
    // x 2e6 sketches 254 us (a sixteenth 262, an eighth 259).
    const int64_t f = c.m <= 256 ? 12 : c.streamed ? 8 : 6;
    // four minima per candidate, from groups of 128, 32 or (small databases) 4 rows
    const int64_t quarter = n_full / 4;
    const int most = 8 * quarter < 4 * kk ? 64 : 8;
    const int64_t least = (4 * kk + most - 1) / most;
    if (least > quarter) return false;
    p->samples = std::max<int64_t>(least, std::min<int64_t>(n_full / f, kListMaxGroups / kListSegs));
    const int64_t expect = int64_t(1.25 * kk * double(n_wide) / double(p->samples)) + kk;
    int64_t keys = 1024;
    while (keys < 2 * expect && keys < 8192) keys *= 2;
    p->keys = int(keys);
    auto split = [&](int64_t splits) {
        splits = std::max<int64_t>(1, std::min<int64_t>(splits, n_wide));
        p->splits = int(splits);
        // (groups of 128 take four wide tiles of a split to keep the places of
        // an atom apart)
        p->per_tile = kListSegs * p->samples >= 4 * kk && p->samples >= 4 * splits ? kListSegs : most;
        p->groups = int(p->samples * p->per_tile);
        const int64_t cap = std::max<int64_t>(std::max(2 * kk, kk + 192) + kListSlack, 4 * expect / (kListSegs * splits) + 64);
        p->cap = int(std::min<int64_t>(kListMaxCap, (cap + 31) / 32 * 32));
        return 256 * list_query_bytes(*p);  // of a pair of query tiles
    };
    // all queries in one pass where their lists and minima fit the budget
    const int64_t tiles = (c.m + 255) / 256;
    size_t one = split(c.splits > 0 ? c.splits : wave_splits(tiles, c.pairs, n_wide));
    // splits that were asked for yield to the budget (every split of a query
    // takes two lists, whatever kk is; the results do not depend on them)
    if (c.splits > 0)
        for (int64_t s = p->splits; one > kListBudget && s > 1;) one = split(--s);
    int64_t chunk = tiles;
    if (size_t(tiles) * one > kListBudget) {
        if (c.splits > 0) {
            chunk = std::max<int64_t>(1, int64_t(kListBudget / one));
        } else {
            // otherwise the pairs of query tiles per pass, and their splits,
            // that take the fewest waves (the minima grow with the database: of
            // 1e8 rows a budget holds 8 pairs, which have to be split to fill
            // the device)
            double best = 1e300;
            int64_t best_s = 1;
            chunk = 1;
            for (int64_t q = std::min<int64_t>(tiles, int64_t(kListBudget / split(1))); q >= 1; --q) {
                const int64_t s = wave_splits(q, c.pairs, n_wide);
                if (size_t(q) * split(s) > kListBudget) continue;
                const int64_t last = tiles % q;
                const int64_t waves = tiles / q * ((q * s + c.pairs - 1) / c.pairs) + (last * s + c.pairs - 1) / c.pairs;
                const double cost = double(waves) / double(s) * split_charge(s);
                if (cost < best * (1.0 - 1e-3)) { best = cost; best_s = s; chunk = q; }
            }
            split(best_s);
        }
    }
    p->chunk = chunk * 256;
    return true;
}

// The list scan of allknn in its locality order.  The bound comes from the
// tiles around each query tile's own group (4,096 rows at least), a minimum
// per four rows: a cluster has to give kk minima by itself, or the bound is
// the distance of other clusters and many of their rows pass (100 rows a
// cluster, 24 candidates: groups of eight let 400 rows through, the scan and
// merge of 100,003 rows took 19.7 ms; groups of four, and compactions whose
// bounds the splits share for the clusters that lie elsewhere, 8.2).
inline bool list_plan_locality(const ListCall &c, ListPlan *p) {
    const int kk = c.kk;
    const int64_t n_wide = (c.n + 255) / 256;
    p->samples = std::max<int64_t>(16, (kk + 7) / 8);
    if (kk > (kListMaxCap - 64) / 2 || 4 * p->samples > n_wide) return false;
    p->per_tile = 64;
    p->groups = int(p->samples * 64);
    const int64_t tiles = ((c.n + 127) / 128 + 1) / 2;
    const int64_t splits = c.splits > 0 ? c.splits : wave_splits(tiles, c.pairs, n_wide);
    p->splits = int(std::max<int64_t>(1, std::min<int64_t>(splits, n_wide)));
    p->cap = std::min(kListMaxCap, (2 * kk + 32 + kListSlack + 31) / 32 * 32);
    p->keys = std::max(1024, 4 * kk);
    // whole waves of query tiles per pass, in as many splits as one wave's lists allow
    const int64_t wave = c.pairs * 256;
    while (p->splits > 1 && size_t(std::min<int64_t>(wave, c.n + 255)) * list_query_bytes(*p) > kListBudget) --p->splits;
    p->chunk = std::max<int64_t>(wave, int64_t(kListBudget / list_query_bytes(*p)) / wave * wave);
    p->chunk = std::min<int64_t>(p->chunk, (c.n + 255) / 256 * 256);
    return true;
}

}  // namespace ssg
