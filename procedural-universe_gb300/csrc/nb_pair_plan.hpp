// nb_pair_plan.hpp -- how k_direct_pairs (nb_direct.cu) cuts a state into units
// and launches.  Plain C++ as well, so that the arithmetic is tested on the host
// at sizes no GPU test reaches.
#pragma once
#include <algorithm>
#include <cstddef>

#ifdef __CUDACC__
#define NB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define NB_HOST_DEVICE inline
#endif

namespace nb {

constexpr int kPairRow = 1024;        // target bodies of a row
constexpr int kPairRowTiles = 8;      // source tiles (kTileJ bodies) of a row
constexpr int kPairBlocksPerSm = 3;

// Padded bodies up to which a handle takes each pair once.  Up to here the
// units of any launch that fits its partials, and every product on the way to
// them, fit the device's 32-bit index arithmetic; a step of this many bodies
// takes more than a minute.
constexpr size_t kPairMax = (size_t)1 << 24;

// A launch of k_direct_pairs: source tiles a unit, first row, rows.
struct PairFold {
    int per, row0, rows;
};

// Units of the rows [row0, row) of a state of `rows` rows, `per` tiles a unit
// (1, 2, 4 or a multiple of 8): row q has (rows - q) * kPairRowTiles source
// tiles.  I: the kernels, which only see plans that fit, count in int; plans are
// made in long long, since those that do not fit are counted too.
template <class I>
NB_HOST_DEVICE I pair_units_before(I row, I row0, I rows, I per) {
    const I a = rows - row0, k = row - row0;
    if (per <= kPairRowTiles) return kPairRowTiles / per * (a * k - k * (k - 1) / 2);
    const I m = per / kPairRowTiles;   // sum of ceil(i / m) over a - k < i <= a
    const I qa = a / m, qb = (a - k) / m;
    return m * (qa * (qa + 1) - qb * (qb + 1)) / 2 + (a % m) * (qa + 1) - ((a - k) % m) * (qb + 1);
}

// Source entries of the rows before `row` in a launch that starts at row0.
NB_HOST_DEVICE size_t pair_source_base(int row, int row0, int n_pad) {
    const size_t r = (size_t)(row - row0), first = (size_t)n_pad - (size_t)(row0 + 1) * kPairRow;
    return r * first - (size_t)kPairRow * (r * (r - (r > 0 ? 1 : 0)) / 2);
}

inline long long pair_units(const PairFold& p, int n_pad) {
    return pair_units_before<long long>(p.row0 + p.rows, p.row0, n_pad / kPairRow, p.per);
}

// Entries of partials: kPairRow for each unit's targets, then the sources'.
inline size_t pair_entries(const PairFold& p, int n_pad) {
    return (size_t)pair_units(p, n_pad) * kPairRow + pair_source_base(p.row0 + p.rows, p.row0, n_pad);
}

// The launch of k_direct_pairs that starts at row0, within cap entries of
// partials: tiles a unit and rows (one row when not even that fits).  The length
// of a launch is estimated in tiles of one SM's time from the units of the fullest
// SM, three resident at a time (fewer take nearly as long: a block alone is a chain
// of latencies), 0.15 tiles a unit for its start and end, 0.3 units for the uneven
// end of the launch and two tiles a launch; rows left over count at the same rate.
// all_rows: the partials are roomy, and only launches of as many rows as fit are
// compared.  Measured with every length forced in turn (1 to 64 tiles, GB300): the
// choice is the fastest or within 0.5% of it at nine sizes from 21,000 (175 us; 207
// at 8 tiles a unit, 846 at 64) to 262,144 bodies (19.8 ms at 8; 20.8 at 1, 20.3 at 64).
inline PairFold pair_plan(int sm_count, int n_pad, int row0, size_t cap, bool all_rows) {
    const int rows = n_pad / kPairRow, sms = std::max(1, sm_count), left = rows - row0;
    const int pers[] = {1, 2, 4, 8, 16, 24, 32, 48, 64};
    const double tail[kPairBlocksPerSm] = {0.0, 2.2, 2.6};
    PairFold best{kPairRowTiles, row0, 1};
    double best_time = 0.0;
    bool any = false;
    for (int per : pers) {
        int most = 0;   // rows that fit (the entries grow with the rows)
        for (int over = left + 1; over - most > 1;) {
            const int mid = most + (over - most) / 2;
            if (pair_entries(PairFold{per, row0, mid}, n_pad) <= cap) most = mid; else over = mid;
        }
        for (int r = most; r >= 1; --r) {
            const PairFold p{per, row0, r};
            const long long k = (pair_units(p, n_pad) + sms - 1) / sms;
            const double work = (double)r * left - 0.5 * r * (r - 1.0), all = 0.5 * left * (left + 1.0);
            const double time = (((double)(k / kPairBlocksPerSm * kPairBlocksPerSm) + tail[k % kPairBlocksPerSm]) * (per + 0.15) +
                                 0.3 * per + 2.0) * (all / work);
            if (!any || time < best_time) {
                any = true;
                best_time = time;
                best = p;
            }
            if (all_rows) break;
        }
    }
    return best;
}

// Entries of partials that the launches of a state need within cap: the largest
// launch's, and two a body for the sums carried over when there are several.
inline size_t pair_scratch(int sm_count, int n_pad, size_t cap, size_t* largest) {
    const int rows = n_pad / kPairRow;
    int launches = 0;
    *largest = 0;
    for (int r0 = 0; r0 < rows; ++launches) {
        const PairFold p = pair_plan(sm_count, n_pad, r0, cap, true);
        *largest = std::max(*largest, pair_entries(p, n_pad));
        r0 += p.rows;
    }
    return *largest + (launches > 1 ? (size_t)2 * n_pad : 0);
}

// Reserves the partials of a state's launches: within cap, or, while there is no
// room (reserve(entries) is false), within half of it and so on down to launches
// of single rows.  Returns the cap that the launches are to be planned with, 0
// when there is no room at all.
template <class Reserve>
size_t pair_reserve(int sm_count, int n_pad, size_t cap, size_t* largest, Reserve reserve) {
    for (;; cap /= 2) {
        const size_t need = pair_scratch(sm_count, n_pad, cap, largest);
        if (reserve(need)) return cap;
        if (*largest > cap) return 0;   // single rows that do not fit cap: no smaller plan
    }
}

}  // namespace nb
