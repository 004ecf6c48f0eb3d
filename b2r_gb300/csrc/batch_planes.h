// batch_planes.h -- planes per work unit of the batched kernels when the caller
// sets none (host side): the length with the shortest run by a model of each
// kernel, among those whose queue the items can name.
#pragma once
#include <algorithm>
#include <vector>

namespace b2r {
namespace wq {

constexpr long long kMaxItems = 1ll << 28;   // of a batch's queue (work_queue.cuh)
constexpr long long kMaxUnits = 1ll << 24;   // of an instance

// An instance: radius, tiles per plane, planes, rounds.
struct Column {
    int D, tiles, planes, rounds;
};

inline bool queue_fits(const std::vector<Column>& in, int lz)
{
    long long items = 0;
    for (const Column& c : in) {
        const long long units = (long long)c.tiles * ((c.planes + lz - 1) / lz);
        if (units >= kMaxUnits) return false;
        items += units * c.rounds;
    }
    return items <= kMaxItems;
}

inline void longest_first(std::vector<Column>& in)
{
    std::sort(in.begin(), in.end(), [](const Column& x, const Column& y) { return x.rounds > y.rounds; });
}

// Heat, one step per unit (batch.cu): a unit takes 3 us and 0.55 us per plane it
// reads, a round of a radius (a launch of its own) lasts one unit at least, or as
// many one after the other as each resident CTA gets, and the radii follow one
// another.  The units of a small batch have to be short for every CTA to get
// one: 18 instances of 24..75 cells a side took 4.98 ms at 16 planes and take
// 2.77 ms at the 2 or 3 this picks, 14 of 32..80 5.31 and 3.01, 39 of 32..140
// 17.1 and 14.7 (12.9 at 6); 64 of 32..192 stay at 16 (46.8 ms, at 8 planes
// 52.4).
inline int heat_planes(std::vector<Column> in)
{
    longest_first(in);
    int best = 16;
    double least = 1e300;
    for (int lz : {16, 12, 8, 6, 4, 3, 2}) {
        if (lz < 16 && !queue_fits(in, lz)) break;
        double us = 0;
        for (int D = 1; D <= 4; ++D) {
            double units = 0, planes = 0, one = 0;   // of a round of the instances so far, which all step longer
            int left = 0;
            for (const Column& c : in) {
                if (c.D != D) continue;
                us += (left - c.rounds) * one;
                const double n = (double)c.tiles * ((c.planes + lz - 1) / lz);
                units += n;
                planes += n * (std::min(lz, c.planes) + 2 * D);
                one = std::max(1.0, units / 304.0) * (3.0 + 0.55 * planes / units);
                left = c.rounds;
            }
            us += left * one;
        }
        if (us < least) {
            least = us;
            best = lz;
        }
    }
    return best;
}

// Elastic wave (eqwp_batch.cu) on `grid` resident CTAs: a unit takes 4 us and
// 2.05 us per plane (eqwp_tile.cuh) and a round lasts one unit at least, or as
// many units one after the other as each resident CTA gets; at most 12 planes,
// beyond which neighbouring tiles lose their L2 hits, unless only a longer
// unit's queue can be named.  GLUPS by planes 3, 4, 6, 8, 12, 16, 32: 16
// instances of 32-128 cells per edge 31.7, 34.2, 37.5, 38.8, 39.7, 39.8, 31.6; 8
// of 64^3 34.9, 37.5, 40.0, 32.8, 25.8, 18.8, 10.1; 12 of 36^3 23.4, 18.5, 13.4,
// 10.6, 7.4, 7.4, 5.3; 6 of 200^3 32.4, 35.7, 38.9, 40.4, 40.1, 38.3, 34.5.
inline int wave_planes(std::vector<Column> in, int grid)
{
    longest_first(in);
    int best = 0;
    double least = 1e300;
    for (int lz = 2; lz <= 12; ++lz) {
        if (!queue_fits(in, lz)) continue;
        double us = 0;
        long long units = 0;   // of a round in which the first j + 1 instances still step
        for (size_t j = 0; j < in.size(); ++j) {
            units += (long long)in[j].tiles * ((in[j].planes + lz - 1) / lz);
            const int rounds = in[j].rounds - (j + 1 < in.size() ? in[j + 1].rounds : 0);
            us += rounds * std::max(1.0, (double)units / grid) * (4 + 2.05 * lz);
        }
        if (us < least) {
            least = us;
            best = lz;
        }
    }
    for (int lz : {16, 24, 32})
        if (!best && (queue_fits(in, lz) || lz == 32)) best = lz;
    return best;
}

}  // namespace wq
}  // namespace b2r
