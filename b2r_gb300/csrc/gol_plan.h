// gol_plan.h -- tile and generations of a Game-of-Life pass on the domain's bit
// grid (gol_domain.cu), chosen on the host.
#pragma once
#include <algorithm>
#include <cstddef>

namespace b2r {

constexpr int kGolDomainMaxGen = 8;   // generations per pass at most
// A pass over the domain's bit grid (gol_domain.cu).
struct GolPass {
    int nx, ny, nz, W;     // cells per axis of the bit grid (shell included), words per row
    int periodic;
    int G;                 // generations of this pass
    int WX, XO, split;     // region words per row, output words, 1: a row is cut into x tiles
    int Ty, Tz, PR, PZ;    // output rows / planes of a tile, region rows (even) / planes
    int RP, RPZ;           // shared pitch of a row and of a plane (words)
    int nzs;               // z segments of a CTA
    int ntx, nty;
    int threads;
    size_t smem;
};
constexpr int kGolRows = 2;               // rows per thread
constexpr int kGolMaxThreads = 1024;
constexpr int kGolMaxRegion = 96;         // region rows / planes at most
constexpr size_t kGolMaxSmem = 200 * 1024;

// The rows of a grid of nx x ny x nz cells.
inline GolPass gol_pass_rows(int nx, int ny, int nz, bool periodic)
{
    GolPass P{};
    P.nx = nx;
    P.ny = ny;
    P.nz = nz;
    P.W = (nx + 31) / 32;
    P.periodic = periodic;
    P.split = P.W > 32;
    P.XO = P.split ? 30 : P.W;
    P.WX = P.split ? 32 : P.W;
    P.ntx = P.split ? (P.W + P.XO - 1) / P.XO : 1;
    return P;
}

// Shared pitch of a row: 2 more than a multiple of 4, so that the rows of
// the threads of a warp (words fastest, then pairs of rows) spread over the
// banks; a template argument of the kernel, so that a thread's loads of a plane
// share three addresses.
inline int gol_row_pitch(int WX) { return WX <= 2 ? 2 : (WX - 2 + 3) / 4 * 4 + 2; }

// A tile of the search: G generations on a region of PR rows x PZ = Tz + 2 G
// planes, of which `ctas` cover the grid.
struct GolTile {
    int G, PR, Tz, PZ, WX;
    long long busiest;      // CTAs of the busiest SM
    size_t smem;
    int fit(int nzs) const  // CTAs that share an SM; 0: a CTA does not run
    {
        const int th = WX * (PR / kGolRows) * nzs, warps = (th + 31) / 32;
        if (th > kGolMaxThreads || (nzs > 1 && Tz < nzs) || smem > kGolMaxSmem) return 0;
        return (int)std::min<size_t>(std::min(2048 / (warps * 32), 65536 / (warps * 32 * 64)), (220 * 1024) / (smem + 1024));
    }
    // Cycles per generation of the busiest SM with `nzs` z segments per CTA.  Each
    // generation of a CTA costs its logic operations (about 22 per word, and 20
    // more for the x and y sums, which a z segment computes for two extra
    // planes), at 64 lanes per cycle and SM, or the chain of one thread where few
    // threads are in flight; a pass costs a launch and the load of its regions on
    // top.
    double cost(int nzs) const
    {
        const int f = fit(nzs), warps = (WX * (PR / kGolRows) * nzs + 31) / 32;
        auto together = [&](int n) {   // n CTAs resident on the SM
            double c = (double)n * PZ * PR * WX * 0.55;               // the load
            for (int g = 1; g <= G; ++g) {
                const int sz = (PZ - 2 * g + nzs - 1) / nzs;
                const double per = kGolRows * (25.0 * sz + 14.0 * (sz + 2)) + 12.0 * sz;   // per thread
                c += std::max(n * warps * 32 * per / 56.0, per * 9.5) + 150.0;
            }
            return c;
        };
        double c = (double)(busiest / f) * together(f);
        if (busiest % f) c += together((int)(busiest % f));
        return (c + 6000.0) / G;
    }
    // What no number of segments can go below: the load, and 25 sz + 14 (sz + 2) +
    // 6 sz operations per word and segment of sz planes.
    double least() const
    {
        return (6000.0 + 150.0 * G +
                (double)busiest * PR * WX * ((45.0 / 56.0) * (G * PZ - G * (G + 1)) + 0.5 * G + 0.55 * PZ)) / G;
    }
    // What `nzs` cannot go below: 9.5 cycles per operation of a thread.
    double least(int nzs) const
    {
        const int f = fit(nzs);
        return (6000.0 + (double)((busiest + f - 1) / f) *
                             (150.0 * G + 0.55 * PZ * PR * WX + 9.5 * (90.0 / nzs * (G * PZ - G * (G + 1)) + 56.0 * G))) / G;
    }
};
inline GolTile gol_tile(const GolPass& base, int G, int PR, int Tz, int sms)
{
    const int PZ = Tz + 2 * G, Ty = PR - 2 * G;
    const long long ctas = (long long)base.ntx * ((base.ny + Ty - 1) / Ty) * ((base.nz + Tz - 1) / Tz);
    return {G, PR, Tz, PZ, base.WX, (ctas + sms - 1) / sms, (size_t)8 * PZ * (PR + 2) * gol_row_pitch(base.WX)};
}

// Tile and generations (at most `left`) of a pass by the cost above.  Tiles are
// passed over by the two bounds, first a few all over the range, so that these
// hold soon: a search takes 10 to 90 us where it took 30 to 500 through every tile.
inline GolPass gol_plan_pass(const GolPass& base, int left, int sms)
{
    GolPass best = base;
    double best_cost = 1e300;
    auto look = [&](const GolTile& t) {
        if (t.least() >= best_cost) return;
        for (int nzs : {4, 8, 2, 16, 3, 6, 12, 1}) {
            if (!t.fit(nzs) || t.least(nzs) >= best_cost) continue;
            const double c = t.cost(nzs);
            if (c >= best_cost) continue;
            best_cost = c;
            best.G = t.G;
            best.Ty = t.PR - 2 * t.G;
            best.Tz = t.Tz;
            best.PR = t.PR;
            best.PZ = t.PZ;
            best.nzs = nzs;
        }
    };
    for (const bool coarse : {true, false})
        for (int G : {4, 6, 8, 3, 5, 2, 1}) {
            if (G > left) continue;
            for (int PR = 4; PR <= kGolMaxRegion; PR += PR < 24 ? kGolRows : 4) {
                const int Ty = PR - 2 * G;
                if (Ty < 1 || (coarse && PR % 8)) continue;
                if (Ty >= base.ny + 4) break;
                // the work of the rows alone, however they are cut along z
                const double tiles = (double)base.ntx * ((base.ny + Ty - 1) / Ty) / sms * PR * base.WX;
                if (6000.0 + 150.0 * G + tiles * ((45.0 / 56.0) * G * (base.nz + G - 1) + 0.55 * (base.nz + 2 * G)) >= best_cost * G)
                    continue;
                // the longest tile of every count of chunks, from the longest whose regions fit
                const int room = (int)(kGolMaxSmem / ((size_t)8 * (PR + 2) * gol_row_pitch(base.WX)));
                for (int Tz = std::min(base.nz, std::min(kGolMaxRegion, room) - 2 * G); Tz >= 1;) {
                    const int n = (base.nz + Tz - 1) / Tz, longest = (base.nz + n - 1) / n;
                    if (longest < 3 && base.nz > 8 && n > 1) break;
                    look(gol_tile(base, G, PR, longest, sms));
                    if (n >= base.nz) break;
                    Tz = std::min((base.nz + n) / (n + 1), longest - 1);     // one chunk more at least
                    if (coarse) Tz -= Tz / 4;
                }
            }
        }
    best.nty = (base.ny + best.Ty - 1) / best.Ty;
    best.RP = gol_row_pitch(best.WX);
    best.RPZ = (best.PR + 2) * best.RP;
    best.smem = (size_t)8 * best.PZ * best.RPZ;
    best.threads = (best.WX * (best.PR / kGolRows) * best.nzs + 31) / 32 * 32;
    return best;
}

}  // namespace b2r
