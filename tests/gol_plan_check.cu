// Host-side check of the Game-of-Life pass's plan (gol_plan.h), compiled and run by
// test_gol_plan.py: over random grids the tile that the search picks is as cheap
// by its model as the best of every tile (the longest of each count of chunks) of
// the same generations, and within the kernel's limits.  Prints the time of a
// search, and "ok" or the first violation.
#include <chrono>
#include <cmath>
#include <cstdio>
#include <random>

#include "gol_plan.h"

using namespace b2r;

int main()
{
    std::mt19937 g(3);
    auto pick = [&](double lo, double hi) {
        return (int)std::exp(std::uniform_real_distribution<>(std::log(lo), std::log(hi))(g));
    };
    double us = 0;
    const int trials = 400;
    for (int trial = 0; trial < trials; ++trial) {
        const GolPass base = gol_pass_rows(pick(2, 1500), pick(2, 700), pick(2, 700), g() % 2);
        const int left = 1 + (int)(g() % kGolDomainMaxGen);
        const auto t0 = std::chrono::steady_clock::now();
        const GolPass p = gol_plan_pass(base, left, 152);
        us += std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count();
        const GolTile mine = gol_tile(base, p.G, p.PR, p.Tz, 152);
        if (p.G < 1 || p.G > left || p.PR % kGolRows || p.PR > kGolMaxRegion || p.PZ > kGolMaxRegion || p.Ty != p.PR - 2 * p.G ||
            p.PZ != p.Tz + 2 * p.G || p.Ty < 1 || p.Tz < 1 || p.smem > kGolMaxSmem || p.threads > kGolMaxThreads ||
            p.threads < p.WX * (p.PR / kGolRows) * p.nzs || !mine.fit(p.nzs) || p.nty * p.Ty < base.ny) {
            printf("%d x %d x %d: outside the limits\n", base.nx, base.ny, base.nz);
            return 1;
        }
        double least = 1e300;
        for (int G : {1, 2, 3, 4, 5, 6, 8})
            for (int PR = 4; PR <= kGolMaxRegion; PR += PR < 24 ? kGolRows : 4)
                for (int n = 1; n <= base.nz; ++n) {   // chunks along z
                    const int Tz = (base.nz + n - 1) / n;
                    if (G > left || PR - 2 * G < 1 || PR - 2 * G >= base.ny + 4 || Tz > kGolMaxRegion - 2 * G || (Tz < 3 && base.nz > 8))
                        continue;
                    const GolTile t = gol_tile(base, G, PR, Tz, 152);
                    for (int nzs : {4, 2, 3, 6, 8, 12, 16, 1})
                        if (t.fit(nzs)) least = std::min(least, t.cost(nzs));
                }
        if (mine.cost(p.nzs) > least * (1 + 1e-9)) {
            printf("%d x %d x %d, %d to go: %g, the best %g\n", base.nx, base.ny, base.nz, left, mine.cost(p.nzs), least);
            return 1;
        }
    }
    fprintf(stderr, "%.1f us per search\n", us / trials);
    printf("ok\n");
    return 0;
}
