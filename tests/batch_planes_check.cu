// Host-side check of the batched kernels' rule for planes per unit
// (batch_planes.h), compiled and run by test_batch_planes.py: whatever mix of
// instances, the length it picks gives a queue that the items can name if any of
// the lengths it may pick does, and so wherever fixed units of 16 planes (heat), of
// 8 or 32 (elastic wave) do.  Prints "ok" or the first violation.
#include <cmath>
#include <cstdio>
#include <random>

#include "batch_planes.h"

using namespace b2r::wq;

int main()
{
    std::mt19937 g(7);
    auto pick = [&](double lo, double hi) { return std::exp(std::uniform_real_distribution<>(std::log(lo), std::log(hi))(g)); };
    int long_heat = 0, long_wave = 0;   // mixes of which some length's queue is too long, and some length's is not
    for (int trial = 0; trial < 20000; ++trial) {
        std::vector<Column> in((size_t)pick(1, 60));
        const double steps = pick(10, 3e6);
        for (Column& c : in)
            c = {1 + (int)(g() % 4), (int)pick(1, 100), (int)pick(1, 4000), (int)std::min(16777215.0, steps * pick(0.2, 1.0))};
        const int h = heat_planes(in), w = wave_planes(in, 304);
        if (queue_fits(in, 16) && !queue_fits(in, h)) {
            printf("heat, trial %d: %d planes\n", trial, h);
            return 1;
        }
        if ((queue_fits(in, 8) || queue_fits(in, 32)) && !queue_fits(in, w)) {
            printf("wave, trial %d: %d planes\n", trial, w);
            return 1;
        }
        if (h < 2 || h > 16 || w < 2 || w > 32 || (queue_fits(in, 2) && w > 12)) {
            printf("trial %d: %d and %d planes\n", trial, h, w);
            return 1;
        }
        long_heat += queue_fits(in, 16) && !queue_fits(in, 2);
        long_wave += queue_fits(in, 32) && !queue_fits(in, 12);
    }
    if (long_heat < 100 || long_wave < 100) {
        printf("only %d and %d mixes near the limit\n", long_heat, long_wave);
        return 1;
    }
    printf("ok\n");
    return 0;
}
