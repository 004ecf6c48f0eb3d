// Host-side check of the elastic-wave stages' launch grids (eqwp_tile.cuh,
// stage_grid), compiled and run by test_stage_grid.py: over random domains, some
// of tens of thousands of blocks, the grid's z extent is one that a launch
// takes wherever a grid without z chunks is, and the chunks cover the window.
// Prints "ok" or the first violation.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>

#include "b2r_common.cuh"
#include "eqwp_tile.cuh"

using namespace b2r;

int main()
{
    std::mt19937 g(11);
    int many = 0;
    for (int trial = 0; trial < 3000; ++trial) {
        BlockLayout L{};
        const int R = 1 + (int)(g() % 2), H = 4 * R;
        L.nblk = 1;
        for (int a = 0; a < 3; ++a) {
            L.nb[a] = 1 + (int)(g() % (trial % 3 ? 5 : 40));
            L.B[a] = H + (int)(g() % 60);
            L.n[a] = L.B[a] + 2 * H;
            L.nblk *= L.nb[a];
        }
        if (L.nblk > 65535) continue;
        L.H = H;
        L.xoff = (H + 4 + 31) / 32 * 32 - H;
        L.P = (L.xoff + L.n[0] + 8 + 31) / 32 * 32;
        L.periodic = (int)(g() % 2);
        L.fixed_edge = -1;
        for (int shrink : {2, 4}) {
            const eqk::Grid q = eqk::stage_grid(L, shrink);
            const int nz = L.n[2] - (L.periodic || L.nb[2] > 2 ? 2 * shrink : 0);
            if (q.g.z > 65535u || q.g.y > 65535u || q.t.nzc < 1 || (int)q.g.z != L.nblk * q.t.nzc || q.t.nzc > std::max(1, nz)) {
                printf("%d blocks of %dx%dx%d: grid z %u, %d chunks\n", L.nblk, L.B[0], L.B[1], L.B[2], q.g.z, q.t.nzc);
                return 1;
            }
            many += L.nblk > 32767;
        }
    }
    if (many < 20) {
        printf("only %d grids of many blocks\n", many);
        return 1;
    }
    printf("ok\n");
    return 0;
}
