// heat_far.cu -- one heat time step of radius 1..4.
//
// The sweep of heat.cu with what bounds it taken out of its way.  There, the plane loop could not be unrolled by the queue's depth at radius
// 4 without spilling, so the queue moved 64 registers per plane, and all
// eight warps met at a barrier per plane.  Here
//   * a CTA is one producer warp, which streams the input planes by TMA into
//     a ring of shared planes, and 15, 11 or 7 consumer warps; planes are handed over
//     by two mbarriers per slot (loaded; read by every consumer warp), so no
//     warp waits for another one's arithmetic and the warps drift apart by
//     the depth of the ring;
//   * with 16 warps per SM a consumer thread has the registers for the 2D+1
//     planes of its 4 cells of 2 rows and the loop unrolled by them, so the
//     queue turns by names;
//   * the y neighbours of the two rows are read pair by pair as the radius
//     grows, each row once for both.
// A thread's cells run the sweep's operations in its order (heat_unit.cuh):
// the same bits.
//
// Measured (us per step against heat.cu's default schedule): 512^3 radius 2
// 168 from 191 (798 GLUPS, 0.94 of the copy rate at one read and one write per
// cell), radius 3 175 from 237, radius 4 188 from 275; 256^3 radius 4 29.6
// from 41.7; 128^3 radius 2 5.0 from 8.4; 64^3 radius 3 4.2 from 6.0; 32^3
// radius 2 3.3 from 5.2.
//
// Every wait is bounded; a warp that gives up reports
// DEV_TIMEOUT and leaves, and so does every warp that waits for it.
#include "heat_far.cuh"

namespace b2r {
namespace {

using namespace farx;

constexpr int kTW = 128;             // output cells per tile row

// NC consumer warps, two output rows each
template <int D, int NC>
struct FCfg {
    static constexpr int TH = 2 * NC, THR = 32 * (NC + 1);
    static constexpr int BW = kTW + 8, BH = TH + 2 * D;    // TMA box (cells)
    static constexpr int SLOT = (BW * BH + 31) / 32 * 32;   // floats per ring slot (a multiple of 128 bytes)
    static constexpr int S = D + 4;                         // ring slots: D + 1 planes in use, three ahead
    static constexpr size_t SMEM = (size_t)S * SLOT * 4 + 2 * S * 8 + 128;
};

template <int D, int NC>
__global__ void __launch_bounds__(32 * (NC + 1), NC <= 7 ? 2 : 1)
heat_far_kernel(const __grid_constant__ CUtensorMap tin, float* __restrict__ out, const BlockLayout L,
                const int step_i, const HeatCoef C, const HeatTiles sch, int* __restrict__ status)
{
    using Cfg = FCfg<D, NC>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* const ring = reinterpret_cast<float*>(smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127));
    uint64_t* const full = reinterpret_cast<uint64_t*>(ring + Cfg::S * Cfg::SLOT);
    uint64_t* const empty = full + Cfg::S;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < Cfg::S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], NC);
        }
        fence_mbar_init();
    }
    __syncthreads();
    pdl_begin();

    int u = blockIdx.x;
    const int tx = u % sch.ntx;
    u /= sch.ntx;
    const int ty = u % sch.nty;
    u /= sch.nty;
    const int zc = u % sch.nzc, blk = u / sch.nzc;
    const int edge = edge_bits(L, blk);
    int lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) stage_region(L, edge, a, D * (step_i + 1), lo[a], hi[a]);
    const int xs0 = sch.x0 + tx * kTW;                  // storage x of the tile's first cell
    const int y0 = sch.y0 + ty * Cfg::TH;               // its first row
    if (xs0 - L.xoff > hi[0] || xs0 + kTW - 1 - L.xoff < lo[0] || y0 > hi[1] || y0 + Cfg::TH - 1 < lo[1]) return;
    const int zs = max(sch.z0 + zc * sch.Lz, lo[2]), ze = min(sch.z0 + (zc + 1) * sch.Lz - 1, hi[2]);
    if (zs > ze) return;
    const int first = zs - D, np = ze + D - first + 1;  // input planes

    if (warp == NC) {                                // the producer
        if (lane != 0) return;
        int slot = 0, phase = 0;
        bool ok = true;
        int i = 0;
        for (; i < np; ++i) {
            if (i >= Cfg::S && !mbar_wait_bounded(&empty[slot], phase ^ 1)) {
                ok = false;
                break;
            }
            mbar_expect_tx(&full[slot], Cfg::BW * Cfg::BH * 4);
            tma_load_4d(ring + slot * Cfg::SLOT, &tin, xs0 - 4, y0 - D, first + i, blk, &full[slot]);
            if (++slot == Cfg::S) slot = 0, phase ^= 1;
        }
        if (!ok) {                                      // the loads in flight land before the CTA leaves (bounded)
            report(status, DEV_TIMEOUT);
            for (int k = max(0, i - Cfg::S); k < i; ++k)
                mbar_wait_bounded(&full[k % Cfg::S], (k / Cfg::S) & 1, 100000000ull);
        }
        return;
    }
    FCtx<D, Cfg::S, Cfg::SLOT, Cfg::BW> c;
    c.full = full;
    c.empty = empty;
    c.plane = L.plane;
    c.P = L.P;
    c.np = np;
    c.lane0 = lane == 0;
    c.ring = ring + (D + 2 * warp) * Cfg::BW + 4 + 4 * lane;
    const int y = y0 + 2 * warp, xb = xs0 + 4 * lane - L.xoff;
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) m |= (xb + j >= lo[0] && xb + j <= hi[0] ? 1u : 0u) << j;
    c.m0 = y >= lo[1] && y <= hi[1] ? m : 0u;
    c.m1 = y + 1 >= lo[1] && y + 1 <= hi[1] ? m : 0u;
    c.dst = out + (long long)blk * L.bstride + (long long)zs * L.plane + (long long)y * L.P + xs0 + 4 * lane;
    int slot = 0, phase = 0, cslot = 0;
    if (!f_unit(c, ParamCoef{C}, slot, phase, cslot) && lane == 0) report(status, DEV_TIMEOUT);
}

// Tile height and z chunk of a launch: the least busy busiest SM.  A unit of
// lz planes costs lz + 2D planes and about two more until the ring is full; a
// plane about 0.07 + 0.0222 us per row of the tile (radius 4, 512^3: 0.737 us
// for 30 rows, 0.567 for 22, 0.709 for two tiles of 14).  Measured us per step
// for 30 / 22 / 14 rows: radius 4, 512^3 197 / 207 / 188, 160^3 14.4 / 13.3 /
// 14.2, 128^3 8.1 / 6.9 / 7.9; radius 2, 100x90x80 4.5 / 4.1 / 4.4, 32^3 4.3 /
// 3.8 / 3.4.
struct FPlan {
    int rows = 0, lz = 0;
    double cost = 1e300;
};
FPlan f_plan(int nblk, int D, int ntx, int NY, int NZ, int sms)
{
    FPlan best;
    for (int rows : {30, 22, 14}) {
        const long long tiles = (long long)ntx * ((NY + rows - 1) / rows) * nblk;
        const int slots = rows == 14 ? 2 * sms : sms;
        const double one = 0.07 + 0.0222 * rows;
        for (int n = 1; n <= NZ; ++n) {
            const int lz = (NZ + n - 1) / n;
            if (n > 1 && lz < 3) break;
            const long long units = tiles * ((NZ + lz - 1) / lz);
            // two CTAs of 14 rows share an SM, or one has it alone
            const double plane = rows > 14 ? one : (units > sms ? 1.85 : 1.4) * one;
            const double cost = (double)((units + slots - 1) / slots) * (lz + 2 * D + 2) * plane;
            if (cost < best.cost) best = FPlan{rows, lz, cost};
        }
    }
    return best;
}

template <int D, int NC>
cudaError_t launch_f(const CUtensorMap* tin, float* out, const BlockLayout& L, const HeatTiles& sch, int step_i,
                     const HeatCoef& c, int* status, cudaStream_t st)
{
    using Cfg = FCfg<D, NC>;
    static KernelSetup setup;
    if (cudaError_t e = kernel_setup(setup, heat_far_kernel<D, NC>, Cfg::THR, Cfg::SMEM, nullptr, nullptr)) return e;
    return launch_pdl(heat_far_kernel<D, NC>, (unsigned)((long long)sch.ntx * sch.nty * sch.nzc * L.nblk), Cfg::THR,
                      Cfg::SMEM, st, *tin, out, L, step_i, c, sch, status);
}

// Tiles over the union of the blocks' windows, which shrink from sub-step to
// sub-step: 250 cells take two tile columns where 258 take three
// (250x186x132 torus as one block, radius 2, three steps between exchanges:
// 670 us for 48 steps against 716 with tiles over all that a period computes).
cudaError_t f_tiles(const BlockLayout& L, int D, int step_i, HeatTiles& sch)
{
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    int lo[3] = {1 << 30, 1 << 30, 1 << 30}, hi[3] = {-1, -1, -1};
    for (int b = 0; b < L.nblk; ++b)
        for (int a = 0; a < 3; ++a) {
            int l, h;
            stage_region(L, edge_bits(L, b), a, D * (step_i + 1), l, h);
            lo[a] = std::min(lo[a], l);
            hi[a] = std::max(hi[a], h);
        }
    sch = HeatTiles{};
    sch.x0 = (L.xoff + lo[0]) & ~3;
    sch.y0 = lo[1];
    sch.z0 = lo[2];
    const int NY = hi[1] - lo[1] + 1, NZ = hi[2] - lo[2] + 1;
    if (hi[0] < lo[0] || NY < 1 || NZ < 1) {
        sch.rows = 1;        // nothing to compute
        return cudaSuccess;
    }
    sch.ntx = (L.xoff + hi[0] - sch.x0) / kTW + 1;
    const FPlan p = f_plan(L.nblk, D, sch.ntx, NY, NZ, sms);
    sch.rows = p.rows;
    sch.Lz = p.lz;
    sch.nty = (NY + p.rows - 1) / p.rows;
    sch.nzc = (NZ + p.lz - 1) / p.lz;
    return cudaSuccess;
}

template <int D>
cudaError_t launch_d(const CUtensorMap* tin, float* out, const BlockLayout& L, int step_i, const HeatCoef& c,
                     int* status, cudaStream_t st, HeatTiles& sch)
{
    if (!sch.rows)
        if (cudaError_t e = f_tiles(L, D, step_i, sch)) return e;
    // rows of the tile by the tensor map's box: tin[0], [1], [2] for 30, 22, 14
    switch (sch.rows) {
    case 30: return launch_f<D, 15>(&tin[0], out, L, sch, step_i, c, status, st);
    case 22: return launch_f<D, 11>(&tin[1], out, L, sch, step_i, c, status, st);
    case 14: return launch_f<D, 7>(&tin[2], out, L, sch, step_i, c, status, st);
    default: return cudaSuccess;
    }
}

}  // namespace

int heat_far_box_w() { return kTW + 8; }
int heat_far_box_h(int D, int k) { return (k == 0 ? 30 : k == 1 ? 22 : 14) + 2 * D; }

cudaError_t launch_heat_far(const CUtensorMap* tin, float* out, const BlockLayout& L, int D, int step_i,
                            const HeatCoef& c, int* status, cudaStream_t st, HeatTiles& tiles)
{
    switch (D) {
    case 1: return launch_d<1>(tin, out, L, step_i, c, status, st, tiles);
    case 2: return launch_d<2>(tin, out, L, step_i, c, status, st, tiles);
    case 3: return launch_d<3>(tin, out, L, step_i, c, status, st, tiles);
    case 4: return launch_d<4>(tin, out, L, step_i, c, status, st, tiles);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace b2r
