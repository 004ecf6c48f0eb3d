// heat_rows.cu -- T = 2, 3 or 4 heat time steps per HBM pass, radius 1, four
// rows per thread.
//
// The same scheme as heat_tb.cu (a CTA reads a tile of the field once,
// advances it T sub-steps on chip and writes it once; bit-identical to T
// launches of the plain sweep), laid out for the fewest instructions per
// update, which is what bounds several steps per pass on this GPU:
//   * a thread holds 4 consecutive x cells (float4) of 4 rows, a warp 128
//     cells of 4 rows, so of the y neighbours only the rows above and below
//     the warp's four come from shared memory: per stage and 16 cells two
//     128-bit loads and two stores of edge rows, against eight and eight when
//     whole planes are exchanged between threads of two rows;
//   * the tile's first and last lane only feed x neighbours (by shuffles), so
//     every stored row piece is a whole float4 and no column is read apart;
//   * cells outside a window are computed like any other (nothing stored
//     depends on them); only a tile that touches a fixed face restores the
//     shell layer there, behind one branch that is uniform over the CTA;
//   * the pipeline fills and drains without conditions: a stage's first planes
//     are computed from whatever the queues hold and never reach a stored
//     plane.
// Per input plane p (one TMA box of 128 x (4 NW + 2) cells into a 4-slot
// mbarrier ring), stage s = 1..T computes plane p-s from stage s-1's planes
// p-s-1, p-s, p-s+1, which the thread holds in registers (the newest made in
// this iteration); the edge rows of plane p-s were exchanged one iteration
// earlier, so one barrier per plane orders everything.
#include <algorithm>
#include <climits>

#include "b2r_common.cuh"
#include "heat.h"
#include "heat_upd.cuh"

namespace b2r {
namespace {

constexpr int kRY = 4;              // rows per thread
constexpr int kBoxW = 128;          // computed cells per tile row
constexpr int kOutW = 120;          // stored cells per tile row: lanes 1..30
constexpr int kSlots = 4;           // ring slots

template <int T, int NW>
struct RCfg {
    static constexpr int ROWS = kRY * NW;              // computed rows
    static constexpr int BH = ROWS + 2;                // box rows
    static constexpr int SLOT = kBoxW * BH;            // floats per ring slot (a multiple of 128 bytes)
    static constexpr int OH = ROWS - 2 * (T - 1);      // stored rows: T-1 .. ROWS-T
    static constexpr int XE = 2 * NW * kBoxW;          // floats of one stage's edge rows
    static constexpr size_t SMEM = (size_t)kSlots * SLOT * 4 + (size_t)(T - 1) * 2 * XE * 4 + kSlots * 8 + 128;
};

__device__ __forceinline__ float4 rld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void rst4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

template <int T, int NW>
struct RCtx {
    float4 q[T][3][kRY];        // [level s-1's planes][slot][row]
    const float* ring;          // + the thread's first cell of its first row (box row 1 + 4 warp)
    float* xch;                 // edge rows, + the thread's x
    uint64_t* bar;
    const CUtensorMap* tmap;
    HeatCoef C;
    float* dst;                 // the thread's first cell, row 0, of the plane stage T makes next
    long long plane;
    int P, tid, warp, blk, X0, Y0;
    int np, first, zs, ze;
    int zk0, zk1;               // fixed-shell planes next to the window, or INT_MIN
    unsigned ykm, xkm, mst;     // rows / cells that keep their value; cells stored (4 bits per row)
    bool edge;                  // the tile touches a fixed face (uniform over the CTA)
    bool xkw;                   // some lane of the warp has xkm
};

// One input plane.  PH = pr mod 3: the queue slot of the newest planes.
// Returns false when a bounded wait gave up (all threads agree).
template <int T, int NW, int PH>
__device__ __forceinline__ bool r_iter(RCtx<T, NW>& c, int pr)
{
    using Cfg = RCfg<T, NW>;
    constexpr int NEW = PH, CUR = (PH + 2) % 3, OLD = (PH + 1) % 3;
    const bool bad = !mbar_wait_bounded(&c.bar[pr % kSlots], (pr / kSlots) & 1);
    const int p = c.first + pr;
    {
        const float* pl = c.ring + (pr % kSlots) * Cfg::SLOT;
#pragma unroll
        for (int r = 0; r < kRY; ++r) c.q[0][NEW][r] = rld4(pl + r * kBoxW);
    }
#pragma unroll
    for (int s = 1; s <= T; ++s) {
        const int z = p - s;
        // the rows above and below the warp's four in stage s-1's plane z
        float4 up, dn;
        if (s == 1) {
            const float* pc = c.ring + ((pr + kSlots - 1) % kSlots) * Cfg::SLOT;
            up = rld4(pc - kBoxW);
            dn = rld4(pc + kRY * kBoxW);
        } else {
            const float* xi = c.xch + (size_t)((s - 2) * 2 + (z & 1)) * Cfg::XE;
            const int wu = c.warp > 0 ? c.warp - 1 : 0, wd = c.warp < NW - 1 ? c.warp + 1 : NW - 1;
            up = rld4(xi + (2 * wu + 1) * kBoxW);
            dn = rld4(xi + 2 * wd * kBoxW);
        }
        float4 res[kRY];
#pragma unroll
        for (int r = 0; r < kRY; ++r) {
            const float4 ce = c.q[s - 1][CUR][r];
            const float l = __shfl_up_sync(0xffffffffu, ce.w, 1);
            const float rt = __shfl_down_sync(0xffffffffu, ce.x, 1);
            const float4 ym = r == 0 ? up : c.q[s - 1][CUR][r > 0 ? r - 1 : 0];
            const float4 yp = r == kRY - 1 ? dn : c.q[s - 1][CUR][r < kRY - 1 ? r + 1 : r];
            res[r] = heat_upd4(c.C, ce, l, rt, ym, yp, c.q[s - 1][OLD][r], c.q[s - 1][NEW][r]);
        }
        if (s < T) {
            if (c.edge) {
                const bool zk = z == c.zk0 || z == c.zk1;
                const unsigned rows = zk ? 15u : c.ykm;
                if (rows) {
#pragma unroll
                    for (int r = 0; r < kRY; ++r)
                        if (rows & (1u << r)) res[r] = c.q[s - 1][CUR][r];
                }
                if (c.xkw) {
#pragma unroll
                    for (int r = 0; r < kRY; ++r) {
                        const float4 ce = c.q[s - 1][CUR][r];
                        res[r].x = c.xkm & 1u ? ce.x : res[r].x;
                        res[r].y = c.xkm & 2u ? ce.y : res[r].y;
                        res[r].z = c.xkm & 4u ? ce.z : res[r].z;
                        res[r].w = c.xkm & 8u ? ce.w : res[r].w;
                    }
                }
            }
            float* xo = c.xch + (size_t)((s - 1) * 2 + (z & 1)) * Cfg::XE + 2 * c.warp * kBoxW;
            rst4(xo, res[0]);
            rst4(xo + kBoxW, res[kRY - 1]);
#pragma unroll
            for (int r = 0; r < kRY; ++r) c.q[s < T ? s : 0][NEW][r] = res[r];
        } else {
            if (z >= c.zs && z <= c.ze) {
                if (c.mst == 0xFFFFu) {
#pragma unroll
                    for (int r = 0; r < kRY; ++r) rst4(c.dst + r * c.P, res[r]);
                } else if (c.mst) {
#pragma unroll
                    for (int r = 0; r < kRY; ++r) {
                        const unsigned b = (c.mst >> (4 * r)) & 15u;
                        float* d = c.dst + r * c.P;
                        if (b == 15u) {
                            rst4(d, res[r]);
                        } else if (b) {
                            if (b & 1u) d[0] = res[r].x;
                            if (b & 2u) d[1] = res[r].y;
                            if (b & 4u) d[2] = res[r].z;
                            if (b & 8u) d[3] = res[r].w;
                        }
                    }
                }
            }
            c.dst += c.plane;
        }
    }
    if (__syncthreads_or(bad)) return false;
    // plane p-1 is no longer needed: refill its slot
    if (c.tid == 0 && pr >= 1) {
        const int nxt = pr - 1 + kSlots;
        if (nxt < c.np) {
            mbar_expect_tx(&c.bar[nxt % kSlots], Cfg::SLOT * 4);
            tma_load_4d(const_cast<float*>(c.ring) + (nxt % kSlots) * Cfg::SLOT - kBoxW, c.tmap, c.X0, c.Y0 - 1,
                        c.first + nxt, c.blk, &c.bar[nxt % kSlots]);
        }
    }
    return true;
}

template <int T, int NW>
__global__ void __launch_bounds__(32 * NW, 1)
heat_rows_kernel(const __grid_constant__ CUtensorMap tin, float* __restrict__ out, const BlockLayout L,
                 const int step_i, const HeatCoef C, const HeatTiles sch, int* __restrict__ status)
{
    using Cfg = RCfg<T, NW>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* const ring = reinterpret_cast<float*>(smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127));
    RCtx<T, NW> c;
    c.tid = threadIdx.x;
    c.warp = __shfl_sync(0xffffffffu, c.tid >> 5, 0);   // uniform over the warp, and known to be
    const int lane = c.tid & 31;
    c.xch = ring + kSlots * Cfg::SLOT;
    c.bar = reinterpret_cast<uint64_t*>(c.xch + (T - 1) * 2 * Cfg::XE);
    if (c.tid == 0) {
        for (int s = 0; s < kSlots; ++s) mbar_init(&c.bar[s], 1);
        fence_mbar_init();
    }
    __syncthreads();
    pdl_begin();

    // the unit: tile column fastest, then tile row, z chunk, block
    int u = blockIdx.x;
    const int tx = u % sch.ntx;
    u /= sch.ntx;
    const int ty = u % sch.nty;
    u /= sch.nty;
    const int zc = u % sch.nzc;
    c.blk = u / sch.nzc;
    const int edge = edge_bits(L, c.blk);
    int lo[3], hi[3];                               // window of the last stage: the stored cells
#pragma unroll
    for (int a = 0; a < 3; ++a) stage_region(L, edge, a, step_i + T, lo[a], hi[a]);
    c.X0 = sch.x0 - 4 + tx * kOutW;                 // storage x of the first computed cell
    c.Y0 = sch.y0 + ty * Cfg::OH - (T - 1);         // block y of computed row 0
    c.zs = max(sch.z0 + zc * sch.Lz, lo[2]);
    c.ze = min(sch.z0 + (zc + 1) * sch.Lz - 1, hi[2]);   // output planes [zs, ze]
    if (c.zs > c.ze) return;
    const int ox0 = c.X0 + 4 - L.xoff, oy0 = c.Y0 + T - 1;   // first stored cell (block x, y)
    if (ox0 > hi[0] || ox0 + kOutW - 1 < lo[0] || oy0 > hi[1] || oy0 + Cfg::OH - 1 < lo[1]) return;
    c.first = c.zs - T;
    c.np = c.ze + T - c.first + 1;
    c.tmap = &tin;
    if (c.tid == 0)
        for (int s = 0; s < kSlots && s < c.np; ++s) {
            mbar_expect_tx(&c.bar[s], Cfg::SLOT * 4);
            tma_load_4d(ring + s * Cfg::SLOT, &tin, c.X0, c.Y0 - 1, c.first + s, c.blk, &c.bar[s]);
        }
    c.C = C;
    c.plane = L.plane;
    c.P = L.P;
    c.ring = ring + kBoxW;                          // row 0 of the computed rows (thread 0 of the refill)
    const int wrow = kRY * c.warp, xb = c.X0 + 4 * lane - L.xoff, ya = c.Y0 + wrow;
    // the fixed-shell layer next to the window on fixed faces
    c.zk0 = ((edge >> 4) & 1) ? L.H - 1 : INT_MIN;
    c.zk1 = ((edge >> 5) & 1) ? L.n[2] - L.H : INT_MIN;
    c.xkm = c.ykm = c.mst = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int x = xb + j;
        const bool k = ((edge & 1) && x == L.H - 1) || (((edge >> 1) & 1) && x == L.n[0] - L.H);
        c.xkm |= (k ? 1u : 0u) << j;
    }
#pragma unroll
    for (int r = 0; r < kRY; ++r) {
        const int y = ya + r;
        const bool k = (((edge >> 2) & 1) && y == L.H - 1) || (((edge >> 3) & 1) && y == L.n[1] - L.H);
        c.ykm |= (k ? 1u : 0u) << r;
        const bool in = y >= lo[1] && y <= hi[1] && wrow + r >= T - 1 && wrow + r <= Cfg::ROWS - T && lane >= 1 &&
                        lane <= 30;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            c.mst |= (in && xb + j >= lo[0] && xb + j <= hi[0] ? 1u : 0u) << (4 * r + j);
    }
    c.xkw = __any_sync(0xffffffffu, c.xkm != 0);
    const bool zedge = (c.zk0 >= c.first && c.zk0 <= c.ze + T) || (c.zk1 >= c.first && c.zk1 <= c.ze + T);
    c.edge = __syncthreads_or(c.xkm || c.ykm) || zedge;
    c.dst = out + (long long)c.blk * L.bstride + (long long)(c.first - T) * L.plane + (long long)ya * L.P + c.X0 +
            4 * lane;
    c.ring += wrow * kBoxW + 4 * lane;
    c.xch += 4 * lane;
#pragma unroll
    for (int s = 0; s < T; ++s)
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int r = 0; r < kRY; ++r) c.q[s][k][r] = make_float4(0.f, 0.f, 0.f, 0.f);
    int pr = 0;
    bool ok = true;
    while (pr < c.np) {
        if (!(ok = r_iter<T, NW, 0>(c, pr++)) || pr >= c.np) break;
        if (!(ok = r_iter<T, NW, 1>(c, pr++)) || pr >= c.np) break;
        if (!(ok = r_iter<T, NW, 2>(c, pr++))) break;
    }
    if (!ok && c.tid == 0) {
        // the loads still in flight land before the CTA leaves (bounded)
        report(status, DEV_TIMEOUT);
        for (int g = pr - 1; g < min(c.np, pr - 2 + kSlots); ++g)
            mbar_wait_bounded(&c.bar[g % kSlots], (g / kSlots) & 1, 100000000ull);
    }
}

// Output planes per unit: the count of z chunks that leaves the busiest SM
// the fewest planes, a unit reading T planes beyond its chunk on each side
// and costing about two more to start.
int r_chunk(long long tiles, int NZ, int T, int sms, long long& least)
{
    int best = NZ;
    least = 1ll << 62;
    for (int n = 1; n <= NZ; ++n) {
        const int lz = (NZ + n - 1) / n;
        if (n > 1 && lz < 4) break;
        const long long cost = (tiles * ((NZ + lz - 1) / lz) + sms - 1) / sms * (lz + 2 * T + 2);
        if (cost < least) {
            least = cost;
            best = lz;
        }
    }
    return best;
}

template <int T, int NW>
HeatTiles r_sched(const BlockLayout& L, int step_i, int sms, long long& cost)
{
    // tiles over the union of the blocks' windows after the pass
    int lo[3] = {1 << 30, 1 << 30, 1 << 30}, hi[3] = {-1, -1, -1};
    for (int b = 0; b < L.nblk; ++b)
        for (int a = 0; a < 3; ++a) {
            int l, h;
            stage_region(L, edge_bits(L, b), a, step_i + T, l, h);
            lo[a] = std::min(lo[a], l);
            hi[a] = std::max(hi[a], h);
        }
    HeatTiles sch;
    sch.rows = RCfg<T, NW>::ROWS;
    sch.x0 = (L.xoff + lo[0]) & ~3;
    sch.y0 = lo[1];
    sch.z0 = lo[2];
    const int NZ = std::max(1, hi[2] - lo[2] + 1);
    sch.ntx = std::max(0, L.xoff + hi[0] - sch.x0) / kOutW + 1;
    sch.nty = (std::max(1, hi[1] - lo[1] + 1) + RCfg<T, NW>::OH - 1) / RCfg<T, NW>::OH;
    sch.Lz = r_chunk((long long)sch.ntx * sch.nty * L.nblk, NZ, T, sms, cost);
    sch.nzc = (NZ + sch.Lz - 1) / sch.Lz;
    return sch;
}

template <int T, int NW>
cudaError_t launch_r(const CUtensorMap* tin, float* out, const BlockLayout& L, int step_i, const HeatCoef& c,
                     int* status, cudaStream_t st, HeatTiles& sch)
{
    using Cfg = RCfg<T, NW>;
    static KernelSetup setup;
    int total = 0;      // one CTA per SM
    if (cudaError_t e = kernel_setup(setup, heat_rows_kernel<T, NW>, 32 * NW, Cfg::SMEM, nullptr, &total)) return e;
    long long cost;
    if (!sch.rows) sch = r_sched<T, NW>(L, step_i, total, cost);
    return launch_pdl(heat_rows_kernel<T, NW>, (unsigned)((long long)sch.ntx * sch.nty * L.nblk * sch.nzc), 32 * NW,
                      Cfg::SMEM, st, *tin, out, L, step_i, c, sch, status);
}

constexpr int kNW2 = 12, kNW3 = 12, kNW4 = 8;   // warps by steps per pass

}  // namespace

int heat_rows_box_w() { return kBoxW; }
// three steps per pass: a plane takes a CTA 1.05 to 1.2 us
double heat_rows_us(const BlockLayout& L)
{
    long long cost;
    r_sched<3, kNW3>(L, 0, 152, cost);
    return 1.12 * (double)cost;
}
int heat_rows_box_h(int T) { return kRY * (T == 2 ? kNW2 : T == 3 ? kNW3 : kNW4) + 2; }

cudaError_t launch_heat_rows(int T, const CUtensorMap* tin, float* out, const BlockLayout& L, int step_i,
                             const HeatCoef& c, int* status, cudaStream_t st, HeatTiles& tiles)
{
    switch (T) {
    case 2: return launch_r<2, kNW2>(tin, out, L, step_i, c, status, st, tiles);
    case 3: return launch_r<3, kNW3>(tin, out, L, step_i, c, status, st, tiles);
    case 4: return launch_r<4, kNW4>(tin, out, L, step_i, c, status, st, tiles);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace b2r
