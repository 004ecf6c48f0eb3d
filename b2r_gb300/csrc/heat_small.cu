// heat_small.cu -- any number of heat time steps of a small domain in one
// launch, radius 1 and 2: the domain lives in the shared memory of one cluster.
//
// A step of a small domain is all latency: a launch, its loads and its drain
// (1.86 us at 48x40x32, two steps per launch) for 0.1 us of arithmetic.  Here a
// cluster of up to 16 CTAs reads the domain once from the blocks of any split,
// each CTA a slab of z planes with its halo, and keeps two copies in shared
// memory.  A thread has 4 cells of one row in up to four planes, in registers
// too, and a step reads one copy and writes the other; the planes next to a
// neighbour are also stored into its halo (st.async, counted on an mbarrier of
// the neighbour's), on a torus the cells that wrap in x and y as well.  So a
// CTA waits for its two neighbours' planes only, and for its own threads.  That
// a neighbour has all of a step's planes means that every read of its halo here
// is done, so the two copies are enough.  At the end the interiors go back into
// the blocks.  Every cell runs the sweep's operations in its order
// (heat_unit.cuh): the same bits.
//
// Measured, us per step and for 20 steps (radius 1, against two steps per
// launch): 48x40x32 0.93, 31 (1.86, 44; in 2x2x1 blocks 52), 32^3 0.58, 23, a
// torus 40x33x32 in 2x1x1 0.92, 31 (3.2, 92); radius 2, 48x40x32 1.75, 50 (3.1,
// 74).  A step with cluster barriers and plain stores to the neighbours: 1.33.
// What bounds it is the rate of shared-memory operations of 16 SMs, so that at
// 64^3 (2.7 against 2.35) the whole GPU is faster.
#include <algorithm>

#include "b2r_common.cuh"
#include "heat.h"

namespace b2r {
namespace {

constexpr int kThr = 1024;
constexpr int kPadX = 4;            // floats before x = 0: the widest halo, and 16-byte rows
constexpr int kMaxCtas = 16;
constexpr int kMaxRun = 4;          // planes per thread
constexpr size_t kSmemMax = 226 * 1024;   // beside the barriers

struct SGeo {
    int e[3];                       // cells
    int P, rows, planes;            // shared layout: floats per row, rows per plane, planes per copy
    int G;                          // float4s per row
    int base, rem;                  // planes per CTA, the first `rem` CTAs one more
    int ctas, run;                  // run: planes per thread
};

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer(uint32_t addr, int rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// 16 bytes into another CTA's shared memory, counted there on the mbarrier
__device__ __forceinline__ void st_peer(uint32_t addr, float4 v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     addr),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ float4 s4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float lane4(const float4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }

// block and block coordinate of the interior cell that holds domain coordinate
// g, or of the shell cell beyond the first / last block; on a torus wrapped
__device__ __forceinline__ int owner(int g, const BlockLayout& M, int a, int e, int& at)
{
    if (M.periodic) g = g < 0 ? g + e : g >= e ? g - e : g;
    int b = g < 0 ? 0 : g / M.B[a];
    b = b < M.nb[a] ? b : M.nb[a] - 1;
    at = g - b * M.B[a] + M.H;
    return b;
}
__device__ __forceinline__ int row_of(const BlockLayout& M, const int (&e)[3], int y, int z)
{
    int cy, cz;
    const int by = owner(y, M, 1, e[1], cy), bz = owner(z, M, 2, e[2], cz);
    return (bz * M.nb[1] + by) * M.nb[0] * (int)M.bstride + cz * (int)M.plane + cy * M.P + M.xoff;
}

template <int D, int ZR>
__global__ void __launch_bounds__(kThr, 1)
heat_small_kernel(float* __restrict__ buf, const BlockLayout M, const SGeo s, const HeatCoef C, const int n,
                  int* __restrict__ status)
{
    extern __shared__ __align__(16) float sm[];
    __shared__ uint64_t bar[2];                          // halos of even and odd steps received
    const int rank = (int)cluster_rank();
    const int z0 = rank * s.base + min(rank, s.rem), nzl = s.base + (rank < s.rem);
    const int plane = s.rows * s.P, copy = s.planes * plane;
    const int origin = D * plane + D * s.P + kPadX;      // cell (0, 0, z0)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;

    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    // rows (y, z) of the slab and its halo, into both copies: a lane finds where
    // one row lies, the warp copies up to 32 of them
    const int ny = s.e[1] + 2 * D, nrow = ny * (nzl + 2 * D);
    for (int rb = warp; rb < nrow; rb += 32 * warps) {
        const int mine = min(rb + lane * warps, nrow - 1), mz = mine / ny - D, my = mine - (mz + D) * ny - D;
        const int from = row_of(M, s.e, my, z0 + mz), into = origin + mz * plane + my * s.P;
        const int have = min(32, (nrow - rb + warps - 1) / warps);
        for (int xb = -D; xb < s.e[0] + D; xb += 32) {
            const int x = xb + lane;
            const bool in = x < s.e[0] + D;
            int cx = 0;
            const int bx = in ? owner(x, M, 0, s.e[0], cx) * (int)M.bstride + cx : 0;
            for (int u0 = 0; u0 < have; u0 += 8) {
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int f = __shfl_sync(0xffffffffu, from, min(u0 + u, have - 1));
                    v[u] = in ? buf[f + bx] : 0.f;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    float* d = sm + __shfl_sync(0xffffffffu, into, min(u0 + u, have - 1)) + x;
                    if (in) d[0] = d[copy] = v[u];
                }
            }
        }
    }
    // the thread's column: 4 cells of row y, ZR planes from zr on; a thread too
    // many works on the last column, and planes beyond the slab are worked on
    // too, but none of that is stored
    const int cols = s.G * s.e[1], items = cols * ((nzl + ZR - 1) / ZR);
    const int it = min((int)threadIdx.x, items - 1);
    const int zr = it / cols * ZR, y = it % cols / s.G, g = it % s.G;
    const int nzr = min(ZR, nzl - zr);
    const int left = s.e[0] - 4 * g;                     // cells of the row from here on
    const int o = zr * plane + y * s.P + 4 * g;
    const bool first = g == 0 || lane == 0, last = g == s.G - 1 || lane == 31;
    const bool k1 = left > 1, k2 = left > 2, k3 = left > 3;
    const int store = (int)threadIdx.x < items ? nzr : 0;   // planes stored
    // where the neighbours' copies of this CTA's outer planes lie (shared
    // addresses of cell (0, 0, plane 0 of this CTA) as the neighbour counts, which
    // may lie before its memory, at 0 even)
    const uint32_t here = smem_u32(sm) + 4u * (uint32_t)origin;
    uint32_t below = 0, above = 0, bar_below = 0, bar_above = 0;
    const bool has_below = rank > 0 || M.periodic, has_above = rank < s.ctas - 1 || M.periodic;
    if (has_below) {
        const int q = rank > 0 ? rank - 1 : s.ctas - 1;
        bar_below = peer(smem_u32(bar), q);
        below = peer(here, q) + 4u * (uint32_t)((s.base + (q < s.rem)) * plane);
    }
    if (has_above) {
        const int q = rank < s.ctas - 1 ? rank + 1 : 0;
        bar_above = peer(smem_u32(bar), q);
        above = peer(here, q) - 4u * (uint32_t)(nzl * plane);
    }
    const uint32_t bytes = 16u * (uint32_t)(D * cols) * ((has_below ? 1 : 0) + (has_above ? 1 : 0));   // received per step
    const bool waits = (has_below && zr < D) || (has_above && zr + nzr > nzl - D);
    // planes stored there: the first `down`, and from `up` on
    const int down = has_below ? min(store, D - zr) : 0, up = has_above ? max(0, nzl - D - zr) : ZR;
    const float2 a0 = make_float2(C.a0, C.a0);
    cluster_sync();

    float4 w[ZR + 2 * D];                                // planes zr-D .. zr+ZR+D-1, the own ones kept from step to step
#pragma unroll
    for (int j = 0; j < ZR; ++j) w[D + j] = s4(sm + origin + o + j * plane);
    bool bad = false;
    for (int t = 0; t < n; ++t) {
        if (threadIdx.x == 0 && bytes) mbar_expect_tx(&bar[t & 1], bytes);
        if (waits && t > 0) bad = !mbar_wait_bounded(&bar[(t - 1) & 1], ((t - 1) >> 1) & 1);
        const float* src = sm + (t & 1) * copy + origin + o;
        const int to = copy - 2 * (t & 1) * copy;        // to the same cell of the other copy
#pragma unroll
        for (int j = 0; j < D; ++j) {
            w[j] = s4(src + (j - D) * plane);
            w[D + ZR + j] = s4(src + (ZR + j) * plane);
        }
        if (nzr < ZR) {
#pragma unroll
            for (int j = 1; j < ZR; ++j)
                if (j >= nzr) w[D + j] = s4(src + j * plane);
        }
        if (M.periodic && !k3) {                         // cells of the torus's other end in the float4
#pragma unroll
            for (int j = 0; j < ZR; ++j) w[D + j] = s4(src + j * plane);
        }
        float4 nw[ZR];
#pragma unroll
        for (int j = 0; j < ZR; ++j) {
            const float* p = src + j * plane;
            const float4 c = w[D + j];
            float x[4 + 2 * D];
            x[D] = c.x;
            x[D + 1] = c.y;
            x[D + 2] = c.z;
            x[D + 3] = c.w;
#pragma unroll
            for (int k = 1; k <= D; ++k) {
                x[D - k] = __shfl_up_sync(0xffffffffu, lane4(c, 4 - k), 1);
                x[D + 3 + k] = __shfl_down_sync(0xffffffffu, lane4(c, k - 1), 1);
                if (first) x[D - k] = p[-k];
                if (last) x[D + 3 + k] = p[3 + k];
            }
            float2 lo = __fmul2_rn(a0, make_float2(x[D], x[D + 1])), hi = __fmul2_rn(a0, make_float2(x[D + 2], x[D + 3]));
#pragma unroll
            for (int k = 1; k <= D; ++k) {
                const float2 ax = make_float2(C.ax[k - 1], C.ax[k - 1]), ay = make_float2(C.ay[k - 1], C.ay[k - 1]),
                             az = make_float2(C.az[k - 1], C.az[k - 1]);
                const float4 ym = s4(p - k * s.P), yp = s4(p + k * s.P), zm = w[D + j - k], zp = w[D + j + k];
                lo = __ffma2_rn(ax, make_float2(x[D - k] + x[D + k], x[D + 1 - k] + x[D + 1 + k]), lo);
                hi = __ffma2_rn(ax, make_float2(x[D + 2 - k] + x[D + 2 + k], x[D + 3 - k] + x[D + 3 + k]), hi);
                lo = __ffma2_rn(ay, __fadd2_rn(make_float2(ym.x, ym.y), make_float2(yp.x, yp.y)), lo);
                hi = __ffma2_rn(ay, __fadd2_rn(make_float2(ym.z, ym.w), make_float2(yp.z, yp.w)), hi);
                lo = __ffma2_rn(az, __fadd2_rn(make_float2(zm.x, zm.y), make_float2(zp.x, zp.y)), lo);
                hi = __ffma2_rn(az, __fadd2_rn(make_float2(zm.z, zm.w), make_float2(zp.z, zp.w)), hi);
            }
            // cells beyond the row's end keep their value
            nw[j] = make_float4(lo.x, k1 ? lo.y : c.y, k2 ? hi.x : c.z, k3 ? hi.y : c.w);
        }
        float* dst = sm + (src - sm) + to;
        const uint32_t at = 4u * (uint32_t)((int)(src - sm) - origin + to);
#pragma unroll
        for (int j = 0; j < ZR; ++j) {
            const float4 v = w[D + j] = nw[j];
            if (j < store) {
                float* d = dst + j * plane;
                if (!M.periodic || k3) {
                    *reinterpret_cast<float4*>(d) = v;
                } else {
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (k < left) d[k] = lane4(v, k);
                }
                // beyond the row's end nobody reads a neighbour's halo
                if (j < down) st_peer(below + at + 4u * (uint32_t)(j * plane), v, bar_below + 8u * (t & 1));
                if (j >= up) st_peer(above + at + 4u * (uint32_t)(j * plane), v, bar_above + 8u * (t & 1));
                if (M.periodic) {
                    // an axis of fewer than 2D cells wraps both ways
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int xx = 4 * g + k;
                        const float u = lane4(v, k);
                        if (k >= left) continue;
                        if (y < D) d[k + s.e[1] * s.P] = u;
                        if (y >= s.e[1] - D) d[k - s.e[1] * s.P] = u;
                        if (xx < D) d[k + s.e[0]] = u;
                        if (xx >= s.e[0] - D) d[k - s.e[0]] = u;
                    }
                }
            }
        }
        if (__syncthreads_or(bad)) break;
    }
    if (bad) report(status, DEV_TIMEOUT);
    // the last step's halos have arrived everywhere before a CTA leaves
    if (n > 0 && bytes) mbar_wait_bounded(&bar[(n - 1) & 1], ((n - 1) >> 1) & 1);
    cluster_sync();
    // the interiors back
    const float* res = sm + (n & 1) * copy;
    const int rows = s.e[1] * nzl;
    for (int rb = warp; rb < rows; rb += 32 * warps) {
        const int mine = min(rb + lane * warps, rows - 1), mz = mine / s.e[1], my = mine - mz * s.e[1];
        const int into = row_of(M, s.e, my, z0 + mz), from = origin + mz * plane + my * s.P;
        const int have = min(32, (rows - rb + warps - 1) / warps);
        for (int xb = 0; xb < s.e[0]; xb += 32) {
            const int x = xb + lane;
            int cx = 0;
            const int bx = x < s.e[0] ? owner(x, M, 0, s.e[0], cx) * (int)M.bstride + cx : 0;
            for (int u = 0; u < have; ++u) {
                const int d = __shfl_sync(0xffffffffu, into, u), f = __shfl_sync(0xffffffffu, from, u);
                if (x < s.e[0]) buf[d + bx] = res[f + x];
            }
        }
    }
}

// layout of the domain on `ctas` CTAs, the fewest planes per thread with which
// 1024 threads take a slab; bytes of shared memory, 0 if there is no such run
size_t s_geo(const int e[3], int D, int ctas, SGeo& s)
{
    for (int a = 0; a < 3; ++a) s.e[a] = e[a];
    s.G = (e[0] + 3) / 4;
    s.P = kPadX + 4 * s.G + 4;
    s.rows = e[1] + 2 * D;
    s.ctas = ctas;
    s.base = e[2] / ctas;
    s.rem = e[2] % ctas;
    const int nz = s.base + (s.rem > 0);
    for (s.run = 1; s.run <= kMaxRun; ++s.run) {
        const int runs = (nz + s.run - 1) / s.run;
        if ((long long)s.G * e[1] * runs > kThr) continue;
        s.planes = runs * s.run + 2 * D;     // a run may reach beyond the slab
        return 2 * sizeof(float) * (size_t)s.planes * s.rows * s.P;
    }
    return 0;
}

using Kernel = void (*)(float*, BlockLayout, SGeo, HeatCoef, int, int*);
template <int D>
Kernel s_kernel(int zr)
{
    return zr == 1 ? heat_small_kernel<D, 1> : zr == 2 ? heat_small_kernel<D, 2> : zr == 3 ? heat_small_kernel<D, 3>
                                                                                             : heat_small_kernel<D, 4>;
}
Kernel s_kernel(int D, int zr) { return D == 1 ? s_kernel<1>(zr) : s_kernel<2>(zr); }
cudaLaunchConfig_t s_config(int ctas, int threads, size_t smem, cudaStream_t st, cudaLaunchAttribute* attr)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

double heat_small_us(const int e[3], int D, int ctas)
{
    SGeo s;
    s_geo(e, D, ctas, s);
    return 0.3 + (D == 1 ? 0.00065 : 0.0015) * s.G * e[1] * (s.base + (s.rem > 0));
}

int heat_small_ctas(const int e[3], int D)
{
    if (D > 2) return 0;
    for (int ctas = std::min(kMaxCtas, e[2] / D); ctas >= 1; --ctas) {
        SGeo s;
        const size_t smem = s_geo(e, D, ctas, s);
        if (smem > kSmemMax || !smem) return 0;     // fewer CTAs need more
        const Kernel k = s_kernel(D, s.run);
        cudaLaunchAttribute attr[1];
        const cudaLaunchConfig_t cfg = s_config(ctas, kThr, smem, nullptr, attr);
        int clusters = 0;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess && clusters >= 1)
            return ctas;
        cudaGetLastError();
    }
    return 0;
}

cudaError_t launch_heat_small(float* buf, const BlockLayout& M, const int e[3], int D, int ctas, const HeatCoef& c,
                              int nsteps, int* status, cudaStream_t st)
{
    SGeo s;
    const size_t smem = s_geo(e, D, ctas, s);
    const int items = s.G * s.e[1] * ((s.base + (s.rem > 0) + s.run - 1) / s.run);
    const int threads = std::max(256, (items + 31) / 32 * 32);
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = s_config(ctas, threads, smem, st, attr);
    constexpr int kSteps = 2048;             // a few milliseconds per launch
    for (int done = 0; done < nsteps; done += kSteps) {
        const cudaError_t e2 = cudaLaunchKernelEx(&cfg, s_kernel(D, s.run), buf, M, s, c, std::min(kSteps, nsteps - done),
                                                  status);
        if (e2 != cudaSuccess) return e2;
        count_launches(1);
    }
    return cudaGetLastError();
}

}  // namespace b2r
