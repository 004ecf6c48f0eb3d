// heat_adjoint.cu -- receiver-misfit gradient of the heat model with respect
// to a per-cell conductivity field kappa (no reference counterpart).
//
// Differentiable form of the heat step (delta D, one block, fixed shell):
//   u^{n+1} = u^n + kappa * (L u^n)          on the interior window W
// where L is the reference's FD Laplacian of order 2D times alpha*dt/dx^2
// per axis (the stencil of fdm_heat_diffuse_deltaD, heat-3D.cu:15-28): with
// kappa = 1 this is the plain heat step.  d_n = u^{n+1}(receivers),
// J = 1/2 sum_n sum_r (d_n,r - obs_n,r)^2.  Reverse step n, lam = adjoint
// of u^{n+1}:
//   lam(rec) += d_n - obs_n
//   g_kappa  += lam * (L u^n)                 on W   (FP32 increment, FP64 sum)
//   y         = kappa * lam on W, 0 elsewhere
//   lam      += L^T y = L y                   on W   (L is symmetric)
// u^n is replayed from checkpoints every K steps.
//
// Measured (radius 2, 160x144x128, 200 steps, checkpoints every 50, 64
// receivers, the whole gradient call): 9.1 ms, from 61 with a thread per
// column over the whole z axis, the reverse step in two sweeps, and a
// separate launch for every receiver sample.
#include <algorithm>
#include <vector>

#include "b2r_common.cuh"
#include "eqwp_tile.cuh"
#include "heat.h"

namespace b2r {

namespace {

using namespace eqk;   // a thread's 4 cells, z chunks, masked float4 reads and writes (eqwp_tile.cuh)

// A field whose stencil a thread needs while it marches z: the 2D+1 planes of
// its 4 cells in a register queue, x neighbours from the float4s on both
// sides of the row and y neighbours from the rows +-1 .. +-D, through L1.
template <int D>
struct LapField {
    const float* p;            // the thread's cells in plane 0
    float4 q[2 * D + 1];
    __device__ __forceinline__ void begin(const float* f, int zs, long long S)
    {
        p = f;
#pragma unroll
        for (int k = 0; k < 2 * D; ++k) q[k + 1] = ld4(p + (long long)(zs - D + k) * S);
    }
    // L u of the 4 cells at plane z (element offset o); planes in increasing
    // order.  w0 u + sum_k (wx_k (u[x+k] + u[x-k]) + wy_k (...) + wz_k (...)):
    // the first x product rounded, w0 u and then every other product fused
    // onto the running sum, in this order in every kernel.
    __device__ __forceinline__ void lap(long long o, long long P, long long S, const HeatLap& c, float (&acc)[4])
    {
#pragma unroll
        for (int k = 0; k < 2 * D; ++k) q[k] = q[k + 1];
        q[2 * D] = ld4(p + o + D * S);
        const float4 l = ld4(p + o - 4), m = q[D], r = ld4(p + o + 4);
        float4 ym[D], yp[D];
#pragma unroll
        for (int k = 1; k <= D; ++k) {
            ym[k - 1] = ld4(p + o - k * P);
            yp[k - 1] = ld4(p + o + k * P);
        }
        const float v[12] = {l.x, l.y, l.z, l.w, m.x, m.y, m.z, m.w, r.x, r.y, r.z, r.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float a = __fmaf_rn(c.w0, v[4 + j], __fmul_rn(c.wx[0], __fadd_rn(v[5 + j], v[3 + j])));
#pragma unroll
            for (int k = 1; k <= D; ++k) {
                if (k > 1) a = __fmaf_rn(c.wx[k - 1], __fadd_rn(v[4 + j + k], v[4 + j - k]), a);
                a = __fmaf_rn(c.wy[k - 1], __fadd_rn(cmp(yp[k - 1], j), cmp(ym[k - 1], j)), a);
                a = __fmaf_rn(c.wz[k - 1], __fadd_rn(cmp(q[D + k], j), cmp(q[D - k], j)), a);
            }
            acc[j] = a;
        }
    }
};

// One conductivity-scaled step.  rec_out (may be null): the receivers of
// `in`, that is of the step before, sampled on the way.
template <int D>
__global__ void __launch_bounds__(kBX * kBY)
heat_kappa_step_kernel(const float* __restrict__ in, float* __restrict__ out, const float* __restrict__ kappa,
                       const BlockLayout L, const HeatLap c, const Tiles T, const long long* __restrict__ rec, int nrec,
                       float* __restrict__ rec_out)
{
    pdl_begin();
    if (rec_out)
        for (unsigned r = grid_thread(); r < (unsigned)nrec; r += grid_threads()) rec_out[r] = in[rec[r]];
    const Win w = window(L, 0, blockIdx.z, T.nzc, L.H);
    Cell cell;
    if (!cell_setup(L, w, 0, cell, T.x0, T.y0)) return;
    const long long P = L.P, S = L.plane;
    LapField<D> u;
    u.begin(in + cell.base, w.zs, S);
    for (int z = w.zs; z <= w.ze; ++z) {
        const long long o = (long long)z * S;
        const float4 kap = ld4(kappa + cell.base + o);
        float a[4];
        u.lap(o, P, S, c, a);
        const float4 m = u.q[D];
        const float nv[4] = {__fmaf_rn(kap.x, a[0], m.x), __fmaf_rn(kap.y, a[1], m.y), __fmaf_rn(kap.z, a[2], m.z),
                             __fmaf_rn(kap.w, a[3], m.w)};
        st4(out + cell.base + o, cell, nv);
    }
}

// One reverse step in one sweep: with lam the adjoint of u^{n+1} (receivers
// added) and y = kappa lam on W, 0 elsewhere,
//     g += lam * (L u^n),  lam += L y,  y_next = kappa lam.
// lam and g are read and written by their own thread only; y, whose stencil
// the neighbours need, goes from one buffer to the other.  40 B per cell (u,
// y, lam and kappa read, lam and y written, g read and written in FP64)
// against 52 in two sweeps.
template <int D>
__global__ void __launch_bounds__(kBX * kBY, 2)
heat_adj_step_kernel(float* __restrict__ lam, const float* __restrict__ y, float* __restrict__ y_next,
                     const float* __restrict__ un, const float* __restrict__ kappa, double* __restrict__ g,
                     const BlockLayout L, const HeatLap c, const Tiles T)
{
    pdl_begin();
    const Win w = window(L, 0, blockIdx.z, T.nzc, L.H);
    Cell cell;
    if (!cell_setup(L, w, 0, cell, T.x0, T.y0)) return;
    const long long P = L.P, S = L.plane;
    LapField<D> u, yb;
    u.begin(un + cell.base, w.zs, S);
    yb.begin(y + cell.base, w.zs, S);
    for (int z = w.zs; z <= w.ze; ++z) {
        const long long o = (long long)z * S;
        const float4 kap = ld4(kappa + cell.base + o);
        const float4 l4 = rd4(lam + cell.base + o, cell);
        double2* gp = reinterpret_cast<double2*>(g + cell.base + o);   // x groups start on 4 elements
        double2 g0 = make_double2(0.0, 0.0), g1 = g0;
        if (cell.all) {
            g0 = gp[0];
            g1 = gp[1];
        }
        float au[4], ay[4];
        u.lap(o, P, S, c, au);
        yb.lap(o, P, S, c, ay);
        float nl[4], ny[4];
        double inc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float l = cmp(l4, j);
            inc[j] = (double)__fmul_rn(l, au[j]);
            nl[j] = __fadd_rn(l, ay[j]);
            ny[j] = __fmul_rn(cmp(kap, j), nl[j]);
        }
        st4(lam + cell.base + o, cell, nl);
        st4(y_next + cell.base + o, cell, ny);
        if (cell.all) {
            gp[0] = make_double2(g0.x + inc[0], g0.y + inc[1]);
            gp[1] = make_double2(g1.x + inc[2], g1.y + inc[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (cell.vx[j]) g[cell.base + o + j] += inc[j];
        }
    }
}

// The residuals of a step into lam at the receivers, and y = kappa lam there:
// receivers that share a cell are all added before y is formed, by a barrier
// where one CTA does both, by two launches where there are many receivers (on
// 128^3, 40 steps, the whole gradient with one CTA for this and the samples, and
// now: 16384 receivers 4.4 and 2.1 ms, 262144 58 and 17).
constexpr int kInjectCta = 1024;
template <bool ADD, bool FORM>
__global__ void __launch_bounds__(kInjectCta)
heat_adj_inject_kernel(float* lam, float* y, const float* kappa, const long long* rec, int nrec, const float* res)
{
    pdl_begin();
    const int r = blockIdx.x * kInjectCta + threadIdx.x;
    if (ADD && r < nrec) atomicAdd(&lam[rec[r]], res[r]);
    if (ADD && FORM) __syncthreads();
    if (FORM && r < nrec) y[rec[r]] = __fmul_rn(kappa[rec[r]], *(volatile float*)&lam[rec[r]]);
}

// The fixed shell of `src` (the D cells around the window on every axis, the
// only cells outside it that a stencil reads) into n buffers `stride`
// elements apart.  A warp takes one row of one buffer.
__global__ void heat_shell_kernel(const float* __restrict__ src, float* __restrict__ dst, long long stride, int n,
                                  const BlockLayout L, int D)
{
    const int lane = threadIdx.x & 31;
    const int lo[3] = {L.H - D, L.H - D, L.H - D};
    const int e[3] = {L.B[0] + 2 * D, L.B[1] + 2 * D, L.B[2] + 2 * D};
    const long long rows = (long long)e[1] * e[2] * n;
    for (long long i = blockIdx.x * 8LL + (threadIdx.x >> 5); i < rows; i += gridDim.x * 8LL) {
        const int y = (int)(i % e[1]);
        const long long r = i / e[1];
        const int z = (int)(r % e[2]);
        const long long o = (long long)(lo[2] + z) * L.plane + (long long)(lo[1] + y) * L.P + L.xoff + lo[0];
        float* d = dst + (r / e[2]) * stride + o;
        const bool whole = y < D || y >= e[1] - D || z < D || z >= e[2] - D;
        if (whole) {
            for (int x = lane; x < e[0]; x += 32) d[x] = src[o + x];
        } else if (lane < 2 * D) {
            const int x = lane < D ? lane : e[0] - 2 * D + lane;
            d[x] = src[o + x];
        }
    }
}

__global__ void fill_kernel(float* p, size_t n, float v)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        p[i] = v;
}

}  // namespace

cudaError_t launch_fill(float* p, size_t n, float v, cudaStream_t st)
{
    const size_t blocks = std::min<size_t>((n + 255) / 256, 152 * 16);
    fill_kernel<<<(unsigned)std::max<size_t>(blocks, 1), 256, 0, st>>>(p, n, v);
    count_launches(1);
    return cudaGetLastError();
}

// Planes per z chunk, as stage_chunk (eqwp_tile.cuh) with these kernels'
// costs: a chunk's start about one plane's latency, a plane of a lone CTA
// 1.075 and of n resident ones 0.9 + 0.175 n (per_sm of them fit).  Measured
// on the whole gradient by forward / reverse planes: radius 2, 160x144x128,
// 11.1 ms at 8/8, 10.2 at 6/8 and 8/6, 10.4 at 8/4; 64x72x60 2.97 at 8/8,
// 1.90 at 1/8, 2.32 at 8/1; radius 3, 100x90x110, 3.54 at 8/8, 3.20 at 8/4,
// 3.60 at 8/1.
static int heat_chunk(long long tiles, int nz, int per_sm)
{
    int best = 1;
    double least = 1e300;
    for (int lz = 1; lz <= 8 && lz <= nz; ++lz) {
        const long long q = (tiles * ((nz + lz - 1) / lz) + 151) / 152;
        auto together = [&](long long n) { return n > 0 ? 1.0 + lz * (0.9 + 0.175 * (double)n) : 0.0; };
        const double cost = (double)(q / per_sm) * together(per_sm) + together(q % per_sm);
        if (cost < least) {
            least = cost;
            best = lz;
        }
    }
    return best;
}

HeatLap heat_lap(int D, double alpha_dt, double dx, double dy, double dz)
{
    static const double cw[5][5] = {
        {0, 0, 0, 0, 0},
        {-2.0, 1.0, 0, 0, 0},
        {-5.0 / 2.0, 4.0 / 3.0, -1.0 / 12.0, 0, 0},
        {-49.0 / 18.0, 3.0 / 2.0, -3.0 / 20.0, 1.0 / 90.0, 0},
        {-205.0 / 72.0, 8.0 / 5.0, -1.0 / 5.0, 8.0 / 315.0, -1.0 / 560.0}};
    const double wx = alpha_dt / (dx * dx), wy = alpha_dt / (dy * dy), wz = alpha_dt / (dz * dz);
    HeatLap c{};
    c.w0 = (float)(cw[D][0] * (wx + wy + wz));
    for (int k = 1; k <= D; ++k) {
        c.wx[k - 1] = (float)(wx * cw[D][k]);
        c.wy[k - 1] = (float)(wy * cw[D][k]);
        c.wz[k - 1] = (float)(wz * cw[D][k]);
    }
    return c;
}

#define B2R_HEAT_ADJ_DISPATCH(D, CALL) \
    switch (D) {                       \
    case 1: CALL(1); break;            \
    case 2: CALL(2); break;            \
    case 3: CALL(3); break;            \
    case 4: CALL(4); break;            \
    default: return cudaErrorInvalidValue; \
    }

cudaError_t launch_heat_kappa_step(const float* in, float* out, const float* kappa, const BlockLayout& L, int D,
                                   const HeatLap& c, const long long* rec, int nrec, float* rec_out, cudaStream_t st)
{
    const Grid g = stage_grid(L, L.H, D <= 2 ? 4 : 3, heat_chunk);
#define CALL(DD) return launch_pdl(heat_kappa_step_kernel<DD>, g.g, g.b, 0, st, in, out, kappa, L, c, g.t, rec, nrec, rec_out)
    B2R_HEAT_ADJ_DISPATCH(D, CALL)
#undef CALL
    return cudaSuccess;
}

cudaError_t launch_heat_adjoint_step(float* lam, const float* y, float* y_next, const float* u, const float* kappa,
                                     double* g, const BlockLayout& L, int D, const HeatLap& c, cudaStream_t st)
{
    const Grid gr = stage_grid(L, L.H, D == 1 ? 3 : 2, heat_chunk);
#define CALL(DD) return launch_pdl(heat_adj_step_kernel<DD>, gr.g, gr.b, 0, st, lam, y, y_next, u, kappa, g, L, c, gr.t)
    B2R_HEAT_ADJ_DISPATCH(D, CALL)
#undef CALL
    return cudaSuccess;
}

cudaError_t launch_heat_adjoint_inject(float* lam, float* y, const float* kappa, const long long* rec, int nrec,
                                       const float* res, cudaStream_t st)
{
    const int ctas = (nrec + kInjectCta - 1) / kInjectCta;
    if (ctas == 1)
        return launch_pdl(heat_adj_inject_kernel<true, true>, 1, (nrec + 31) / 32 * 32, 0, st, lam, y, kappa, rec, nrec, res);
    if (cudaError_t e = launch_pdl(heat_adj_inject_kernel<true, false>, ctas, kInjectCta, 0, st, lam, y, kappa, rec, nrec, res))
        return e;
    return launch_pdl(heat_adj_inject_kernel<false, true>, ctas, kInjectCta, 0, st, lam, y, kappa, rec, nrec, res);
}

cudaError_t launch_heat_shell(const float* src, float* dst, long long stride, int n, const BlockLayout& L, int D,
                              cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const long long rows = (long long)(L.B[1] + 2 * D) * (L.B[2] + 2 * D) * n;
    heat_shell_kernel<<<(unsigned)std::min<long long>((rows + 7) / 8, 152LL * 32), 256, 0, st>>>(src, dst, stride, n, L, D);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace b2r
