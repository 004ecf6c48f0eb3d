// heat.h -- internal interface of the heat sweep kernels (heat.cu).
#pragma once
#include "b2r_common.cuh"

namespace b2r {

// Folded stencil weights: u' = a0*u + sum_k ax[k-1]*(u[x-k]+u[x+k]) + ... .
struct HeatCoef {
    float a0;
    float ax[4], ay[4], az[4];
};

HeatCoef heat_coef(int D, double alpha_dt, double dx, double dy, double dz);

// heat_adjoint.cu: the Laplacian of order 2D times alpha*dt/dx^2 per axis,
// L u = w0*u + sum_k wx[k-1]*(u[x-k]+u[x+k]) + ...; the conductivity-scaled
// step u' = u + kappa * L u on the interior window of one block, and one
// reverse step of its adjoint (lam: adjoint of u^{n+1}, updated to that of
// u^n; y zero outside the window; g += lam * L u^n in FP64).
struct HeatLap {
    float w0;
    float wx[4], wy[4], wz[4];
};
HeatLap heat_lap(int D, double alpha_dt, double dx, double dy, double dz);
// launch_heat_kappa_step also samples the receivers of `in` (element offsets
// rec) into rec_out unless that is null.  launch_heat_adjoint_step: lam and g
// in place, y = kappa * lam read, y_next written; launch_heat_adjoint_inject
// adds the residuals at the receivers to lam and refreshes y there.
// launch_heat_shell copies src's fixed shell into n fields `stride` elements
// apart.
cudaError_t launch_heat_kappa_step(const float* in, float* out, const float* kappa, const BlockLayout& L, int D,
                                   const HeatLap& c, const long long* rec, int nrec, float* rec_out, cudaStream_t st);
cudaError_t launch_heat_adjoint_step(float* lam, const float* y, float* y_next, const float* u, const float* kappa,
                                     double* g, const BlockLayout& L, int D, const HeatLap& c, cudaStream_t st);
cudaError_t launch_heat_adjoint_inject(float* lam, float* y, const float* kappa, const long long* rec, int nrec,
                                       const float* res, cudaStream_t st);
cudaError_t launch_heat_shell(const float* src, float* dst, long long stride, int n, const BlockLayout& L, int D,
                              cudaStream_t st);
cudaError_t launch_fill(float* p, size_t n, float v, cudaStream_t st);
// TMA box of one ring slot (cells): width and height for radius D.
int heat_box_w();
int heat_box_h(int D);
// One sub-step (shrink D*(step_i+1)) of every block: reads the blocks
// through `tin` (a tensor map over the input buffer), writes `out`.
// Launch schedule knobs (the autotuner's search space).
struct HeatTune {
    int zchunk = 0;        // output planes per work unit; 0 = 16 (fewer for small grids)
    int ctas_per_sm = 0;   // 0 = one CTA per unit; k > 0 = persistent, k CTAs per SM
    int pdl = 1;           // programmatic dependent launch on the stream
    int tblock = 2;        // time steps per HBM pass: radius 1 (2 = heat2.cu, 3-4 = heat_tb.cu), radius 2 (2 = heat_tb2.cu, with r2)
    int zchunk2 = 0;       // output planes per unit of the several-step kernels (0 = 16 / 64)
    int tb16 = 0;          // two steps per pass: 0 = heat2.cu (8-warp CTAs), 1 = heat_tb.cu (16 warps)
    int tbn = 0;           // heat_tb.cu tiles: 0 = 128 x 32 cells, 1 = 64 x 64 cells
    int r2 = 0;            // radius 2: 1 = two steps per pass (heat_tb2.cu) when tblock >= 2
    // The library's own rule for the kernel and the steps per pass, while every
    // knob has its default: so knobs read from one handle and set on another
    // choose the same there, and set back they choose the rule again.
    bool own() const
    {
        return zchunk == 0 && ctas_per_sm == 0 && pdl && tblock == 2 && zchunk2 == 0 && !tb16 && !tbn && !r2;
    }
};

// One sub-step of every block: units (block, z-chunk, tile row, tile column)
// dealt round-robin to the CTAs.
cudaError_t launch_heat_substep(const CUtensorMap* tin, float* out, const BlockLayout& L, int D,
                                int step_i, const HeatCoef& c, int* status, cudaStream_t st,
                                const HeatTune& tune = HeatTune());

// Two sub-steps (step_i, step_i+1) of radius 1 per launch (heat2.cu).  The
// tensor map must have the box heat2_box_w() x heat2_box_h().
int heat2_box_w();
int heat2_box_h();
// heat_small.cu: CTAs of the cluster whose shared memory holds the domain of e
// cells, 0 if none does; nsteps steps of the interiors of buf's blocks (the
// halos between blocks are left behind).
int heat_small_ctas(const int e[3], int D);
double heat_small_us(const int e[3], int D, int ctas);   // a step's estimate
cudaError_t launch_heat_small(float* buf, const BlockLayout& M, const int e[3], int D, int ctas, const HeatCoef& c,
                              int nsteps, int* status, cudaStream_t st);
// Estimates of one pass: two steps (heat2.cu), three steps (heat_rows.cu).
double heat2_us(const BlockLayout& L);
double heat_rows_us(const BlockLayout& L);
cudaError_t launch_heat_substep2(const CUtensorMap* tin, float* out, const BlockLayout& L, int step_i,
                                 const HeatCoef& c, int* status, cudaStream_t st, int zchunk);

// Two sub-steps (step_i, step_i+1) of radius 2 per launch (heat_tb2.cu),
// on tiles of 64 x 64 cells.  The tensor map must have the box
// heat_tb2_box_w() x heat_tb2_box_h().
int heat_tb2_box_w();
int heat_tb2_box_h();
cudaError_t launch_heat_substep_tb2(const CUtensorMap* tin, float* out, const BlockLayout& L, int step_i,
                                    const HeatCoef& c, int* status, cudaStream_t st, int zchunk);

// T = 2, 3 or 4 sub-steps (step_i .. step_i+T-1) of radius 1 per launch
// (heat_tb.cu), on tiles of 128 x 32 cells (narrow = 0) or 64 x 64 cells
// (narrow = 1).  The tensor map must have the box heat_tb_box_w(narrow) x
// heat_tb_box_h(narrow).
int heat_tb_box_w(int narrow);
int heat_tb_box_h(int narrow);
cudaError_t launch_heat_substep_tb(int T, int narrow, const CUtensorMap* tin, float* out, const BlockLayout& L,
                                   int step_i, const HeatCoef& c, int* status, cudaStream_t st, int zchunk);

// The tiles of a launch over the union of the blocks' windows; kept by the
// caller for the same layout and sub-step (rows = 0: not made yet), since the
// search goes through every block and z chunk.
struct HeatTiles {
    int rows = 0;                   // computed rows of a tile
    int ntx, nty, nzc, Lz;
    int x0, y0, z0;                 // storage x, row and plane of the windows' first cells
};

// T = 2, 3 or 4 sub-steps (step_i .. step_i+T-1) of radius 1 per launch, four
// rows per thread (heat_rows.cu).  The tensor map must have the box
// heat_rows_box_w() x heat_rows_box_h(T).
int heat_rows_box_w();
int heat_rows_box_h(int T);
cudaError_t launch_heat_rows(int T, const CUtensorMap* tin, float* out, const BlockLayout& L, int step_i,
                             const HeatCoef& c, int* status, cudaStream_t st, HeatTiles& tiles);

// One sub-step of radius D = 1 .. 4 (heat_far.cu).  tin: three tensor maps
// over the input, with boxes of heat_far_box_w() x heat_far_box_h(D, k) cells.
int heat_far_box_w();
int heat_far_box_h(int D, int k);
cudaError_t launch_heat_far(const CUtensorMap* tin, float* out, const BlockLayout& L, int D, int step_i,
                            const HeatCoef& c, int* status, cudaStream_t st, HeatTiles& tiles);

}  // namespace b2r
