// eqwp_ref_tma.cu -- the two stages of the collocated elastic-wave model
// (eqwp.cu) on large blocks, with every input streamed through TMA rings.
//
// The plain stages wait on their own loads: 24 to 28 of 16 bytes per thread and
// plane, the five rows of each neighbourhood read again from L1 and L2, 14 warps
// per SM (long scoreboard 7 of 9 cycles per issue, DRAM at 0.77 of the copy
// rate; 512x256x512 1474 us per step, 45.5 GLUPS).  Here a producer warp issues a tile's boxes ahead into shared memory
// and eight consumer warps compute from there:
//   ring V: the three fields whose z neighbours count (stress stage vx, vy, vz;
//     velocity stage sxz, syz, szz), boxes of the tile and 4 more cells on each
//     side in x, 2 more rows in y, 5 planes: the plane being updated, the two
//     after it (the last feeds the 5-plane z queues in registers), two ahead;
//   ring B, 3 planes: the fields read at the plane alone with x and y neighbours
//     (velocity stage sxx, sxy, syy; the same boxes) and those being updated
//     (the tile itself).
// Planes are handed over by two mbarriers per slot (loaded; read by every
// consumer warp), so no warp waits for another one's arithmetic.  Tile shape and
// arithmetic are the plain stages': the same bits.  512x256x512 1256 us per step,
// 53.4 GLUPS: DRAM at 0.91 of the copy rate.
#include <algorithm>

#include "b2r_common.cuh"
#include "eqwp.h"
#include "eqwp_tile.cuh"

namespace b2r {

namespace {

using namespace eqk;

constexpr int kCW = 8;                           // consumer warps
constexpr int kThr = 32 * (kCW + 1);
constexpr int kHF = 1632;                        // floats per slot of a box with neighbours: the largest, 136 x 12
constexpr int kOF = 1024;                        // floats per slot of the tile itself
constexpr int kSV = 5, kSB = 3;                  // ring slots

template <bool VEL>
struct Cfg {
    static constexpr int NH = VEL ? 3 : 0, NO = VEL ? 4 : 6;
    static constexpr int BF = NH * kHF + NO * kOF;       // floats per slot of ring B
    static constexpr size_t SMEM = ((size_t)kSV * 3 * kHF + (size_t)kSB * BF) * 4 + 2 * (kSV + kSB) * 8 + 128;
};

struct RefArgs {
    float* out[6];          // the fields updated, in the order of ring B
    EqwpRefParams p;
    int ts;
    int tx, ty;             // threads per row, rows
    int* status;
};

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ Row12 lrow(const float* p)
{
    const float4 a = lds4(p - 4), b = lds4(p), c = lds4(p + 4);
    return Row12{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w}};
}

// The plain stages' differences (dcx, dc4) and increments, explicitly rounded,
// with the products fused as the compiler fuses them there (found by comparing
// with every way to fuse them), so that both give the same bits.  Written so in
// the plain stages they take 468 us per step at 256^3 instead of 410.
__device__ __forceinline__ float ref_dx(const Row12& r, int j, float a, float b)
{
    return __fmaf_rn(a, __fsub_rn(r.v[6 + j], r.v[2 + j]), __fmul_rn(b, __fsub_rn(r.v[5 + j], r.v[3 + j])));
}
__device__ __forceinline__ float ref_dy(const float4& m2, const float4& m1, const float4& p1,
                                     const float4& p2, int j, float a, float b)
{
    return __fmaf_rn(b, __fsub_rn(cmp(p1, j), cmp(m1, j)), __fmul_rn(a, __fsub_rn(cmp(p2, j), cmp(m2, j))));
}
__device__ __forceinline__ float ref_dz(const Q5v& q, int j, float a, float b)
{
    return __fmaf_rn(a, __fsub_rn(cmp(q.p2, j), cmp(q.m2, j)), __fmul_rn(b, __fsub_rn(cmp(q.p1, j), cmp(q.m1, j))));
}
// d[f]: increments of sxx, syy, szz, sxy, sxz, syz from the derivatives of vx,
// vy, vz (eqwp.cu:460-473, dt folded into the Lame constants)
__device__ __forceinline__ void ref_stress(const float (&dx)[3], const float (&dy)[3], const float (&dz)[3],
                                           const EqwpRefParams& p, float (&d)[6][4], int j)
{
    d[0][j] = __fmaf_rn(p.l2m_dt, dx[0], __fmul_rn(p.l_dt, __fadd_rn(dy[1], dz[2])));
    d[1][j] = __fmaf_rn(p.l2m_dt, dy[1], __fmul_rn(p.l_dt, __fadd_rn(dx[0], dz[2])));
    d[2][j] = __fmaf_rn(p.l_dt, __fadd_rn(dx[0], dy[1]), __fmul_rn(p.l2m_dt, dz[2]));
    d[3][j] = __fmul_rn(p.mu_dt, __fadd_rn(dy[0], dx[1]));
    d[4][j] = __fmul_rn(p.mu_dt, __fadd_rn(dz[0], dx[2]));
    d[5][j] = __fmul_rn(p.mu_dt, __fadd_rn(dz[1], dy[2]));
}
// d[f]: increments of vx, vy, vz, disp from the divergence of the stresses, the
// body force already in its y component
__device__ __forceinline__ void ref_velocity(float sx, float sy, float sz, const EqwpRefParams& p, float (&d)[4][4],
                                             int j)
{
    d[0][j] = __fmul_rn(p.dt_rho, sx);
    d[1][j] = __fmul_rn(p.dt_rho, sy);
    d[2][j] = __fmul_rn(p.dt_rho, sz);
    d[3][j] = __fmul_rn(p.dt2_rho, sy);
}

template <bool VEL>
__global__ void __launch_bounds__(kThr, 1)
eqwp_ref_tma_kernel(const __grid_constant__ EqwpRefMaps maps, const RefArgs A, const BlockLayout L, const int step_i,
                    const Tiles T)
{
    using C = Cfg<VEL>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* const rv = reinterpret_cast<float*>(smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127));
    float* const rb = rv + kSV * 3 * kHF;
    uint64_t* const fullv = reinterpret_cast<uint64_t*>(rb + kSB * C::BF);
    uint64_t* const emptyv = fullv + kSV;
    uint64_t* const fullb = emptyv + kSV;
    uint64_t* const emptyb = fullb + kSB;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (tid == 0) {
        for (int s = 0; s < kSV; ++s) mbar_init(&fullv[s], 1), mbar_init(&emptyv[s], kCW);
        for (int s = 0; s < kSB; ++s) mbar_init(&fullb[s], 1), mbar_init(&emptyb[s], kCW);
        fence_mbar_init();
    }
    __syncthreads();
    pdl_begin();

    const int blk = blockIdx.z / T.nzc, zc = blockIdx.z % T.nzc;
    const Win w = window(L, blk, zc, T.nzc, 4 * step_i + (VEL ? 4 : 2));
    const int HW = 4 * A.tx + 8, OW = 4 * A.tx;
    const int X0 = T.x0 + blockIdx.x * OW, Y0 = T.y0 + blockIdx.y * A.ty;
    // uniform per CTA: nothing of this tile lies in the window
    if (!w.ok || X0 - L.xoff > w.hi[0] || X0 - L.xoff + OW - 1 < w.lo[0] || Y0 > w.hi[1] || Y0 + A.ty - 1 < w.lo[1])
        return;
    const int zs = w.zs, nv = w.ze - zs + 5, no = w.ze - zs + 1;   // planes of V from zs-2 on, of B from zs on
    if (warp == kCW) {
        // ------------------------------------------------------------ producer
        if ((tid & 31) == 0) {
            const uint32_t hb = (uint32_t)(HW * (A.ty + 4)) * 4u, ob = (uint32_t)(OW * A.ty) * 4u;
            bool ok = true;
            int k = 0;
            for (; k < nv && ok; ++k) {
                const int sv = k % kSV;
                if (k >= kSV) ok = mbar_wait_bounded(&emptyv[sv], ((k - kSV) / kSV) & 1);
                if (!ok) break;
                mbar_expect_tx(&fullv[sv], 3 * hb);
                for (int f = 0; f < 3; ++f)
                    tma_load_4d(rv + (sv * 3 + f) * kHF, &maps.v[f], X0 - 4, Y0 - 2, zs - 2 + k, blk, &fullv[sv]);
                const int j = k - 4;
                if (j < 0) continue;
                const int sb = j % kSB;
                if (j >= kSB) ok = mbar_wait_bounded(&emptyb[sb], ((j - kSB) / kSB) & 1);
                if (!ok) break;
                mbar_expect_tx(&fullb[sb], C::NH * hb + C::NO * ob);
                float* d = rb + sb * C::BF;
                for (int f = 0; f < C::NH; ++f)
                    tma_load_4d(d + f * kHF, &maps.h[f], X0 - 4, Y0 - 2, zs + j, blk, &fullb[sb]);
                for (int f = 0; f < C::NO; ++f)
                    tma_load_4d(d + C::NH * kHF + f * kOF, &maps.o[f], X0, Y0, zs + j, blk, &fullb[sb]);
            }
            if (!ok) report(A.status, DEV_TIMEOUT);
            // the loads land before the CTA leaves (bounded): the last ones issued of
            // either ring; when all went well the consumers wait for them as well
            const int kv = ok ? nv : k + 1;
            for (int t = max(0, kv - kSV); t < min(kv, nv); ++t) mbar_wait_bounded(&fullv[t % kSV], (t / kSV) & 1, 100000000ull);
            const int kb = ok ? no : max(0, k - 4);
            for (int t = max(0, kb - kSB); t < min(kb, no); ++t) mbar_wait_bounded(&fullb[t % kSB], (t / kSB) & 1, 100000000ull);
        }
        return;
    }
    // ------------------------------------------------------------ consumers
    const int tx = tid % A.tx, ty0 = tid / A.tx;
    const bool inrow = ty0 < A.ty;               // the threads beyond tx * ty only keep step
    const int ty = inrow ? ty0 : A.ty - 1;
    Cell c;
    const bool act =
        cell_setup(L, w, blk, c, T.x0, T.y0, TilePos{(int)blockIdx.x, (int)blockIdx.y, tx, ty, A.tx, A.ty}) && inrow;
    const int at = (ty + 2) * HW + 4 + 4 * tx;   // the thread's first cell in a box with neighbours
    auto wait = [&](uint64_t* full, int t, int slots) { return mbar_wait_bounded(&full[t % slots], (t / slots) & 1); };
    auto done = [&](uint64_t* empty, int t, int slots) {
        __syncwarp();
        if ((tid & 31) == 0) arrive(&empty[t % slots]);
    };
    auto vp = [&](int t, int f) { return rv + (t % kSV * 3 + f) * kHF + at; };
    bool ok = true;
    Q5v q[3];
    for (int t = 0; t < 4 && t < nv; ++t) ok = ok && wait(fullv, t, kSV);
    if (ok) {
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            q[f].m1 = lds4(vp(0, f));
            q[f].c = lds4(vp(1, f));
            q[f].p1 = lds4(vp(2, f));
            q[f].p2 = lds4(vp(3, f));
        }
    }
    const EqwpRefParams& p = A.p;
    const float a = p.ca, b = p.cb;
    // body force (velocity stage): the thread's cells of the patch
    unsigned fx = 0;
    if (VEL) {
        const bool frow = (c.y - L.H) % p.every[1] == p.fy && A.ts < p.fsteps;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int x = (c.xb + j - L.H) % p.every[0];
            if (frow && x >= p.fx0 && x < p.fx1) fx |= 1u << j;
        }
    }
    for (int z = zs; z <= w.ze && ok; ++z) {
        const int tv = z - zs + 2, to = z - zs;
        if (!wait(fullv, tv + 2, kSV) || !wait(fullb, to, kSB)) {
            ok = false;
            break;
        }
#pragma unroll
        for (int f = 0; f < 3; ++f) q[f].shift(lds4(vp(tv + 2, f)));
        const float* const hb = rb + to % kSB * C::BF;
        const float* const ob = hb + C::NH * kHF + ty * OW + 4 * tx;
        float4 old[C::NO];
#pragma unroll
        for (int f = 0; f < C::NO; ++f) old[f] = lds4(ob + f * kOF);
        const long long o = (long long)z * L.plane + c.base;
        float d[C::NO][4];
        if constexpr (!VEL) {
            const float *vx = vp(tv, 0), *vy = vp(tv, 1), *vz = vp(tv, 2);
            const Row12 rx = lrow(vx), ry = lrow(vy), rz = lrow(vz);
            const float4 xm2 = lds4(vx - 2 * HW), xm1 = lds4(vx - HW), xp1 = lds4(vx + HW), xp2 = lds4(vx + 2 * HW);
            const float4 ym2 = lds4(vy - 2 * HW), ym1 = lds4(vy - HW), yp1 = lds4(vy + HW), yp2 = lds4(vy + 2 * HW);
            const float4 zm2 = lds4(vz - 2 * HW), zm1 = lds4(vz - HW), zp1 = lds4(vz + HW), zp2 = lds4(vz + 2 * HW);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float dx[3] = {ref_dx(rx, j, a, b), ref_dx(ry, j, a, b), ref_dx(rz, j, a, b)};
                const float dy[3] = {ref_dy(xm2, xm1, xp1, xp2, j, a, b), ref_dy(ym2, ym1, yp1, yp2, j, a, b),
                                     ref_dy(zm2, zm1, zp1, zp2, j, a, b)};
                const float dz[3] = {ref_dz(q[0], j, a, b), ref_dz(q[1], j, a, b), ref_dz(q[2], j, a, b)};
                ref_stress(dx, dy, dz, p, d, j);
            }
        } else {
            const float *xx = hb + at, *xy = xx + kHF, *yy = xy + kHF, *xz = vp(tv, 0), *yz = vp(tv, 1);
            const Row12 rxx = lrow(xx), rxy = lrow(xy), rxz = lrow(xz);
            const float4 xym2 = lds4(xy - 2 * HW), xym1 = lds4(xy - HW), xyp1 = lds4(xy + HW), xyp2 = lds4(xy + 2 * HW);
            const float4 yym2 = lds4(yy - 2 * HW), yym1 = lds4(yy - HW), yyp1 = lds4(yy + HW), yyp2 = lds4(yy + 2 * HW);
            const float4 yzm2 = lds4(yz - 2 * HW), yzm1 = lds4(yz - HW), yzp1 = lds4(yz + HW), yzp2 = lds4(yz + 2 * HW);
            unsigned force = 0;
            if (fx) {
                const int zl = (z - L.H) % p.every[2];
                if (zl >= p.fz0 && zl < p.fz1) force = fx;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float sx = add3(ref_dx(rxx, j, a, b), ref_dy(xym2, xym1, xyp1, xyp2, j, a, b), ref_dz(q[0], j, a, b));
                float sy = add3(ref_dx(rxy, j, a, b), ref_dy(yym2, yym1, yyp1, yyp2, j, a, b), ref_dz(q[1], j, a, b));
                const float sz = add3(ref_dx(rxz, j, a, b), ref_dy(yzm2, yzm1, yzp1, yzp2, j, a, b), ref_dz(q[2], j, a, b));
                if (force & (1u << j)) sy = __fadd_rn(sy, p.fval);
                ref_velocity(sx, sy, sz, p, d, j);
            }
        }
        if (act) {
#pragma unroll
            for (int f = 0; f < C::NO; ++f) wr4(A.out[f] + o, c, old[f], d[f]);
        }
        // the slots read are given back after the stores: a load that has only been
        // issued may still be under way when the barrier counts the arrival, and the
        // refill then overtakes it; a stored result has been loaded
        if (z == zs) {
            done(emptyv, 0, kSV);
            done(emptyv, 1, kSV);
        }
        done(emptyv, tv, kSV);
        done(emptyb, to, kSB);
    }
    if (!ok) report(A.status, DEV_TIMEOUT);
}

template <bool VEL>
cudaError_t launch_stage(const EqwpRefMaps& maps, RefArgs A, const BlockLayout& L, int step_i, cudaStream_t st)
{
    static KernelSetup setup;
    int sms = 152;      // one CTA per SM
    if (cudaError_t e = kernel_setup(setup, eqwp_ref_tma_kernel<VEL>, kThr, Cfg<VEL>::SMEM, nullptr, &sms)) return e;
    const int shrink = 4 * step_i + (VEL ? 4 : 2);
    Grid g = stage_grid(L, shrink);
    A.tx = (int)g.b.x;
    A.ty = (int)g.b.y;
    if ((4 * A.tx + 8) * (A.ty + 4) > kHF || 4 * A.tx * A.ty > kOF) return cudaErrorInvalidValue;
    const long long tiles = (long long)g.g.x * g.g.y * L.nblk;
    int nz = 1;
    for (int k = 0; k < L.nblk; ++k) {
        int lo, hi;
        stage_region(L, edge_bits(L, k), 2, shrink, lo, hi);
        nz = std::max(nz, hi - lo + 1);
    }
    // z chunks: the fewest planes on the busiest SM, four of them to start a chunk
    double least = 1e300;
    for (int k = 1; k <= std::max(1, std::min(nz / 8, 65535 / L.nblk)); ++k) {
        const double cost = (double)((tiles * k + sms - 1) / sms) * ((nz + k - 1) / k + 4);
        if (cost < least - 1e-9) {
            least = cost;
            g.t.nzc = k;
        }
    }
    return launch_pdl(eqwp_ref_tma_kernel<VEL>, dim3(g.g.x, g.g.y, L.nblk * g.t.nzc), dim3(kThr), Cfg<VEL>::SMEM, st, maps,
                      A, L, step_i, g.t);
}

}  // namespace

void eqwp_ref_tma_shape(const BlockLayout& L, int step_i, bool velocity, int* tx, int* ty)
{
    const Grid g = stage_grid(L, 4 * step_i + (velocity ? 4 : 2));
    *tx = (int)g.b.x;
    *ty = (int)g.b.y;
}

cudaError_t launch_eqwp_ref_tma(const EqwpRefMaps& maps, bool velocity, float* const* fld, const BlockLayout& L,
                                int step_i, int ts, const EqwpRefParams& p, int* status, cudaStream_t st)
{
    RefArgs A{};
    A.p = p;
    A.ts = ts;
    A.status = status;
    static constexpr int kStress[6] = {SXX, SYY, SZZ, SXY, SXZ, SYZ}, kVelocity[4] = {VX, VY, VZ, DISP};
    if (velocity) {
        for (int f = 0; f < 4; ++f) A.out[f] = fld[kVelocity[f]];
        return launch_stage<true>(maps, A, L, step_i, st);
    }
    for (int f = 0; f < 6; ++f) A.out[f] = fld[kStress[f]];
    return launch_stage<false>(maps, A, L, step_i, st);
}

}  // namespace b2r
