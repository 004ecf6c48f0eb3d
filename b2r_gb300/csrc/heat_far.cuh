// heat_far.cuh -- the consumer side of the heat step with a producer warp: one
// unit (a tile over a chunk of output planes) of radius 1..4.  Used by the
// one-step launch (heat_far.cu, one unit per CTA) and the batched persistent
// kernel (batch.cu, units from a work queue).
//
// The input planes of a unit arrive in order in a ring of S shared slots, each
// with two mbarriers: `full` (the plane is loaded) and `empty` (every consumer
// warp has read it).  A thread holds four x cells (float4) of two rows and the
// 2D+1 planes around the output plane in registers, the plane loop unrolled by
// them so that the queue turns by names; x and y neighbours come from the
// centre plane in the ring, the rows of the pair's y neighbours read pair by
// pair as the radius grows, each once for both rows.  Operations and their
// order are the sweep's (heat_unit.cuh): the same bits.
#pragma once
#include "b2r_common.cuh"
#include "heat.h"

namespace b2r {
namespace farx {

__device__ __forceinline__ float4 f4(const float* p) { return *reinterpret_cast<const float4*>(p); }

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The weights as the packed operations take them, both lanes the same: of a
// kernel parameter, which the operations read from the constant bank, or
// from pairs in shared memory, where a kernel whose weights change from unit
// to unit keeps them -- read at each use (the volatile loads), since 1 + 3D
// pairs held in registers would spill the queue.  Order: a0, then x, y, z of
// each distance.
struct ParamCoef {
    const HeatCoef& C;
    __device__ __forceinline__ float2 a0() const { return make_float2(C.a0, C.a0); }
    __device__ __forceinline__ float2 x(int k) const { return make_float2(C.ax[k - 1], C.ax[k - 1]); }
    __device__ __forceinline__ float2 y(int k) const { return make_float2(C.ay[k - 1], C.ay[k - 1]); }
    __device__ __forceinline__ float2 z(int k) const { return make_float2(C.az[k - 1], C.az[k - 1]); }
};
constexpr int kCoefPairs = 13;
struct SharedCoef {
    uint32_t at;          // shared address of the pairs
    __device__ __forceinline__ float2 ld(int i) const
    {
        float2 v;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at + 8u * (uint32_t)i));
        return v;
    }
    __device__ __forceinline__ float2 a0() const { return ld(0); }
    __device__ __forceinline__ float2 x(int k) const { return ld(3 * k - 2); }
    __device__ __forceinline__ float2 y(int k) const { return ld(3 * k - 1); }
    __device__ __forceinline__ float2 z(int k) const { return ld(3 * k); }
};

// A consumer thread's state in a unit.  S ring slots of SLOT floats; the row
// pitch of a plane is BWC, or bw where that is 0.
template <int D, int S, int SLOT, int BWC>
struct FCtx {
    float4 q[2 * D + 1][2];     // planes p-2D .. p by slot (pr mod 2D+1), rows
    const float* ring;          // + the thread's first cell of its first row
    uint64_t *full, *empty;
    float* dst;                 // the thread's cells of the next output plane
    long long plane;
    int P, np, bw;
    unsigned m0, m1;            // cells stored of each row
    bool lane0;
};

// Input plane pr (slot PH = pr mod 2D+1 of the queue); from pr = 2D on also
// the output plane D planes back.  False if the wait gave up.
template <int D, int S, int SLOT, int BWC, int PH, class Coef>
__device__ __forceinline__ bool f_iter(FCtx<D, S, SLOT, BWC>& c, const Coef& C, int pr, int slot, int phase, int cslot)
{
    constexpr int N = 2 * D + 1;
    const int BW = BWC > 0 ? BWC : c.bw;
    if (!mbar_wait_bounded(&c.full[slot], phase)) return false;
    {
        const float* pl = c.ring + slot * SLOT;
        c.q[PH][0] = f4(pl);
        c.q[PH][1] = f4(pl + BW);
    }
    if (pr >= 2 * D) {
        constexpr int CE = (PH + N - D) % N;                // the centre plane
        const float* pc = c.ring + cslot * SLOT;
        const float4 c0 = c.q[CE][0], c1 = c.q[CE][1];
        const float4 l0 = f4(pc - 4), r0 = f4(pc + 4), l1 = f4(pc + BW - 4), r1 = f4(pc + BW + 4);
        const float v0[12] = {l0.x, l0.y, l0.z, l0.w, c0.x, c0.y, c0.z, c0.w, r0.x, r0.y, r0.z, r0.w};
        const float v1[12] = {l1.x, l1.y, l1.z, l1.w, c1.x, c1.y, c1.z, c1.w, r1.x, r1.y, r1.z, r1.w};
        const float2 a0 = C.a0();
        float2 lo0 = __fmul2_rn(a0, make_float2(c0.x, c0.y)), hi0 = __fmul2_rn(a0, make_float2(c0.z, c0.w));
        float2 lo1 = __fmul2_rn(a0, make_float2(c1.x, c1.y)), hi1 = __fmul2_rn(a0, make_float2(c1.z, c1.w));
        float4 below = c0, above = c1;                      // rows -(k-1) and k of the pair
#pragma unroll
        for (int k = 1; k <= D; ++k) {
            const float4 yb = f4(pc - k * BW), ya = f4(pc + (k + 1) * BW);   // rows -k and k+1
            const float4 zm0 = c.q[(CE + N - k) % N][0], zp0 = c.q[(CE + k) % N][0];
            const float4 zm1 = c.q[(CE + N - k) % N][1], zp1 = c.q[(CE + k) % N][1];
            const float2 cx = C.x(k), cy = C.y(k), cz = C.z(k);
            lo0 = __ffma2_rn(cx, make_float2(v0[4 - k] + v0[4 + k], v0[5 - k] + v0[5 + k]), lo0);
            hi0 = __ffma2_rn(cx, make_float2(v0[6 - k] + v0[6 + k], v0[7 - k] + v0[7 + k]), hi0);
            lo1 = __ffma2_rn(cx, make_float2(v1[4 - k] + v1[4 + k], v1[5 - k] + v1[5 + k]), lo1);
            hi1 = __ffma2_rn(cx, make_float2(v1[6 - k] + v1[6 + k], v1[7 - k] + v1[7 + k]), hi1);
            // row 0: rows -k and k; row 1: rows 1-k and 1+k
            lo0 = __ffma2_rn(cy, __fadd2_rn(make_float2(yb.x, yb.y), make_float2(above.x, above.y)), lo0);
            hi0 = __ffma2_rn(cy, __fadd2_rn(make_float2(yb.z, yb.w), make_float2(above.z, above.w)), hi0);
            lo1 = __ffma2_rn(cy, __fadd2_rn(make_float2(below.x, below.y), make_float2(ya.x, ya.y)), lo1);
            hi1 = __ffma2_rn(cy, __fadd2_rn(make_float2(below.z, below.w), make_float2(ya.z, ya.w)), hi1);
            lo0 = __ffma2_rn(cz, __fadd2_rn(make_float2(zm0.x, zm0.y), make_float2(zp0.x, zp0.y)), lo0);
            hi0 = __ffma2_rn(cz, __fadd2_rn(make_float2(zm0.z, zm0.w), make_float2(zp0.z, zp0.w)), hi0);
            lo1 = __ffma2_rn(cz, __fadd2_rn(make_float2(zm1.x, zm1.y), make_float2(zp1.x, zp1.y)), lo1);
            hi1 = __ffma2_rn(cz, __fadd2_rn(make_float2(zm1.z, zm1.w), make_float2(zp1.z, zp1.w)), hi1);
            below = yb;
            above = ya;
        }
        const float4 o0 = make_float4(lo0.x, lo0.y, hi0.x, hi0.y), o1 = make_float4(lo1.x, lo1.y, hi1.x, hi1.y);
        float* d = c.dst;
        if (c.m0 == 15u) *reinterpret_cast<float4*>(d) = o0;
        else if (c.m0) {
            if (c.m0 & 1u) d[0] = o0.x;
            if (c.m0 & 2u) d[1] = o0.y;
            if (c.m0 & 4u) d[2] = o0.z;
            if (c.m0 & 8u) d[3] = o0.w;
        }
        d += c.P;
        if (c.m1 == 15u) *reinterpret_cast<float4*>(d) = o1;
        else if (c.m1) {
            if (c.m1 & 1u) d[0] = o1.x;
            if (c.m1 & 2u) d[1] = o1.y;
            if (c.m1 & 4u) d[2] = o1.z;
            if (c.m1 & 8u) d[3] = o1.w;
        }
        c.dst += c.plane;
    }
    if (pr >= D) {
        // plane pr - D is read: its slot may be refilled.  What the stores above were
        // made of has been loaded; while nothing is stored yet, a load that has only
        // been issued could still be under way when the barrier counts the arrival.
        if (pr < 2 * D) __threadfence_block();
        __syncwarp();
        if (c.lane0) mbar_arrive(&c.empty[cslot]);
    }
    return true;
}

template <int D, int S, int SLOT, int BWC, int PH, class Coef>
__device__ __forceinline__ bool f_round(FCtx<D, S, SLOT, BWC>& c, const Coef& C, int& pr, int& slot, int& phase,
                                        int& cslot)
{
    if (pr >= c.np) return true;
    if (!f_iter<D, S, SLOT, BWC, PH>(c, C, pr, slot, phase, cslot)) return false;
    if (pr >= D && ++cslot == S) cslot = 0;
    ++pr;
    if (++slot == S) slot = 0, phase ^= 1;
    if constexpr (PH + 1 < 2 * D + 1) return f_round<D, S, SLOT, BWC, PH + 1>(c, C, pr, slot, phase, cslot);
    return true;
}

// Every plane of a unit; slot, phase and cslot are the ring positions of the
// next plane to come and of the next to release, carried from unit to unit.
// The unit's last D planes are released at its end.  False if a wait gave up.
template <int D, int S, int SLOT, int BWC, class Coef>
__device__ __forceinline__ bool f_unit(FCtx<D, S, SLOT, BWC>& c, const Coef& C, int& slot, int& phase, int& cslot)
{
    for (int pr = 0; pr < c.np;)
        if (!f_round<D, S, SLOT, BWC, 0>(c, C, pr, slot, phase, cslot)) return false;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        if (c.lane0) mbar_arrive(&c.empty[cslot]);
        if (++cslot == S) cslot = 0;
    }
    return true;
}

}  // namespace farx
}  // namespace b2r
