// heat2.cu -- two heat time steps per HBM pass (temporal blocking), radius 1:
// the launch of heat2_unit.cuh's units over every tile of every block.
#include <algorithm>

#include "heat2_unit.cuh"

namespace b2r {
namespace {

using namespace h2k;

constexpr int kS2 = 4;                // input ring slots
constexpr size_t kSmem2 = size_t(kS2) * kPlane * 4 + 2 * size_t(kP1) * 4 + kS2 * 8 + 16 + 128;

__device__ __forceinline__ void pdl_wait2() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger2() { asm volatile("griddepcontrol.launch_dependents;"); }

struct H2Sched {
    int ntx, nty, NZ, Lz, nzc;
    long long U;
};

template <bool ROW>
__global__ void __launch_bounds__(kT2, 2)
heat2_kernel(const __grid_constant__ CUtensorMap tin, float* __restrict__ out, const BlockLayout L,
             const int step_i, const HeatCoef C, const H2Sched sch, int* __restrict__ status)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    H2Ctx c;
    float* ring = reinterpret_cast<float*>(smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127));
    c.ring = ring;
    c.s1 = ring + kS2 * kPlane;                          // 2 stage-1 planes
    c.bar = reinterpret_cast<uint64_t*>(c.s1 + 2 * kP1);
    c.tid = threadIdx.x;
    c.lane = c.tid & 31;
    c.warp = c.tid >> 5;
    c.tmap = &tin;
    c.C = C;
    c.plane = L.plane;
    c.P = L.P;
    if (c.tid == 0) {
        for (int s = 0; s < kS2; ++s) mbar_init(&c.bar[s], 1);
        fence_mbar_init();
    }
    __syncthreads();
    pdl_wait2();
    pdl_trigger2();

    c.gp = 0;
    c.issued_hi = 0;
    c.stop = 0;
    c.aborted = false;
    for (long long u = blockIdx.x; u < sch.U && !c.aborted; u += gridDim.x) {
        const int tx = (int)(u % sch.ntx);
        long long r = u / sch.ntx;
        const int ty = (int)(r % sch.nty);
        r /= sch.nty;
        const int zc = (int)(r % sch.nzc);
        const int blk = (int)(r / sch.nzc);
        if (!h2_unit<kS2, kPlane, ROW>(c, &tin, out, L, step_i, blk, tx, ty, zc * sch.Lz, sch.Lz, false)) break;
    }
    if (c.aborted && c.tid == 0) {
        report(status, DEV_TIMEOUT);
        for (unsigned g = c.stop; g < c.issued_hi; ++g)
            mbar_wait_bounded(&c.bar[g % kS2], (g / kS2) & 1, 100000000ull);
    }
}

bool h2_whole_rows(const BlockLayout& L)
{
    return L.nb[0] == 1 && !L.periodic && L.fixed_edge < 0 && L.B[0] > kOutW && L.B[0] <= kBoxW;
}

// The launch's tiles, and output planes per unit.  A CTA takes about 1 us to
// start and 0.52 us per plane (whole rows 0.61), of which it reads four beyond
// its chunk; two on an SM 0.71 us per plane of both (0.8).  The chunk with the
// least busy busiest SM, at most 32 planes: us per step at 48x40x32 1.86 in
// chunks of 1, 2.63 of 4; 64^3 2.32 of 3, 2.57 of 4, 2.45 of 2; 94x200x300 7.9
// of 16, 9.4 of 8.  The 0.52 us are neither the ring's depth (eight slots
// instead of four: the same) nor too few warps (16 of one row each: the same
// alone, slower two on an SM) nor the refill (a producer warp: 0.59).
struct H2Plan {
    int ntx, nty, Lz;
    double us;
};
H2Plan h2_plan(const BlockLayout& L)
{
    const bool row = h2_whole_rows(L);
    const int NZ = L.n[2] - 2, sms = 152;
    H2Plan p{row ? 1 : h2_ntx(L), h2_nty(L), 1, 1e300};
    const long long tiles = (long long)p.ntx * p.nty * L.nblk;
    for (int lz = 1; lz <= 32 && lz <= NZ; ++lz) {
        const long long q = (tiles * ((NZ + lz - 1) / lz) + sms - 1) / sms;
        const double us = (q / 2) * (1.0 + (row ? 0.80 : 0.71) * (lz + 4)) + (q % 2) * (0.9 + (row ? 0.61 : 0.52) * (lz + 4));
        if (us < p.us) {
            p.us = us;
            p.Lz = lz;
        }
    }
    return p;
}

}  // namespace

int heat2_box_w() { return kBoxW; }
int heat2_box_h() { return kBoxH; }
double heat2_us(const BlockLayout& L) { return h2_plan(L).us; }

cudaError_t launch_heat_substep2(const CUtensorMap* tin, float* out, const BlockLayout& L, int step_i,
                                 const HeatCoef& c, int* status, cudaStream_t st, int zchunk)
{
    static KernelSetup setup[2];
    const bool row = h2_whole_rows(L);
    if (cudaError_t e = kernel_setup(setup[row], row ? heat2_kernel<true> : heat2_kernel<false>, kT2, kSmem2, nullptr, nullptr)) return e;
    H2Sched sch;
    const H2Plan plan = h2_plan(L);
    sch.ntx = plan.ntx;
    sch.nty = plan.nty;
    sch.NZ = L.n[2] - 2;
    sch.Lz = std::min(zchunk > 0 ? zchunk : plan.Lz, sch.NZ);
    sch.nzc = (sch.NZ + sch.Lz - 1) / sch.Lz;
    sch.U = (long long)sch.ntx * sch.nty * L.nblk * sch.nzc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sch.U < 1 ? 1 : sch.U));
    cfg.blockDim = dim3(kT2);
    cfg.dynamicSmemBytes = kSmem2;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, row ? heat2_kernel<true> : heat2_kernel<false>, *tin, out, L, step_i, c, sch, status);
    count_launches(1);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace b2r
