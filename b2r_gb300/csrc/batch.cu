// batch.cu -- many independent heat instances of uneven sizes and stencil
// orders advanced in persistent launches (one per stencil order) driven by
// device work queues.
//
// No reference counterpart (the reference runs one model per MPI rank); each
// instance is a single-block heat domain with a fixed shell, stepped with the
// scheme of heat-3D.cu:228-231/315-318/410-413/514-517 exactly as the plain
// sweep does, so results are bit-identical to per-instance plain runs.
//
// Work items (round t, instance k, unit u) go through device work queues
// (work_queue.cuh).  A round is one time step of an instance on one-step
// units (heat_unit.cuh, tile shape per instance) or two of an instance on
// two-step units (heat2_unit.cuh, radius 1; the last round of an odd step
// count takes one), chosen per (order, size class) by the autotuner.
#include <algorithm>
#include <mutex>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include "batch_planes.h"
#include "heat2_unit.cuh"
#include "heat_far.cuh"
#include "heat_unit.cuh"
#include "work_queue.cuh"

namespace b2r {
namespace {

using heatk::kThreads;
// One ring for every stencil order: 5 slots (D = 4 needs D+1), each as large
// as the biggest plane.  D <= 2 tiles have 2 rows per warp, D >= 3 tiles one
// (their register queues are 2D+1 planes deep); 2 CTAs/SM without spills.
constexpr int kS = 5;
template <int D>
struct RowsPerWarp {
    static constexpr int value = D <= 2 ? 2 : 1;
};
constexpr int cmax(int a, int b) { return a > b ? a : b; }
// tile shapes: LPR lanes per row = 32, 16, 8 -> 128, 64, 32 cells wide
template <int D, int LPR>
using BCfg = heatk::Cfg<D, RowsPerWarp<D>::value, kS, 0, LPR>;
template <int LPR>
constexpr int slot_max()
{
    return cmax(cmax(BCfg<1, LPR>::SLOT, BCfg<2, LPR>::SLOT), cmax(BCfg<3, LPR>::SLOT, BCfg<4, LPR>::SLOT));
}
constexpr int kSlot = cmax(cmax(slot_max<32>(), slot_max<16>()), slot_max<8>());
static_assert(kSlot >= h2k::kPlane, "the two-step units stream through the same ring slots");
constexpr size_t kSmem = size_t(kS) * kSlot * sizeof(float) + kS * sizeof(uint64_t) + 16 + 128;
// the two-step units' two stage-1 planes, after the schedule tables
constexpr size_t kSmemS1 = 2 * size_t(h2k::kP1) * sizeof(float) + 128;
// tile shapes 0..2: one step per unit, LPR lanes per row = 32, 16, 8 -> 128,
// 64, 32 cells wide; shape 3: two steps per unit on 128 x 16-cell tiles
// (radius 1 only, heat2_unit.cuh)
constexpr int kShapes = 4;
constexpr int kTwoStep = 3;
constexpr int kLpr[kShapes] = {32, 16, 8, 32};
constexpr int kBoxH[5][3] = {{0, 0, 0},
                             {BCfg<1, 32>::BH, BCfg<1, 16>::BH, BCfg<1, 8>::BH},
                             {BCfg<2, 32>::BH, BCfg<2, 16>::BH, BCfg<2, 8>::BH},
                             {BCfg<3, 32>::BH, BCfg<3, 16>::BH, BCfg<3, 8>::BH},
                             {BCfg<4, 32>::BH, BCfg<4, 16>::BH, BCfg<4, 8>::BH}};
constexpr int kTileY[5][3] = {{0, 0, 0},
                              {BCfg<1, 32>::TY, BCfg<1, 16>::TY, BCfg<1, 8>::TY},
                              {BCfg<2, 32>::TY, BCfg<2, 16>::TY, BCfg<2, 8>::TY},
                              {BCfg<3, 32>::TY, BCfg<3, 16>::TY, BCfg<3, 8>::TY},
                              {BCfg<4, 32>::TY, BCfg<4, 16>::TY, BCfg<4, 8>::TY}};

struct InstDev {
    BlockLayout L;
    float* buf[2];
    HeatCoef C;
    int D, nsteps, ntx, nty, NZ, Lz, nzc, units;
    int shape;                           // tile shape: index into kLpr
    int lpr;                             // its lanes per tile row (kLpr[shape])
    int tb;                              // time steps per unit: 1, or 2 (shape kTwoStep)
    int rounds;                          // rounds of units: nsteps / tb, rounded up
    int done0;                           // its counters: one per z chunk, or one (two-step kernel)
};

struct BatchArgs {
    const InstDev* inst;                 // sorted by rounds, descending
    const CUtensorMap* maps;             // 2 per instance: buffer 0, buffer 1
    const unsigned long long* items;     // the queue: work items in claim order
    unsigned long long* head;            // next item (zeroed per run)
    unsigned* done;                      // finished units per instance and z chunk (zeroed per run)
    int* status;
    long long total;
};

// ---------------------------------------------------------------- one step per unit
// The default kernel (no instance on two-step units): CTAs of one producer
// warp and kQC consumer warps (heat_far.cuh), two per SM.  The producer claims
// items, waits for an item's instance to finish the round before, and streams
// the unit's planes into the ring while the consumers still work on the units
// before it, so neither the claim, nor the wait, nor filling the ring stops
// them.  A consumer warp reads the next unit's description (a ring of four,
// written before the unit's first plane is loaded; a unit has at least three
// planes and the ring of planes eight, so the producer is never four units
// ahead), runs it, and counts itself into the instance's counter.  An item
// still waits only for items claimed before it, whose CTAs' consumers need
// nothing but their ring, so the queue cannot deadlock.
//
// Measured, 64 instances of edges 32..192, radii 1..4, 50..500 steps: 49.2 ms
// with upload and download from 94.4 (478 GLUPS alone from 242; 50.6 ms with
// one counter per instance instead of one per z chunk; z chunks of 8, 12, 20,
// 32 planes instead of 16: 55, 50, 52, 59 ms).  All 64 with radius 1 / 2 / 3 /
// 4: 653 / 610 / 513 / 404 GLUPS.
//
// One launch and one queue per radius in the batch: with all radii in one
// kernel the four unrolled plane loops share one register allocation and
// spill (radius 2: 313 GLUPS alone in such a kernel).  The launches run on
// streams of their own, so one's CTAs take the room that another's tail
// leaves.
//
constexpr int kQC = 7, kQS = 8;
constexpr int kQThreads = 32 * (kQC + 1);
constexpr int kQTileY[3] = {2 * kQC, 4 * kQC, 8 * kQC};     // rows of a tile by shape
constexpr int q_slot(int D, int s) { return (4 * kLpr[s] + 8) * (kQTileY[s] + 2 * D); }
constexpr int kQSlot = (cmax(cmax(q_slot(4, 0), q_slot(4, 1)), q_slot(4, 2)) + 31) / 32 * 32;
constexpr size_t kQSmem = size_t(kQS) * kQSlot * sizeof(float) + 2 * kQS * sizeof(uint64_t) + 128;

__device__ __forceinline__ float* q_ring(unsigned char* smem_raw)   // TMA destinations are 128-byte aligned
{
    return reinterpret_cast<float*>(smem_raw + ((128 - (smem_u32(smem_raw) & 127)) & 127));
}

struct QUnit {
    int k, t, u;           // instance (-1: no more units), round, unit
};

// Ring positions after the unit (packed), or -1 if a wait gave up.  Not
// inlined: a register allocation of its own does not spill (radius 4).
template <int D>
__device__ __noinline__ int consume_unit(const InstDev& in, int t, int u, uint32_t coef, int pos)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* const ring = q_ring(smem_raw);    // found again here, so that its loads are known to be shared ones
    farx::FCtx<D, kQS, kQSlot, 0> c;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    uint64_t* const full = reinterpret_cast<uint64_t*>(ring + kQS * kQSlot);
    uint64_t* const empty = full + kQS;
    int slot = pos & 15, phase = (pos >> 4) & 1, cslot = pos >> 5;
    const int tx = u % in.ntx, r = u / in.ntx, ty = r % in.nty, zc = r / in.nty;
    const int lpr = in.lpr, lg = lpr == 32 ? 5 : (lpr == 16 ? 4 : 3);
    const int lx = lane & (lpr - 1);
    const int row = 2 * ((warp << (5 - lg)) + (lane >> lg));     // the thread's first row in the tile
    const BlockLayout& L = in.L;
    const int zs = D + zc * in.Lz, ze = min(D + (zc + 1) * in.Lz - 1, L.n[2] - 1 - D);
    const int xs = ((L.xoff + D) & ~3) + tx * 4 * lpr + 4 * lx, y = D + ty * (2 * kQC << (5 - lg)) + row;
    c.full = full;
    c.empty = empty;
    c.plane = L.plane;
    c.P = L.P;
    c.np = ze - zs + 1 + 2 * D;
    c.bw = 4 * lpr + 8;
    c.lane0 = lane == 0;
    c.ring = ring + (D + row) * c.bw + 4 + 4 * lx;
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        m |= (xs + j - L.xoff >= D && xs + j - L.xoff <= L.n[0] - 1 - D ? 1u : 0u) << j;
    c.m0 = y <= L.n[1] - 1 - D ? m : 0u;
    c.m1 = y + 1 <= L.n[1] - 1 - D ? m : 0u;
    c.dst = in.buf[(t + 1) & 1] + (long long)zs * L.plane + (long long)y * L.P + xs;
    return farx::f_unit(c, farx::SharedCoef{coef}, slot, phase, cslot) ? slot | (phase << 4) | (cslot << 5) : -1;
}

template <int D>
__global__ void __launch_bounds__(kQThreads, 2) batch_far_kernel(const BatchArgs a)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ QUnit s_unit[4];
    __shared__ float2 s_coef[4][farx::kCoefPairs];
    float* const ring = q_ring(smem_raw);
    uint64_t* const full = reinterpret_cast<uint64_t*>(ring + kQS * kQSlot);
    uint64_t* const empty = full + kQS;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kQS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kQC);
        }
        fence_mbar_init();
    }
    __syncthreads();
    if (warp == kQC) {                       // the producer
        int slot = 0, phase = 0;
        long long i = 0;                     // planes issued
        bool ok = true;
        long long next = lane == 0 ? (long long)atomicAdd(a.head, 1ull) : 0;
        for (int j = 0; ok; ++j) {
            QUnit q{-1, 0, 0};
            next = __shfl_sync(0xffffffffu, next, 0);
            if (next < a.total) wq::unpack_item(a.items[next], q.t, q.k, q.u);
            if (q.k < 0) {                   // no more units: a phase without a plane says so
                if (lane == 0) {
                    if (i >= kQS) ok = mbar_wait_bounded(&empty[slot], phase ^ 1);
                    if (ok) {
                        s_unit[j & 3] = q;
                        farx::mbar_arrive(&full[slot]);
                    }
                }
                break;
            }
            const InstDev& in = a.inst[q.k];
            const int bw = 4 * in.lpr + 8, th = 2 * kQC * (32 / in.lpr), tiles = in.ntx * in.nty;
            const int tx = q.u % in.ntx, r = q.u / in.ntx, ty = r % in.nty, zc = r / in.nty;
            if (lane == 0) next = (long long)atomicAdd(a.head, 1ull);
            if (q.t > 0) {
                // the round before of the chunks this one reads (and whose
                // readers it overwrites): a counter per lane
                const int reach = (D + in.Lz - 1) / in.Lz;
                for (int c = max(0, zc - reach) + lane; ok && c <= min(in.nzc - 1, zc + reach); c += 32)
                    ok = wq::wait_done(&a.done[in.done0 + c], (unsigned)q.t * (unsigned)tiles * (unsigned)kQC);
                ok = __all_sync(0xffffffffu, ok);
                __syncwarp();                // a vote orders no memory: what the other lanes acquired, before lane 0's loads
            }
            if (lane == 0) {
                const int zs = D + zc * in.Lz, ze = min(D + (zc + 1) * in.Lz - 1, in.L.n[2] - 1 - D);
                const int np = ze - zs + 1 + 2 * D, xs0 = ((in.L.xoff + D) & ~3) + tx * 4 * in.lpr;
                const unsigned bytes = (unsigned)(bw * (th + 2 * D)) * 4u;
                const CUtensorMap* map = &a.maps[2 * q.k + (q.t & 1)];
                asm volatile("fence.proxy.async.global;" ::: "memory");
                for (int p = 0; p < np && ok; ++p, ++i) {
                    if (i >= kQS) ok = mbar_wait_bounded(&empty[slot], phase ^ 1);
                    if (!ok) break;
                    if (p == 0) {            // the unit's description and weights, before its first plane
                        s_unit[j & 3] = q;
                        s_coef[j & 3][0] = make_float2(in.C.a0, in.C.a0);
#pragma unroll
                        for (int d = 0; d < 4; ++d) {
                            s_coef[j & 3][3 * d + 1] = make_float2(in.C.ax[d], in.C.ax[d]);
                            s_coef[j & 3][3 * d + 2] = make_float2(in.C.ay[d], in.C.ay[d]);
                            s_coef[j & 3][3 * d + 3] = make_float2(in.C.az[d], in.C.az[d]);
                        }
                    }
                    mbar_expect_tx(&full[slot], bytes);
                    tma_load_4d(ring + slot * kQSlot, map, xs0 - 4, ty * th, zs - D + p, 0, &full[slot]);
                    if (++slot == kQS) slot = 0, phase ^= 1;
                }
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
        }
        if (!ok && lane == 0) {              // the loads in flight land before the CTA leaves (bounded)
            report(a.status, DEV_TIMEOUT);
            for (long long g = i > kQS ? i - kQS : 0; g < i; ++g)
                mbar_wait_bounded(&full[g % kQS], (int)(g / kQS) & 1, 100000000ull);
        }
        return;
    }
    int pos = 0;                             // ring positions: slot, phase, slot to release next
    for (int j = 0;; ++j) {
        // the producer's own wait may take 2 s
        bool ok = mbar_wait_bounded(&full[pos & 15], (pos >> 4) & 1, 4000000000ull);
        const QUnit q = s_unit[j & 3];
        if (ok) {
            if (q.k < 0) return;
            const InstDev& in = a.inst[q.k];
            pos = consume_unit<D>(in, q.t, q.u, smem_u32(s_coef[j & 3]), pos);
            ok = pos >= 0;
        }
        if (!ok) {
            if (lane == 0) report(a.status, DEV_TIMEOUT);
            return;
        }
        __syncwarp();                        // the warp's stores of this unit, then its count
        if (lane == 0) {
            const InstDev& in = a.inst[q.k];
            wq::release_done(&a.done[in.done0 + q.u / (in.ntx * in.nty)]);
        }
    }
}

// ---------------------------------------------------------------- with two-step units
// the four unit bodies are inlined into the kernel (measured faster than
// separate calls, whose calling convention spills the register queues)
#ifdef B2R_BATCH_NOINLINE
#define B2R_UNIT_INLINE __noinline__
#else
#define B2R_UNIT_INLINE __forceinline__
#endif
// the tile shape is the instance's own (run time), so that instances of
// different shapes share the launch
template <int D>
__device__ B2R_UNIT_INLINE bool run_unit(const BatchArgs& a, const InstDev& in, int k, int t, int u,
                                         heatk::Ring& rg)
{
    const int tx = u % in.ntx;
    const int r = u / in.ntx;
    const int ty = r % in.nty;
    const int zc = r / in.nty;
    const int zi0 = zc * in.Lz;
    const int zi1 = min(in.NZ, zi0 + in.Lz);
    return heatk::sweep_unit<D, RowsPerWarp<D>::value, kS, kSlot, 0>(
        &a.maps[2 * k + (t & 1)], in.buf[(t + 1) & 1], in.L, 0, in.C, 0, tx, ty, zi0, zi1, rg, in.lpr);
}

// A two-step unit: round t = sub-steps 2t, 2t+1 (the last round of an odd
// step count: 2t only), through the same ring (positions gp, issued_hi,
// stop in, updated positions and the success flag out).  Not inlined: its
// register queues would otherwise share the budget of the one-step units'.
__device__ __noinline__ uint4 run_two_step(const BatchArgs& a, int k, int t, int u, unsigned gp,
                                           unsigned issued_hi, unsigned stop, float* s1, float* ring)
{
    const InstDev& in = a.inst[k];
    h2k::H2Ctx c;
    c.ring = ring;
    c.s1 = s1;
    c.bar = reinterpret_cast<uint64_t*>(ring + kS * kSlot);
    c.tid = threadIdx.x;
    c.lane = threadIdx.x & 31;
    c.warp = threadIdx.x >> 5;
    c.C = in.C;
    c.plane = in.L.plane;
    c.P = in.L.P;
    c.gp = gp;
    c.issued_hi = issued_hi;
    c.stop = stop;
    c.aborted = false;
    const int tx = u % in.ntx, r = u / in.ntx, ty = r % in.nty, zc = r / in.nty;
    const bool ok = h2k::h2_unit<kS, kSlot>(c, &a.maps[2 * k + (t & 1)], in.buf[(t + 1) & 1], in.L, 0, 0, tx,
                                            ty, zc * in.Lz, in.Lz, 2 * t + 1 == in.nsteps);
    return make_uint4(c.gp, c.issued_hi, c.stop, ok ? 1u : 0u);
}

#ifndef B2R_BATCH_MINB
#define B2R_BATCH_MINB 2   // resident CTAs per SM the register budget is fitted to (no spills)
#endif
// Batches of which some instance runs on two-step units.
__global__ void __launch_bounds__(kThreads, B2R_BATCH_MINB) batch_kernel(const BatchArgs a)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    heatk::Ring rg;
    heatk::ring_init<kS, kSlot>(rg, smem_raw);
    // the two-step units' stage-1 planes after the ring (which ends 16 bytes
    // after its barriers), 128-byte aligned
    float* s1 = reinterpret_cast<float*>(
        (reinterpret_cast<uintptr_t>(rg.abort_flag) + 16 + 127) & ~uintptr_t(127));
    __shared__ long long s_next, s_cur;
    __shared__ int s_t, s_k, s_u, s_ok;
    if (threadIdx.x == 0) s_next = (long long)atomicAdd(a.head, 1ull);
    for (;;) {
        __syncthreads();                     // every thread is done with the last item's values
        if (threadIdx.x == 0) {
            const long long item = s_next;
            s_cur = item;
            if (item < a.total) {
            int t, k, u;
            wq::unpack_item(a.items[item], t, k, u);
            int ok = 1;
            // wait for round t-1 of this instance (bounded)
            if (t > 0) ok = wq::wait_done(&a.done[a.inst[k].done0], (unsigned)t * (unsigned)a.inst[k].units) ? 1 : 0;
            s_t = t;
            s_k = k;
            s_u = u;
            s_ok = ok;
            // claim the next item now, so it is ready when this one is done
            s_next = (long long)atomicAdd(a.head, 1ull);
            }
        }
        __syncthreads();
        if (s_cur >= a.total) break;
        if (!s_ok) {
            if (threadIdx.x == 0) report(a.status, DEV_TIMEOUT);
            return;                          // no load of this CTA is in flight here
        }
        const int t = s_t, k = s_k, u = s_u;
        const InstDev& in = a.inst[k];
        bool ok;
        if (in.tb == 2) {
            const uint4 r = run_two_step(a, k, t, u, rg.gp, rg.issued_hi, rg.stop, s1, rg.smem);
            rg.gp = r.x;
            rg.issued_hi = r.y;
            rg.stop = r.z;
            ok = r.w != 0;
        } else switch (in.D) {
        case 1: ok = run_unit<1>(a, in, k, t, u, rg); break;
        case 2: ok = run_unit<2>(a, in, k, t, u, rg); break;
        case 3: ok = run_unit<3>(a, in, k, t, u, rg); break;
        default: ok = run_unit<4>(a, in, k, t, u, rg); break;
        }
        if (!ok) {
            if (threadIdx.x == 0) report(a.status, DEV_TIMEOUT);
            heatk::ring_drain<kS>(rg);
            return;
        }
        __syncthreads();                     // every store of this unit is issued
        if (threadIdx.x == 0) wq::release_done(&a.done[in.done0]);
    }
}

}  // namespace
}  // namespace b2r

using namespace b2r;

struct b2r_batch {
    int n = 0;
    std::vector<b2r_batch_item> items;
    std::vector<int> order;          // sorted position -> caller index
    std::vector<int> pos;            // caller index -> sorted position
    std::vector<InstDev> host;       // sorted by step count
    std::vector<CUtensorMap> maps;   // sorted by step count, 2 per instance
    std::vector<int> sched;          // queue position -> host index (by rounds, descending)
    InstDev* d_inst = nullptr;
    CUtensorMap* d_maps = nullptr;
    unsigned long long* d_items = nullptr;   // the queue (capacity items_cap)
    long long items_cap = 0;
    unsigned long long* d_head = nullptr;
    unsigned* d_done = nullptr;
    int ndone = 0;                   // its counters
    int* d_status = nullptr;
    float* staging = nullptr;
    size_t staging_bytes = 0;
    int maxrounds = 0;               // rounds of the current schedule's longest instance
    long long total = 0;
    int lz_policy = -1;              // z chunk cap per unit; -1: by the batch's sizes (auto_planes)
    int grid[5] = {};                // persistent grid (every resident slot): radius 1..4, with two-step units
    bool two = false;                // some instance runs on two-step units
    // launches of a run: one per radius (instances sched[first .. first + n), queue d_items + at),
    // or one for all with two-step units
    struct Launch {
        int D, first, n;
        long long at, total;
    };
    std::vector<Launch> runs;
    cudaStream_t side[3] = {};       // the second to fourth launch's streams
    cudaEvent_t fork = nullptr, join[3] = {};
    size_t smem = 0;                 // ring + the two-step units' planes
    cudaGraphExec_t gexec = nullptr;
    cudaStream_t gstream = nullptr;
    long long launches = 0;
};

namespace {

thread_local char g_berr[512];

b2r_status bfail(b2r_status s, const char* msg, cudaError_t e = cudaSuccess)
{
    if (e != cudaSuccess) snprintf(g_berr, sizeof g_berr, "%s: %s", msg, cudaGetErrorString(e));
    else snprintf(g_berr, sizeof g_berr, "%s", msg);
    return s;
}

#define BCK(call, msg)                                                                       \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess) {                                                             \
            cudaGetLastError(); /* a non-sticky error must not resurface in a later check */ \
            return bfail(e_ == cudaErrorMemoryAllocation ? B2R_ERR_OOM : B2R_ERR_CUDA, msg, e_); \
        }                                                                                    \
    } while (0)

inline int roundup(int v, int m) { return (v + m - 1) / m * m; }

// cells one plane of an instance computes with tile shape s; two: in a batch
// with two-step units
long long plane_cells(const b2r_batch* b, int k, int s, bool two)
{
    const InstDev& in = b->host[k];
    const BlockLayout& L = in.L;
    const int D = in.D;
    const int X = L.xoff + L.n[0] - D - ((L.xoff + D) & ~3), Y = L.n[1] - 2 * D;
    const int tw = 4 * kLpr[s], th = two ? kTileY[D][s] : kQTileY[s];
    return (long long)((X + tw - 1) / tw) * tw * ((Y + th - 1) / th) * th;
}

// The tile shape of instance k: the fewest cells computed per plane, narrow
// tiles paying a little for their wider skirt (their boxes re-read a larger
// share of the neighbouring tiles).
int default_shape(const b2r_batch* b, int k, bool two)
{
    static const double penalty[3] = {1.0, 1.03, 1.08};
    int best = 0;
    double bc = 1e300;
    for (int s = 0; s < 3; ++s) {
        const double c = (double)plane_cells(b, k, s, two) * penalty[s];
        if (c < bc - 1e-9) {
            bc = c;
            best = s;
        }
    }
    return best;
}

std::vector<int> default_shapes(const b2r_batch* b, bool two)
{
    std::vector<int> sh(b->n);
    for (int k = 0; k < b->n; ++k) sh[k] = default_shape(b, k, two);
    return sh;
}

b2r_status build_schedule(b2r_batch* b);

// tile counts, steps per unit and tensor-map boxes of every instance for
// its shape sh[k] (two-step units for radius 1 only)
b2r_status set_shapes(b2r_batch* b, const std::vector<int>& sh)
{
    b->two = false;
    for (int k = 0; k < b->n; ++k) b->two = b->two || (sh[k] == kTwoStep && b->host[k].D == 1);
    for (int k = 0; k < b->n; ++k) {
        InstDev& in = b->host[k];
        const BlockLayout& L = in.L;
        const int D = in.D;
        const int s = (sh[k] == kTwoStep && D != 1) ? default_shape(b, k, b->two) : sh[k];
        in.shape = s;
        in.lpr = kLpr[s];
        int bw, bh;
        if (s == kTwoStep) {
            in.tb = 2;
            in.ntx = h2k::h2_ntx(L);
            in.nty = h2k::h2_nty(L);
            bw = h2k::kBoxW;
            bh = h2k::kBoxH;
        } else {
            in.tb = 1;
            const int X = L.xoff + L.n[0] - D - ((L.xoff + D) & ~3), Y = L.n[1] - 2 * D;
            const int tw = 4 * kLpr[s], th = b->two ? kTileY[D][s] : kQTileY[s];
            in.ntx = (X + tw - 1) / tw;
            in.nty = (Y + th - 1) / th;
            bw = tw + 8;
            bh = b->two ? kBoxH[D][s] : kQTileY[s] + 2 * D;
        }
        in.rounds = (in.nsteps + in.tb - 1) / in.tb;
        for (int f = 0; f < 2; ++f)
            if (!make_block_tmap(&b->maps[2 * k + f], in.buf[f], L, 4, bw, bh, 1))
                return bfail(B2R_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    }
    return build_schedule(b);
}

// ... and where that fails (a queue too long), the shapes and the queue of before
b2r_status apply_shapes(b2r_batch* b, const std::vector<int>& sh)
{
    const std::vector<InstDev> host = b->host;
    const std::vector<CUtensorMap> maps = b->maps;
    const bool two = b->two;
    const b2r_status st = set_shapes(b, sh);
    if (st != B2R_OK) {
        b->host = host;
        b->maps = maps;
        b->two = two;
    }
    return st;
}

b2r_status apply_shape(b2r_batch* b, int s) { return apply_shapes(b, std::vector<int>(b->n, s)); }

// Planes per unit when the caller set none (batch_planes.h).
static int auto_planes(const b2r_batch* b)
{
    if (b->two) return 16;
    std::vector<wq::Column> in;
    for (const InstDev& i : b->host) in.push_back({i.D, i.ntx * i.nty, i.NZ, i.rounds});
    return wq::heat_planes(in);
}

// The queue for the current shapes and Lz policy: work items (round,
// instance, unit) written out in claim order, round-major.  A round is one
// step of a one-step instance or two of a two-step one; the instances are
// sorted by their round count (descending), so those still stepping at round
// t are a prefix.  A unit waits only for the previous round of its own
// instance, which the queue holds earlier, so the queue cannot deadlock.
b2r_status build_schedule(b2r_batch* b)
{
    // everything that a run uses changes at the end, together: a queue that is
    // refused leaves the one before it, with its descriptors, in place
    std::vector<int> sched(b->n);
    for (int k = 0; k < b->n; ++k) sched[k] = k;
    std::stable_sort(sched.begin(), sched.end(), [&](int x, int y) {
        const InstDev &p = b->host[x], &q = b->host[y];
        return !b->two && p.D != q.D ? p.D > q.D : p.rounds > q.rounds;
    });
    std::vector<InstDev> host = b->host, dev(b->n);
    std::vector<CUtensorMap> maps(2 * b->n);
    std::vector<int> rounds(b->n), units(b->n);
    int maxrounds = 0, ndone = 0;
    const int policy = b->lz_policy >= 0 ? b->lz_policy : auto_planes(b);
    for (int j = 0; j < b->n; ++j) {
        InstDev& in = host[sched[j]];
        in.Lz = std::min(in.NZ, policy > 0 ? policy : in.NZ);
        in.nzc = (in.NZ + in.Lz - 1) / in.Lz;
        in.units = in.ntx * in.nty * in.nzc;
        in.done0 = ndone;
        ndone += b->two ? 1 : in.nzc;
        dev[j] = in;
        rounds[j] = in.rounds;
        units[j] = in.units;
        maps[2 * j] = b->maps[2 * sched[j]];
        maps[2 * j + 1] = b->maps[2 * sched[j] + 1];
        maxrounds = std::max(maxrounds, in.rounds);
    }
    std::vector<unsigned long long> items, part;
    std::vector<b2r_batch::Launch> runs;
    for (int first = 0; first < b->n;) {
        int n = 1;
        while (first + n < b->n && (b->two || dev[first + n].D == dev[first].D)) ++n;
        if (!wq::round_major_items(rounds.data() + first, units.data() + first, n, part) ||
            (long long)(items.size() + part.size()) > wq::kMaxItems)
            return bfail(B2R_ERR_ARG, "the batch queue is too long (an instance with more than 2^24 units or "
                                      "rounds, or more than 2^28 work items): split the batch");
        runs.push_back({dev[first].D, first, n, (long long)items.size(), (long long)part.size()});
        items.insert(items.end(), part.begin(), part.end());
        first += n;
    }
    const long long total = (long long)items.size();
    // no run of this batch may still read the queue or the descriptors
    BCK(cudaDeviceSynchronize(), "waiting for the batch's runs");
    auto no_graph = [&] {
        if (b->gexec) cudaGraphExecDestroy(b->gexec);
        b->gexec = nullptr;
    };
    BCK(wq::grow(b->d_done, b->ndone, ndone, no_graph), "counter allocation");
    BCK(wq::grow(b->d_items, b->items_cap, std::max<long long>(1, total), no_graph), "queue allocation");
    no_graph();
    BCK(cudaMemcpy(b->d_inst, dev.data(), sizeof(InstDev) * b->n, cudaMemcpyHostToDevice), "copy descriptors");
    BCK(cudaMemcpy(b->d_maps, maps.data(), sizeof(CUtensorMap) * 2 * b->n, cudaMemcpyHostToDevice),
        "copy tensor maps");
    if (total > 0)
        BCK(cudaMemcpy(b->d_items, items.data(), sizeof(unsigned long long) * total, cudaMemcpyHostToDevice),
            "copy the queue");
    b->host = host;
    b->sched = sched;
    b->runs = runs;
    b->total = total;
    b->maxrounds = maxrounds;
    return B2R_OK;
}

b2r_status enqueue_run(b2r_batch* b, cudaStream_t st)
{
    if (!b->d_items || !b->d_done) return bfail(B2R_ERR_STATE, "no memory was left for the batch's queue");
    BCK(cudaMemsetAsync(b->d_head, 0, 4 * sizeof(unsigned long long), st), "reset queue");
    BCK(cudaMemsetAsync(b->d_done, 0, sizeof(unsigned) * b->ndone, st), "reset counters");
    if (b->runs.size() > 1) BCK(cudaEventRecord(b->fork, st), "batch launch");
    for (size_t r = 0; r < b->runs.size(); ++r) {
        const b2r_batch::Launch& u = b->runs[r];
        cudaStream_t s = r == 0 ? st : b->side[r - 1];
        if (r > 0) BCK(cudaStreamWaitEvent(s, b->fork, 0), "batch launch");
        BatchArgs a;
        a.inst = b->d_inst + u.first;
        a.maps = b->d_maps + 2 * u.first;
        a.items = b->d_items + u.at;
        a.head = b->d_head + r;
        a.done = b->d_done;
        a.status = b->d_status;
        a.total = u.total;
        if (b->two) batch_kernel<<<b->grid[4], kThreads, b->smem, s>>>(a);
        else
            switch (u.D) {
            case 1: batch_far_kernel<1><<<b->grid[0], kQThreads, kQSmem, s>>>(a); break;
            case 2: batch_far_kernel<2><<<b->grid[1], kQThreads, kQSmem, s>>>(a); break;
            case 3: batch_far_kernel<3><<<b->grid[2], kQThreads, kQSmem, s>>>(a); break;
            default: batch_far_kernel<4><<<b->grid[3], kQThreads, kQSmem, s>>>(a); break;
            }
        BCK(cudaGetLastError(), "batch launch");
        if (r > 0) {
            BCK(cudaEventRecord(b->join[r - 1], s), "batch launch");
            BCK(cudaStreamWaitEvent(st, b->join[r - 1], 0), "batch launch");
        }
    }
    return B2R_OK;
}

}  // namespace

extern "C" {

const char* b2r_batch_last_error(void) { return g_berr; }

b2r_status b2r_batch_create(const b2r_batch_item* items, int n, b2r_batch** out)
{
    if (!items || n <= 0 || !out) return bfail(B2R_ERR_ARG, "invalid batch description");
    *out = nullptr;
    for (int i = 0; i < n; ++i) {
        const b2r_batch_item& it = items[i];
        if (it.D < 1 || it.D > 4) return bfail(B2R_ERR_ARG, "stencil radius D must be 1..4");
        if (it.nsteps < 0) return bfail(B2R_ERR_ARG, "nsteps must be >= 0");
        for (int a = 0; a < 3; ++a)
            if (it.env[a] < 1) return bfail(B2R_ERR_ARG, "instance sizes must be positive");
    }
    b2r_batch* b = new (std::nothrow) b2r_batch();
    if (!b) return bfail(B2R_ERR_OOM, "host allocation failed");
    b->n = n;
    b->items.assign(items, items + n);
    b->order.resize(n);
    for (int i = 0; i < n; ++i) b->order[i] = i;
    std::stable_sort(b->order.begin(), b->order.end(),
                     [&](int x, int y) { return items[x].nsteps > items[y].nsteps; });
    b->pos.resize(n);
    for (int k = 0; k < n; ++k) b->pos[b->order[k]] = k;
    b->host.resize(n);
    b->maps.resize(2 * n);
    auto bail = [&](b2r_status s) {
        b2r_batch_destroy(b);
        return s;
    };
    for (int k = 0; k < n; ++k) {
        const b2r_batch_item& it = items[b->order[k]];
        InstDev& in = b->host[k];
        const int D = it.D;
        BlockLayout& L = in.L;
        L = BlockLayout{};
        for (int a = 0; a < 3; ++a) {
            L.n[a] = it.env[a] + 2 * D;
            L.B[a] = it.env[a];
            L.nb[a] = 1;
        }
        L.nblk = 1;
        L.H = D;
        L.xoff = roundup(D + 4, 32) - D;
        L.P = roundup(L.xoff + L.n[0] + 8, 32);
        L.periodic = 0;
        L.fixed_edge = 63;
        L.plane = (long long)L.P * L.n[1];
        L.bstride = L.plane * L.n[2];
        in.D = D;
        in.nsteps = it.nsteps;
        in.C = heat_coef(D, it.alpha_dt, it.dx, it.dy, it.dz);
        in.NZ = L.n[2] - 2 * D;
        const size_t fb = (size_t)L.bstride * sizeof(float);
        for (int s = 0; s < 2; ++s) {
            if (cudaMalloc(&in.buf[s], fb) != cudaSuccess)
                return bail(bfail(B2R_ERR_OOM, "instance allocation failed"));
            cudaMemset(in.buf[s], 0, fb);
        }
    }
    if (cudaMalloc(&b->d_inst, sizeof(InstDev) * n) != cudaSuccess ||
        cudaMalloc(&b->d_maps, sizeof(CUtensorMap) * 2 * n) != cudaSuccess ||
        cudaMalloc(&b->d_head, 4 * sizeof(unsigned long long)) != cudaSuccess ||
        cudaMalloc(&b->d_status, sizeof(int)) != cudaSuccess)
        return bail(bfail(B2R_ERR_OOM, "batch table allocation failed"));
    cudaMemset(b->d_status, 0, sizeof(int));
    // a launch per radius, the first on the caller's stream
    bool has[5] = {};
    for (const b2r_batch_item& it : b->items) has[it.D] = true;
    const int sides = has[1] + has[2] + has[3] + has[4] - 1;
    for (int k = 0; k < sides; ++k)
        if (cudaStreamCreateWithFlags(&b->side[k], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&b->join[k], cudaEventDisableTiming) != cudaSuccess)
            return bail(bfail(B2R_ERR_CUDA, "batch streams"));
    if (sides > 0 && cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming) != cudaSuccess)
        return bail(bfail(B2R_ERR_CUDA, "batch streams"));
    // persistent grid: every resident slot
    b->smem = kSmem + 16 + kSmemS1;
    static KernelSetup setup[5];
    using Kernel = void (*)(BatchArgs);
    static const Kernel kerns[5] = {batch_far_kernel<1>, batch_far_kernel<2>, batch_far_kernel<3>, batch_far_kernel<4>,
                                    batch_kernel};
    for (int v = 0; v < 5; ++v)
        if (kernel_setup(setup[v], kerns[v], v < 4 ? kQThreads : kThreads, v < 4 ? kQSmem : b->smem, nullptr, &b->grid[v]) !=
            cudaSuccess)
            return bail(bfail(B2R_ERR_CUDA, "smem attribute"));
    b2r_status st = apply_shapes(b, default_shapes(b, false));
    if (st != B2R_OK) return bail(st);
    if (cudaDeviceSynchronize() != cudaSuccess) return bail(bfail(B2R_ERR_CUDA, "batch set-up failed"));
    *out = b;
    return B2R_OK;
}

b2r_status b2r_batch_destroy(b2r_batch* b)
{
    if (!b) return B2R_OK;
    if (b->gexec) cudaGraphExecDestroy(b->gexec);
    for (int k = 0; k < 3; ++k) {
        if (b->side[k]) cudaStreamDestroy(b->side[k]);
        if (b->join[k]) cudaEventDestroy(b->join[k]);
    }
    if (b->fork) cudaEventDestroy(b->fork);
    for (auto& in : b->host)
        for (int s = 0; s < 2; ++s)
            if (in.buf[s]) cudaFree(in.buf[s]);
    cudaFree(b->d_inst);
    cudaFree(b->d_maps);
    cudaFree(b->d_items);
    cudaFree(b->d_head);
    cudaFree(b->d_done);
    cudaFree(b->d_status);
    if (b->staging) cudaFree(b->staging);
    delete b;
    return B2R_OK;
}

b2r_status b2r_batch_upload(b2r_batch* b, int i, const float* src, int src_is_device, void* stream)
{
    if (!b || !src || i < 0 || i >= b->n) return bfail(B2R_ERR_ARG, "invalid argument");
    const InstDev& in = b->host[b->pos[i]];
    const BlockLayout& L = in.L;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const cudaMemcpyKind kind = src_is_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    for (int s = 0; s < 2; ++s)   // both buffers carry the fixed shell
        BCK(cudaMemcpy2DAsync(in.buf[s] + L.xoff, L.P * sizeof(float), src, L.n[0] * sizeof(float),
                              L.n[0] * sizeof(float), (size_t)L.n[1] * L.n[2], kind, st),
            "upload");
    return B2R_OK;
}

b2r_status b2r_batch_download(b2r_batch* b, int i, float* dst, int dst_is_device, void* stream)
{
    if (!b || !dst || i < 0 || i >= b->n) return bfail(B2R_ERR_ARG, "invalid argument");
    const InstDev& in = b->host[b->pos[i]];
    const BlockLayout& L = in.L;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float* src = in.buf[in.rounds & 1];
    BCK(cudaMemcpy2DAsync(dst, L.n[0] * sizeof(float), src + L.xoff, L.P * sizeof(float),
                          L.n[0] * sizeof(float), (size_t)L.n[1] * L.n[2],
                          dst_is_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st),
        "download");
    if (!dst_is_device) BCK(cudaStreamSynchronize(st), "download sync");
    return B2R_OK;
}

b2r_status b2r_batch_run(b2r_batch* b, void* stream, int use_graph)
{
    if (!b) return bfail(B2R_ERR_ARG, "null batch");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (use_graph && st) {
        if (!b->gexec || b->gstream != st) {
            if (b->gexec) cudaGraphExecDestroy(b->gexec);
            b->gexec = nullptr;
            BCK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal), "begin capture");
            b2r_status s = enqueue_run(b, st);
            cudaGraph_t g = nullptr;
            cudaError_t e = cudaStreamEndCapture(st, &g);
            if (s != B2R_OK) {
                if (g) cudaGraphDestroy(g);
                return s;
            }
            BCK(e, "end capture");
            e = cudaGraphInstantiate(&b->gexec, g, 0);
            cudaGraphDestroy(g);
            BCK(e, "graph instantiate");
            b->gstream = st;
        }
        BCK(cudaGraphLaunch(b->gexec, st), "graph launch");
    } else {
        b2r_status s = enqueue_run(b, st);
        if (s != B2R_OK) return s;
    }
    count_launches((long long)b->runs.size());
    return B2R_OK;
}

b2r_status b2r_batch_synchronize(b2r_batch* b, void* stream)
{
    if (!b) return bfail(B2R_ERR_ARG, "null batch");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int s = 0;
    BCK(cudaMemcpyAsync(&s, b->d_status, sizeof(int), cudaMemcpyDeviceToHost, st), "status");
    BCK(cudaStreamSynchronize(st), "sync");
    if (s != DEV_OK) {
        cudaMemset(b->d_status, 0, sizeof(int));
        return bfail(B2R_ERR_TIMEOUT, "a device-side bounded wait of the batch queue gave up");
    }
    return B2R_OK;
}

int64_t b2r_batch_lups(const b2r_batch* b)
{
    if (!b) return 0;
    int64_t s = 0;
    for (const auto& it : b->items) s += (int64_t)it.env[0] * it.env[1] * it.env[2] * it.nsteps;
    return s;
}

static b2r_status set_policy(b2r_batch* b, int policy)
{
    const int before = b->lz_policy;
    b->lz_policy = policy;
    const b2r_status st = build_schedule(b);
    if (st != B2R_OK) b->lz_policy = before;
    return st;
}

b2r_status b2r_batch_set_zchunk(b2r_batch* b, int zchunk)
{
    if (!b || zchunk < 0) return bfail(B2R_ERR_ARG, "invalid argument");
    return set_policy(b, zchunk);
}

b2r_status b2r_batch_autotune(b2r_batch* b, void* stream, int* best_zchunk, double* best_ms)
{
    if (!b) return bfail(B2R_ERR_ARG, "null batch");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the runs overwrite the instance buffers: keep buffer 0 of every instance
    // (freed on every return path)
    struct SaveBufs {
        std::vector<float*> p;
        ~SaveBufs()
        {
            for (float* q : p)
                if (q) cudaFree(q);
        }
    } saved;
    saved.p.assign(b->n, nullptr);
    std::vector<float*>& save = saved.p;
    for (int k = 0; k < b->n; ++k) {
        const size_t fb = (size_t)b->host[k].L.bstride * sizeof(float);
        BCK(cudaMalloc(&save[k], fb), "autotune save");
        BCK(cudaMemcpyAsync(save[k], b->host[k].buf[0], fb, cudaMemcpyDeviceToDevice, st), "save");
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    // one whole run from the saved inputs, timed
    auto trial = [&](float& ms) -> b2r_status {
        for (int k = 0; k < b->n; ++k)
            cudaMemcpyAsync(b->host[k].buf[0], save[k], (size_t)b->host[k].L.bstride * sizeof(float),
                            cudaMemcpyDeviceToDevice, st);
        cudaEventRecord(e0, st);
        b2r_status r = enqueue_run(b, st);
        if (r != B2R_OK) return r;
        cudaEventRecord(e1, st);
        if ((r = b2r_batch_synchronize(b, st)) != B2R_OK) return r;
        cudaEventElapsedTime(&ms, e0, e1);
        return B2R_OK;
    };
    // the size class is the interior width (the extent a tile width divides)
    auto cls = [&](int k) {
        const int w = b->items[b->order[k]].env[0];
        return (b->host[k].D - 1) * 3 + (w <= 64 ? 0 : (w <= 128 ? 1 : 2));
    };
    struct Found {
        float ms = 1e30f;
        int z = 0;
        std::vector<int> sh;
    };
    // the best schedule found from one set of z chunks (-1: by the sizes)
    auto search = [&](const std::vector<int>& zs, Found& f) -> b2r_status {
        // the z chunk for the current shapes (a change must gain 0.5 %)
        auto tune_zchunk = [&]() -> b2r_status {
            for (int z : zs) {
                float ms = 0.f;
                b2r_status r = set_policy(b, z);
                if (r == B2R_OK) r = trial(ms);
                if (r != B2R_OK) return r;
                if (ms < f.ms * (z == f.z ? 1.f : 0.995f)) {
                    f.ms = ms;
                    f.z = z;
                }
            }
            return set_policy(b, f.z);
        };
        // 1. the z chunk with every instance on its fewest-cells shape
        f.sh = default_shapes(b, false);
        b2r_status s = apply_shapes(b, f.sh);
        if (s == B2R_OK) s = tune_zchunk();
        // 2. tile shapes per (stencil order, size class): the instances of one
        // class try each other shape while the rest keep theirs (radius 1 also
        // the two-step units)
        bool changed = false;
        for (int c = 0; c < 12 && s == B2R_OK; ++c)
            for (int t = 0; t < kShapes && s == B2R_OK; ++t) {
                if (t == kTwoStep && c >= 3) continue;      // two-step units: radius 1 only
                std::vector<int> cand = f.sh;
                bool differs = false;
                for (int k = 0; k < b->n; ++k)
                    if (cls(k) == c && cand[k] != t) {
                        cand[k] = t;
                        differs = true;
                    }
                if (!differs) continue;
                float ms = 0.f;
                if ((s = apply_shapes(b, cand)) != B2R_OK || (s = trial(ms)) != B2R_OK) break;
                if (ms < f.ms * 0.995f) {
                    f.ms = ms;
                    f.sh = cand;
                    changed = true;
                }
            }
        // 3. the z chunk again for the shapes picked
        if (s == B2R_OK) s = apply_shapes(b, f.sh);
        if (s == B2R_OK && changed && zs.size() > 1) s = tune_zchunk();
        return s;
    };
    // once with the units that the sizes give, as at creation, and once with
    // fixed z chunks, which two-step units may want (ms of 18 instances of 24..75
    // cells a side, of 12 of 24..39 with radius 4: 4.73, 1.30 with the former,
    // 4.43, 1.98 with the latter)
    Found own, fixed;
    b2r_status s = search({-1}, own);
    if (s == B2R_OK) s = search({8, 16, 32, 64, 0}, fixed);
    const Found& best = fixed.ms < own.ms * 0.995f ? fixed : own;
    const int bestz = best.z;
    if (s == B2R_OK) s = set_policy(b, bestz);
    if (s == B2R_OK) s = apply_shapes(b, best.sh);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    // restore every instance even after a failed trial; report the first failure
    cudaError_t rerr = cudaSuccess;
    for (int k = 0; k < b->n; ++k) {
        const cudaError_t e = cudaMemcpyAsync(b->host[k].buf[0], save[k],
                                              (size_t)b->host[k].L.bstride * sizeof(float),
                                              cudaMemcpyDeviceToDevice, st);
        if (rerr == cudaSuccess) rerr = e;
    }
    const cudaError_t se = cudaStreamSynchronize(st);
    if (rerr == cudaSuccess) rerr = se;
    if (s != B2R_OK) return s;
    BCK(rerr, "restoring the instances after the trials");
    if (best_zchunk) *best_zchunk = bestz >= 0 ? bestz : auto_planes(b) <= 8 ? 8 : 16;
    if (best_ms) *best_ms = best.ms;
    return B2R_OK;
}

b2r_status b2r_batch_set_tile(b2r_batch* b, int width)
{
    if (!b) return bfail(B2R_ERR_ARG, "null batch");
    switch (width) {
    case 0: return apply_shapes(b, default_shapes(b, false));
    case 128: return apply_shape(b, 0);
    case 64: return apply_shape(b, 1);
    case 32: return apply_shape(b, 2);
    default: return bfail(B2R_ERR_ARG, "tile width must be 128, 64, 32 or 0");
    }
}

int b2r_batch_tile(const b2r_batch* b)
{
    if (!b) return 0;
    for (int k = 1; k < b->n; ++k)
        if (b->host[k].lpr != b->host[0].lpr) return 0;
    return 4 * b->host[0].lpr;
}

int b2r_batch_instance_tile(const b2r_batch* b, int i)
{
    return b && i >= 0 && i < b->n ? 4 * b->host[b->pos[i]].lpr : 0;
}

b2r_status b2r_batch_set_pass_steps(b2r_batch* b, int steps)
{
    if (!b) return bfail(B2R_ERR_ARG, "null batch");
    if (steps != 1 && steps != 2) return bfail(B2R_ERR_ARG, "steps per pass must be 1 or 2");
    std::vector<int> sh(b->n);
    for (int k = 0; k < b->n; ++k)
        sh[k] = b->host[k].D == 1 ? (steps == 2 ? kTwoStep : default_shape(b, k, false)) : b->host[k].shape;
    return apply_shapes(b, sh);
}

int b2r_batch_instance_pass_steps(const b2r_batch* b, int i)
{
    return b && i >= 0 && i < b->n ? b->host[b->pos[i]].tb : 0;
}

}  // extern "C"
