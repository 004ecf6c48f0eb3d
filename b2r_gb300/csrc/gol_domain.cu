// gol_domain.cu -- Game of Life generations on the whole domain as a bit grid.
//
// Between two looks at the cells (b2r_step over several generations) the
// blocks and their halos are not needed: the domain's cells are packed once
// into one bit per cell (rows of 32-cell words, the fixed shell included, or
// the bare torus), the generations run on two ping-pong bit grids, and the
// block interiors are written once at the end.  The grid of the 256^3 torus
// is 2 MB, so every pass runs out of L2, there is no halo exchange, and a
// pass is bound by the integer pipe instead of by bytes moving through L2.
//
// Rule (gol-3D.cu:83-99) on the 27-cell total T that includes the cell:
// live -> 3 <= T <= 8, dead -> T == 5, added with bit-sliced full adders in
// the order x, y, z: the two-bit x sums of a row are shared by the three rows
// of the y sums, and the four-bit y sums by the three planes of the z sums,
// which a thread keeps in registers as it marches z -- 42 logic operations
// per word against 60 with z summed first (gol_bits.cu), and no shuffles.
//
// One launch advances G generations: a CTA loads a region of PR rows x PZ
// planes (its output and G more on each side; wrapped on a torus) of whole
// rows -- or of XO output words and a halo word on each side where a row has
// more than 32 words -- into shared memory, runs the generations between two
// shared buffers, each valid one cell less deep, and stores the output.  A
// thread owns one word of two rows and marches a z segment, one barrier per
// generation.
//
// Measured, 256^3 torus in 2x2x2 blocks, R = 4: 3.8 us per generation against
// 17.1 for the several-generation block pass with its halo gather (400
// generations with upload and download 1.63 ms against 7.02); 512^3 with a
// shell 27 against 56; 64^3 torus 1.3 against 14.7.  A pass of four
// generations takes 15.5 us, about 5 of them launch and load (G = 2 to 8
// measured: 4.9, 4.4, 3.8, 4.1, 4.6, 4.8 us per generation); the integer pipe
// is 55 % busy over the whole pass.
#include <algorithm>
#include <array>
#include <map>
#include <mutex>

#include "b2r_common.cuh"
#include "gol.h"

namespace b2r {

namespace {

constexpr int kMaxG = kGolDomainMaxGen;
constexpr int kNR = kGolRows, kMaxThreads = kGolMaxThreads;
constexpr int kMaxPR = kGolMaxRegion, kMaxPZ = kGolMaxRegion;


// One three-input logic instruction each, by its truth table (bit 4a + 2b + c).  Written out because the compiler
// otherwise shares two-input parts between neighbouring sums, which costs more instructions than it saves.
template <int TABLE>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(TABLE));
    return d;
}
__device__ __forceinline__ uint32_t x3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0x96>(a, b, c); }   // a ^ b ^ c
__device__ __forceinline__ uint32_t mj(uint32_t a, uint32_t b, uint32_t c) { return lop3<0xE8>(a, b, c); }   // two or more
__device__ __forceinline__ uint32_t or3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0xFE>(a, b, c); }
__device__ __forceinline__ uint32_t sel(uint32_t m, uint32_t a, uint32_t b) { return lop3<0xCA>(m, a, b); }  // m ? a : b

// 32 cells of a torus row of nx cells from cell s on (any s): the pieces up
// to the wraps one after another
__device__ __forceinline__ uint32_t row_bits(const uint32_t* row, int s, int nx)
{
    s %= nx;
    if (s < 0) s += nx;
    uint32_t v = 0;
    for (int got = 0; got < 32;) {
        const int off = s & 31;
        const int take = min(32 - got, min(32 - off, nx - s));
        uint32_t b = __ldcg(row + (s >> 5)) >> off;
        if (take < 32) b &= (1u << take) - 1u;
        v |= b << got;
        got += take;
        s += take;
        if (s >= nx) s = 0;
    }
    return v;
}

// RAG: a torus whose rows end inside a word; the last cell's right neighbour
// and the first cell's left one are then found by shifts
template <bool RAG, int RP>
__global__ void __launch_bounds__(kMaxThreads)
gol_domain_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, const GolPass P)
{
    extern __shared__ uint32_t sm[];
    __shared__ int row_of[kMaxPR], plane_of[kMaxPZ];   // grid row / plane of a region row / plane, -1 outside
    const int tid = threadIdx.x;
    const int G = P.G, WX = P.WX, RPZ = P.RPZ;
    int b = blockIdx.x;
    const int tx = b % P.ntx;
    b /= P.ntx;
    const int y0 = (b % P.nty) * P.Ty, z0 = (b / P.nty) * P.Tz;   // first output row / plane
    const int buf_w = P.PZ * RPZ;
    for (int i = tid; i < P.PR + P.PZ; i += blockDim.x) {
        const bool isrow = i < P.PR;
        const int n = isrow ? P.ny : P.nz;
        int c = (isrow ? y0 + i : z0 + i - P.PR) - G;
        if (P.periodic) {
            c %= n;
            if (c < 0) c += n;
        }
        if (c >= n) c = -1;
        (isrow ? row_of[i] : plane_of[i - P.PR]) = c;
    }
    const int w = tid % WX, wq = tid / WX;
    {   // the padding rows: read, never used
        for (int q = wq; q < 2 * P.PZ; q += blockDim.x / WX)
            if (wq < blockDim.x / WX) {
                const int o = (q >> 1) * RPZ + (q & 1 ? P.PR + 1 : 0) * RP + w;
                sm[o] = 0u;
                sm[buf_w + o] = 0u;
            }
    }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");             // the previous pass wrote `in`
    asm volatile("griddepcontrol.launch_dependents;");
    {
        // the region: rows y0-G .., planes z0-G ..; a thread keeps its word
        // and steps through the rows of all planes
        const int step = blockDim.x / WX;
        int r = wq, p = 0;
        const int k = tx * P.XO - 1 + w;
        if (wq < step)
            while (p < P.PZ) {
                uint32_t v[4];
                int o[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    while (r >= P.PR) r -= P.PR, ++p;
                    v[u] = 0u;
                    o[u] = -1;
                    if (p < P.PZ) {
                        o[u] = p * RPZ + (r + 1) * RP + w;
                        const int y = row_of[r], z = plane_of[p];
                        if (y >= 0 && z >= 0) {
                            const uint32_t* row = in + ((long long)z * P.ny + y) * P.W;
                            if (!P.split) v[u] = __ldcg(row + w);
                            else if (k >= 0 && 32 * k + 32 <= P.nx) v[u] = __ldcg(row + k);
                            else if (P.periodic) v[u] = row_bits(row, 32 * k, P.nx);
                            else if (k >= 0 && k < P.W) v[u] = __ldcg(row + k);
                        }
                        r += step;
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (o[u] >= 0) sm[o[u]] = v[u];
            }
    }
    const int yg = wq % (P.PR / kNR), seg = wq / (P.PR / kNR);
    const bool thread_ok = seg < P.nzs;
    // the words left and right of this one; ends of a whole torus row wrap,
    // any other end is a shell cell or a halo word, whose value is not used
    int wl = w - 1, wr = w + 1, sl = 0, sr = 0;
    if (w == 0) {
        wl = !P.split && P.periodic ? WX - 1 : 0;
        if (RAG) sl = 31 - ((P.nx - 1) & 31);
    }
    if (w == WX - 1) {
        wr = !P.split && P.periodic ? 0 : WX - 1;
        if (RAG) sr = 31 - ((P.nx - 1) & 31);
    }
    // cells of this word that change: every cell of a torus, the cells inside a shell
    const int kw = P.split ? tx * P.XO - 1 + w : w;
    uint32_t xm = 0xFFFFFFFFu;
    if (!P.periodic || !P.split) {
        const int lo = P.periodic ? 0 : 1, hi = P.periodic ? P.nx - 1 : P.nx - 2;
        const int a = max(lo - 32 * kw, 0), e = min(hi - 32 * kw, 31);
        xm = a > e ? 0u : (e - a == 31 ? 0xFFFFFFFFu : (((1u << (e - a + 1)) - 1u) << a));
    }
    const bool wout = !P.split || (w >= 1 && w <= P.XO && kw < P.W);
    const uint32_t row_end = P.nx - 32 * kw < 32 ? (1u << max(P.nx - 32 * kw, 0)) - 1u : 0xFFFFFFFFu;
    uint32_t ym[kNR];
#pragma unroll
    for (int k = 0; k < kNR; ++k) {
        const int y = y0 - G + kNR * yg + k;
        ym[k] = P.periodic || (y >= 1 && y <= P.ny - 2) ? xm : 0u;
    }
    const uint32_t* src = sm;
    uint32_t* dst = sm + buf_w;
    for (int g = 1; g <= G; ++g) {
        __syncthreads();
        const int np = P.PZ - 2 * g, sz = (np + P.nzs - 1) / P.nzs;
        const int p0 = g + seg * sz, p1 = min(p0 + sz, P.PZ - g);
        if (thread_ok && p0 < p1 && kNR * yg + kNR - 1 >= g && kNR * yg < P.PR - g) {
            // y sums (0..9, in four words of weights 1, 2, 2, 4) of this word's rows in plane p, and the
            // cells themselves
            auto ysum = [&](int p, uint32_t (&v)[kNR][4], uint32_t (&cur)[kNR]) {
                const uint32_t* q = src + p * RPZ + kNR * yg * RP;     // its first padded row is the row below the thread's
                uint32_t c0[kNR + 2], c1[kNR + 2];
#pragma unroll
                for (int k = 0; k < kNR + 2; ++k) {
                    const uint32_t m = q[k * RP + w];
                    uint32_t l = q[k * RP + wl], r = q[k * RP + wr];
                    if (RAG) {
                        l = __funnelshift_l(l << sl, m, 1);
                        r = (m >> 1) | ((r << 31) >> sr);
                    } else {
                        l = __funnelshift_l(l, m, 1);
                        r = __funnelshift_r(m, r, 1);
                    }
                    c0[k] = x3(l, m, r);
                    c1[k] = mj(l, m, r);
                    if (k >= 1 && k <= kNR) cur[k - 1] = m;
                }
#pragma unroll
                for (int k = 0; k < kNR; ++k) {
                    v[k][0] = x3(c0[k], c0[k + 1], c0[k + 2]);   // of weight 1
                    v[k][1] = mj(c0[k], c0[k + 1], c0[k + 2]);   // of weight 2
                    v[k][2] = x3(c1[k], c1[k + 1], c1[k + 2]);   // of weight 2
                    v[k][3] = mj(c1[k], c1[k + 1], c1[k + 2]);   // of weight 4
                }
            };
            // plane p from the y sums of planes p-1 (va), p (vb) and p+1 (vc, made here)
            auto plane = [&](int p, uint32_t (&va)[kNR][4], uint32_t (&vb)[kNR][4], uint32_t (&cb)[kNR],
                             uint32_t (&vc)[kNR][4], uint32_t (&cc)[kNR]) {
                ysum(p + 1, vc, cc);
                const int z = z0 - G + p;
                uint32_t res[kNR];
#pragma unroll
                for (int k = 0; k < kNR; ++k) {
                    const uint32_t s0 = x3(va[k][0], vb[k][0], vc[k][0]), a1 = mj(va[k][0], vb[k][0], vc[k][0]);
                    const uint32_t b1 = x3(va[k][1], vb[k][1], vc[k][1]), b2 = mj(va[k][1], vb[k][1], vc[k][1]);
                    const uint32_t c1 = x3(va[k][2], vb[k][2], vc[k][2]), c2 = mj(va[k][2], vb[k][2], vc[k][2]);
                    const uint32_t s1 = x3(a1, b1, c1), d2 = mj(a1, b1, c1);
                    const uint32_t e2 = x3(va[k][3], vb[k][3], vc[k][3]), e3 = mj(va[k][3], vb[k][3], vc[k][3]);
                    const uint32_t f2 = x3(b2, c2, d2), f3 = mj(b2, c2, d2);
                    const uint32_t s2 = e2 ^ f2, g3 = e2 & f2;
                    // T = s0 + 2 s1 + 4 s2 + 8 (e3 + f3 + g3)
                    const uint32_t c = cb[k];
                    // T <= 7, live 3..7 or dead 5: s2 & (c | (~s1 & s0)) | (c & s1 & s0)
                    const uint32_t low = lop3<0xEA>(s2, lop3<0xF2>(c, s1, s0), lop3<0x80>(c, s1, s0));
                    // T == 8, live: c & ~(s2 | s1 | s0), one of the eights
                    const uint32_t eight = lop3<0x10>(c, or3(s2, s1, s0), mj(e3, f3, g3));
                    res[k] = sel(ym[k], sel(or3(e3, f3, g3), eight, low), c);
                }
                if (!P.periodic && (z < 1 || z > P.nz - 2)) {   // a shell plane
#pragma unroll
                    for (int k = 0; k < kNR; ++k) res[k] = cb[k];
                }
                if (g < G) {
                    uint32_t* d = dst + p * RPZ + (kNR * yg + 1) * RP + w;
#pragma unroll
                    for (int k = 0; k < kNR; ++k) d[k * RP] = res[k];
                } else if (wout && p < G + P.Tz && z < P.nz) {
                    uint32_t* d = out + ((long long)z * P.ny + y0 - G + kNR * yg) * P.W + kw;
#pragma unroll
                    for (int k = 0; k < kNR; ++k) {
                        const int r = kNR * yg + k;
                        // cells past the row's end stay 0 (a cut torus row carries wrapped cells there)
                        if (r >= G && r < G + P.Ty && y0 - G + r < P.ny) d[(long long)k * P.W] = res[k] & row_end;
                    }
                }
            };
            uint32_t va[kNR][4], vb[kNR][4], vc[kNR][4], ca[kNR], cb[kNR], cc[kNR];
            ysum(p0 - 1, va, ca);
            ysum(p0, vb, cb);
            for (int p = p0; p < p1; p += 3) {   // the queue turns by names
                plane(p, va, vb, cb, vc, cc);
                if (p + 1 < p1) plane(p + 1, vb, vc, cc, va, ca);
                if (p + 2 < p1) plane(p + 2, vc, va, ca, vb, cb);
            }
        }
        const uint32_t* t = src;
        src = dst;
        dst = const_cast<uint32_t*>(t);
    }
}

// Cell c (-1 .. env: shell cells of a shelled domain) of an axis in block b
// at storage coordinate i.
__device__ __forceinline__ void cell_of(int c, int B, int nb, int H, int& b, int& i)
{
    b = min(max(c, 0) / B, nb - 1);
    i = c - b * B + H;
}

// 32 byte cells (0 / not 0) of a storage row at a multiple of 32 -> one word
__device__ __forceinline__ uint32_t pack16(const uint4 a)
{
    // 0/1 bytes at bits 0, 8, 16, 24 -> bits 28 .. 31, no carries
    return ((a.x * 0x10204080u) >> 28) | (((a.y * 0x10204080u) >> 28) << 4) | (((a.z * 0x10204080u) >> 28) << 8) |
           (((a.w * 0x10204080u) >> 28) << 12);
}
__device__ __forceinline__ uint32_t pack_chunk(const uint8_t* p)
{
    const uint4* q = reinterpret_cast<const uint4*>(p);
    return pack16(__ldg(q)) | (pack16(__ldg(q + 1)) << 16);
}
__device__ __forceinline__ uint4 unpack16(uint32_t v)
{
    // bits n0..n3 -> bytes 0/1: bit i lands on i + 7m (m = 0..3), all distinct
    return make_uint4(((v & 15u) * 0x00204081u) & 0x01010101u, (((v >> 4) & 15u) * 0x00204081u) & 0x01010101u,
                      (((v >> 8) & 15u) * 0x00204081u) & 0x01010101u,
                      (((v >> 12) & 15u) * 0x00204081u) & 0x01010101u);
}

// Block cells -> bit grid (shell cells from the edge blocks' halos).  A
// thread makes one word of a row from the 32-byte chunks of the block rows
// that hold its cells: one chunk where block rows are multiples of 32 cells.
__global__ void __launch_bounds__(256)
gol_pack_kernel(const uint8_t* __restrict__ blocks, uint32_t* __restrict__ bits, const BlockLayout L, const int shell,
                const int nx, const int ny, const int nz, const int W)
{
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int w = i % W, y = i / W;
    if (y >= ny) return;
    for (int z = blockIdx.y; z < nz; z += gridDim.y) {
        int by, iy, bz, iz;
        cell_of(y - shell, L.B[1], L.nb[1], L.H, by, iy);
        cell_of(z - shell, L.B[2], L.nb[2], L.H, bz, iz);
        const uint8_t* base = blocks + (long long)L.nb[0] * (by + (long long)L.nb[1] * bz) * L.bstride +
                              iz * L.plane + (long long)iy * L.P;
        const int n = min(32, nx - 32 * w);
        uint32_t v = 0;
        for (int got = 0; got < n;) {
            int bx, ix;
            cell_of(32 * w + got - shell, L.B[0], L.nb[0], L.H, bx, ix);
            // cells of this block's row from ix on: its interior, and the shell cell after the last block
            const int take = min(n - got, L.H + L.B[0] + (bx == L.nb[0] - 1 ? shell : 0) - ix);
            const int pos = L.xoff + ix, a = pos & 31;
            const uint8_t* c = base + bx * L.bstride + (pos - a);
            uint32_t u = pack_chunk(c) >> a;
            if (a + take > 32) u |= pack_chunk(c + 32) << (32 - a);
            if (take < 32) u &= (1u << take) - 1u;
            v |= u << got;
            got += take;
        }
        bits[((long long)z * ny + y) * W + w] = v;
    }
}

// Bit grid -> block interiors.  A thread writes the interior cells of one
// 32-byte chunk of a block row (interior rows start on a 128-byte boundary).
__global__ void __launch_bounds__(256)
gol_unpack_kernel(uint8_t* __restrict__ blocks, const uint32_t* __restrict__ bits, const BlockLayout L,
                  const int shell, const int ny, const int W)
{
    const int chunks = (L.B[0] + 31) / 32;
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int c = i % chunks, yd = i / chunks;                  // chunk and row of the domain's interior
    const int rows = L.B[1] * L.nb[1], planes = L.B[2] * L.nb[2];
    if (yd >= rows * L.nb[0]) return;
    const int bx = yd / rows, y = yd % rows;
    const int by = y / L.B[1], iy = y % L.B[1] + L.H;
    const int x0 = bx * L.B[0] + 32 * c + shell;                // grid cell of the chunk's first cell
    const int n = min(32, L.B[0] - 32 * c);
    for (int z = blockIdx.y; z < planes; z += gridDim.y) {
        const int bz = z / L.B[2], iz = z % L.B[2] + L.H;
        const uint32_t* row = bits + ((long long)(z + shell) * ny + y + shell) * W;
        uint32_t v = __ldcg(row + (x0 >> 5)) >> (x0 & 31);
        if ((x0 & 31) + n > 32) v |= __ldcg(row + (x0 >> 5) + 1) << (32 - (x0 & 31));
        uint8_t* d = blocks + (bx + (long long)L.nb[0] * (by + (long long)L.nb[1] * bz)) * L.bstride + iz * L.plane +
                     (long long)iy * L.P + L.xoff + L.H + 32 * c;
        const uint4 lo = unpack16(v), hi = unpack16(v >> 16);
        if (n == 32) {
            reinterpret_cast<uint4*>(d)[0] = lo;
            reinterpret_cast<uint4*>(d)[1] = hi;
        } else {
            for (int k = 0; k < n; ++k) d[k] = (v >> k) & 1u;
        }
    }
}

// The plan of a pass, once per domain and generations to go: kept for the process
// (512 at most), so that a new domain of a known size has it at hand.
GolPass plan_of(const GolPass& base, int left, int sms)
{
    static std::mutex mu;
    static std::map<std::array<int, 6>, GolPass> known;
    const std::array<int, 6> key{base.nx, base.ny, base.nz, base.periodic, left, sms};
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = known.find(key);
        if (it != known.end()) return it->second;
    }
    const GolPass p = gol_plan_pass(base, left, sms);
    std::lock_guard<std::mutex> lock(mu);
    if (known.size() >= 512) known.clear();
    known[key] = p;
    return p;
}

}  // namespace

size_t gol_domain_words(const int env[3], int shell)
{
    return (size_t)((env[0] + 2 * shell + 31) / 32) * (env[1] + 2 * shell) * (env[2] + 2 * shell);
}

cudaError_t launch_gol_domain(uint8_t* blocks, uint32_t* bits, const int env[3], int shell, const BlockLayout& L,
                              int gens, GolDomainPlans& plans, cudaStream_t st)
{
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const GolPass P = gol_pass_rows(env[0] + 2 * shell, env[1] + 2 * shell, env[2] + 2 * shell, shell == 0);
    const bool rag = P.periodic && !P.split && P.nx % 32 != 0;
    uint32_t* grid[2] = {bits, bits + gol_domain_words(env, shell)};

    gol_pack_kernel<<<dim3((unsigned)((P.W * (long long)P.ny + 255) / 256), std::min(P.nz, 65535)), 256, 0, st>>>(
        blocks, grid[0], L, shell, P.nx, P.ny, P.nz, P.W);
    count_launches(1);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;

    using Kern = void (*)(const uint32_t*, uint32_t*, GolPass);
#define B2R_GOL_PITCHES(RAG)                                                                          \
    {gol_domain_kernel<RAG, 2>,  gol_domain_kernel<RAG, 6>,  gol_domain_kernel<RAG, 10>,               \
     gol_domain_kernel<RAG, 14>, gol_domain_kernel<RAG, 18>, gol_domain_kernel<RAG, 22>,               \
     gol_domain_kernel<RAG, 26>, gol_domain_kernel<RAG, 30>, gol_domain_kernel<RAG, 34>}
    static const Kern kerns[2][9] = {B2R_GOL_PITCHES(false), B2R_GOL_PITCHES(true)};
#undef B2R_GOL_PITCHES
    static SmemLimit limit[2][9];
    const int pitch = gol_row_pitch(P.WX) / 4;
    const Kern kern = kerns[rag][pitch];
    int cur = 0;
    for (int left = gens; left > 0;) {
        GolPass& plan = plans.p[std::min(left, kMaxG)];
        if (plan.G == 0) plan = plan_of(P, std::min(left, kMaxG), sms);
        if ((e = raise_smem_limit(limit[rag][pitch], (const void*)kern, std::max<size_t>(plan.smem, 48 * 1024)))) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(plan.ntx * plan.nty * ((plan.nz + plan.Tz - 1) / plan.Tz)));
        cfg.blockDim = dim3(plan.threads);
        cfg.dynamicSmemBytes = plan.smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kern, (const uint32_t*)grid[cur], grid[1 - cur], plan);
        count_launches(1);
        if (e != cudaSuccess) return e;
        cur = 1 - cur;
        left -= plan.G;
    }
    const long long chunk_rows = (long long)((L.B[0] + 31) / 32) * env[1] * L.nb[0];
    gol_unpack_kernel<<<dim3((unsigned)((chunk_rows + 255) / 256), std::min(env[2], 65535)), 256, 0, st>>>(
        blocks, grid[cur], L, shell, P.ny, P.W);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace b2r
