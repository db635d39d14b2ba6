// Low-octave desert proxy on zone grids (stage S4).
//
// Reference: src/gpu/gproxy.cu:91-120 (k_proxy, FP32) and src/desert_proxy.hpp:24-31 (DesertProxy::prob,
// FP64).  The reference GPU kernel evaluates the proxy in FP32 and is not bit-exact with the CPU
// (`gpucheck` only reports a difference count, dsearch_desert.cpp:445-450).  This kernel evaluates it in
// FP64 with the CPU's exact operation order, so every bitmap cell equals the CPU proxy's decision:
// T (2 octaves x 2 sides) >= 0.55, then C octaves 0-2 and E octaves 0-1 of both sides binned into the
// 40 x 40 probability table, passable iff prob >= cut.  One thread per step-32 cell; a zone's cells
// spread over many blocks so that a single large zone fills the GPU (gproxy.cu:91-93).
#include "noise.cuh"
#include "zones.cuh"
#include <algorithm>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace dsg {
namespace {
float g_cut = 0.35f;
using zones::DZone;
using zones::CHUNK;
using zones::ZoneWork;
using zones::CompStat;
// The chunks of CHUNK cells a block handles: (zone blockIdx.x, chunk blockIdx.y) when the host knows the zones
// (w.chunk == null), else chunks w.chunk[k] for k = blockIdx.x, blockIdx.x + gridDim.x, ... < *w.nchunk (zones and
// their cell offsets built on the device).  f(zone index, zone, first cell, end cell) runs for each.
template <class F> __device__ __forceinline__ void each_chunk(const DZone *__restrict__ zones, const ZoneWork &w, F &&f) {
    if (!w.chunk) {
        const DZone z = zones[blockIdx.x];
        const int64_t n = int64_t(z.nx) * z.nz, c0 = int64_t(blockIdx.y) * CHUNK;
        if (c0 < n) f(blockIdx.x, z, c0, min(n, c0 + CHUNK));
        return;
    }
    const uint32_t nch = *w.nchunk;
    for (uint32_t k = blockIdx.x; k < nch; k += gridDim.x) {
        const uint2 zc = w.chunk[k];
        const DZone z = zones[zc.x];
        const int64_t n = int64_t(z.nx) * z.nz, c0 = int64_t(zc.y) * CHUNK;
        f(zc.x, z, c0, min(n, c0 + CHUNK));
    }
}

// ---- the proxy over tiles of 32 x 32 cells
// The cells of a zone lie on a regular grid, so per octave a tile's positions, fractions and fades depend on the column
// or the row alone, and the lattice columns under the tile are few (3 x 3 at frequency 2^-10, 10 x 10 at 2^-7).  The
// block works those out once per tile: 32 (fraction, fade) pairs per axis and the gradient terms of the lattice columns
// (LatticePoint, as the flood engine's patches).  A cell then takes about 35 FP64 instructions per octave and no hashing,
// where it took 69 and 137 others.  The values are the same doubles: the same expressions, evaluated once per column or row.
// C and E follow only where a cell of the tile is hot.
// Measured (B200, 160 zones of about 195 x 195 cells): 412 us before, 266 now; one launch is bound by the latency of its
// FP64 chains (FP64 pipe 52%, issue 52%, shared-memory wavefronts 68%, 4 blocks of 8 warps per SM by registers).  A cell
// per thread, every corner loaded, was bound by shared memory (78% of its wavefronts; 350 us); rows that test one by one
// for a new lattice row serialised (316 us); 2 or 3 blocks per SM without spills 314 and 277 us.
// A zone narrower than 8 cells, or one whose coordinates wrap, is evaluated cell by cell (zones::tiled).
constexpr int PT = 32, POCT = 14;                         // tile side; octaves: T (A 0-1, B 0-1), C 0-2 (A, B), E 0-1 (A, B)
struct ProxyOct { int oct, side, log2f; };                // octave in SeedNoise, side, -log2 of its frequency
constexpr ProxyOct kPO[POCT] = {{0, 0, 10}, {1, 0, 8}, {2, 1, 10}, {3, 1, 8}, {8, 0, 9}, {9, 0, 8}, {10, 0, 7}, {17, 1, 9}, {18, 1, 8}, {19, 1, 7},
                                {26, 0, 9}, {27, 0, 8}, {30, 1, 9}, {31, 1, 8}};
// lattice columns under 31 steps of 32 quarts (x 337/331 on side B): the span in whole cells, one more and the far corner
constexpr int lattice_width(int log2f) { return int(31 * 32 * 337.0 / 331.0 / double(1 << log2f)) + 3; }
constexpr int lattice_base(int k) { int n = 0; for (int i = 0; i < k; i++) n += lattice_width(kPO[i].log2f) * lattice_width(kPO[i].log2f); return n; }
constexpr int PPTS = lattice_base(POCT), PPTS_T = lattice_base(4);
template <int K> struct TileLattice { static constexpr int oct = kPO[K].oct, side = kPO[K].side, width = lattice_width(kPO[K].log2f), base = lattice_base(K); };
static_assert(lattice_width(10) == 3 && lattice_width(9) == 4 && lattice_width(8) == 6 && lattice_width(7) == 10 && PPTS == 498, "tile lattice");
struct TileOct { double ox, oz, freq, s, fy, vy, amp; int32_t iy, width, base, pad; };
struct __align__(16) ProxyTile {
    LatticePoint pt[PPTS];
    double2 line[2][POCT][PT];                            // [x, z]: (fraction, fade) of each column or row
    TileOct oct[POCT];
    alignas(16) uint8_t perm[POCT][256];
    alignas(4) uint8_t at[2][POCT][PT];                   // its lattice column, counted from the tile's first
    double factor[3];
};
static_assert(sizeof(ProxyTile) <= 48 * 1024, "static shared memory");
// Position of column or row c of the tile whose first lies at x0 (the argument of the octave's floor).
__device__ __forceinline__ double tile_pos(const TileOct &o, int axis, int x0, int c) { return double(x0 + 32 * c) * o.s * o.freq + (axis ? o.oz : o.ox); }
// Octaves k0 .. k1 - 1 of the tile at (x0, z0), of mx x mz cells (columns beyond repeat the last).
__device__ __forceinline__ void tile_build(ProxyTile &T, const uint2 *__restrict__ grad, int k0, int k1, int p0, int p1, int x0, int z0, int mx, int mz) {
    for (int t = threadIdx.x; t < (k1 - k0) * 2 * PT; t += 256) {
        const int c = t % PT, axis = t / PT & 1, k = k0 + t / (2 * PT);
        const TileOct &o = T.oct[k];
        const int first = axis ? z0 : x0;
        const double v = tile_pos(o, axis, first, min(c, (axis ? mz : mx) - 1)), b = floor(v), f = v - b;
        T.line[axis][k][c] = make_double2(f, fade_d(f));
        T.at[axis][k][c] = uint8_t(int(b - floor(tile_pos(o, axis, first, 0))));
    }
    for (int t = p0 + threadIdx.x; t < p1; t += 256) {
        int k = k0;
        while (k + 1 < k1 && t >= T.oct[k + 1].base) k++;
        const TileOct &o = T.oct[k];
        const int j = t - o.base, ix = (int(floor(tile_pos(o, 0, x0, 0))) + j % o.width) & 255, iz = (int(floor(tile_pos(o, 1, z0, 0))) + j / o.width) & 255;
        const uint8_t *P = T.perm[k];
        const int a = P[ix] + o.iy, h0 = P[(P[a & 255] + iz) & 255], h1 = P[(P[(a + 1) & 255] + iz) & 255];
        T.pt[t] = {grad_d(grad, h0, 1., 0., 0.), grad_d(grad, h0, 0., 0., 1.), grad_d(grad, h0, 0., o.fy, 0.),
                   grad_d(grad, h1, 1., 0., 0.), grad_d(grad, h1, 0., 0., 1.), grad_d(grad, h1, 0., o.fy - 1, 0.)};
    }
}
// Sums of octaves k0 .. k1 - 1, amp x perlin(x, 0, z) each, at column cx of the four rows r0 .. r0 + 3 (r0 the same for the
// whole warp).  Where the four rows lie in one row of lattice cells, which at these frequencies is the usual case,
// its corners are loaded once and their x terms are shared: corner = gz z + (gx x + gy dy), the inner sum per column,
// the outer per cell.  (Of the three components one is zero, so one of the two sums is exact or adds a zero, and the
// value is u + v rounded once, whichever of x and z goes first.)
struct Sum4 { double v[4]; };
__device__ __noinline__ Sum4 tile_rows(const ProxyTile &T, int k0, int k1, int cx, int r0) {
    Sum4 s{{0, 0, 0, 0}};
    #pragma unroll 1
    for (int k = k0; k < k1; k++) {
        const TileOct &o = T.oct[k];
        const int W = o.width;
        const double2 x = T.line[0][k][cx];
        const double ty = o.vy, tx = x.y, amp = o.amp, ex = x.x - 1;
        const LatticePoint *col = &T.pt[o.base + int(T.at[0][k][cx])];
        const uint32_t lz = *reinterpret_cast<const uint32_t *>(&T.at[1][k][r0]);      // the four rows' lattice rows
        const double2 *z = &T.line[1][k][r0];
        double lo[4], hi[4];
        #pragma unroll
        for (int h = 0; h < 2; h++) {                     // the lattice row below the cells, then the one above
            double (&v)[4] = h ? hi : lo;
            const LatticePoint *a = col + ((lz & 255) + h) * W, *b = a + 1;
            if ((lz & 255) == lz >> 24) {
                const double A0 = fma(a->gx0, x.x, a->c0), A1 = fma(b->gx0, ex, b->c0), A2 = fma(a->gx1, x.x, a->c1), A3 = fma(b->gx1, ex, b->c1);
                const double g0 = a->gz0, g1 = b->gz0, g2 = a->gz1, g3 = b->gz1;
                #pragma unroll
                for (int q = 0; q < 4; q++) {
                    const double dz = h ? z[q].x - 1 : z[q].x;
                    v[q] = lerp_d(ty, lerp_d(tx, fma(g0, dz, A0), fma(g1, dz, A1)), lerp_d(tx, fma(g2, dz, A2), fma(g3, dz, A3)));
                }
            } else {
                #pragma unroll
                for (int q = 0; q < 4; q++) {
                    const LatticePoint *c = col + ((lz >> (8 * q) & 255) + h) * W, *d = c + 1;
                    const double dz = h ? z[q].x - 1 : z[q].x;
                    v[q] = lerp_d(ty, lerp_d(tx, fma(c->gz0, dz, fma(c->gx0, x.x, c->c0)), fma(d->gz0, dz, fma(d->gx0, ex, d->c0))),
                                      lerp_d(tx, fma(c->gz1, dz, fma(c->gx1, x.x, c->c1)), fma(d->gz1, dz, fma(d->gx1, ex, d->c1))));
                }
            }
        }
        #pragma unroll
        for (int q = 0; q < 4; q++) s.v[q] += amp * lerp_d(z[q].y, lo[q], hi[q]);
    }
    return s;
}
__global__ void __launch_bounds__(256, DSG_PROXY_MINB) k_proxy(const SeedNoise *__restrict__ noise, const DZone *__restrict__ zones, WorldDev w, float cut,
                                               uint8_t *__restrict__ out, ZoneWork wk) {
    __shared__ ProxyTile T;
    int staged = -1;
    each_chunk(zones, wk, [&](uint32_t, const DZone &z, int64_t c0, int64_t c1) {
        const SeedNoise &S = noise[z.seed];
        if (!zones::tiled(z)) {                           // cell by cell, coordinates modulo 2^32
            for (int64_t c = c0 + threadIdx.x; c < c1; c += blockDim.x)
                out[z.off + c] = proxy_prob(S, w, int(uint32_t(z.x0) + 32u * uint32_t(c % z.nx)), int(uint32_t(z.z0) + 32u * uint32_t(c / z.nx))) >= cut;
            return;
        }
        if (z.seed != staged) {                           // block-uniform: every thread walks the same chunks
            __syncthreads();
            if (threadIdx.x < POCT) {
                const int k = threadIdx.x;
                int oi = 0, side = 0, width = 0, base = 0;
                [&]<int... K>(std::integer_sequence<int, K...>) {
                    ((K == k ? void((oi = TileLattice<K>::oct, side = TileLattice<K>::side, width = TileLattice<K>::width, base = TileLattice<K>::base)) : void()), ...);
                }(std::make_integer_sequence<int, POCT>{});
                const NOct &o = S.oct[oi];
                T.oct[k] = {o.ox, o.oz, o.freq, side ? 337. / 331. : 1., o.fy, o.vy, o.amp, o.iy, width, base, 0};
            }
            if (threadIdx.x < 3) T.factor[threadIdx.x] = S.factor[threadIdx.x == 0 ? CH_T : threadIdx.x == 1 ? CH_C : CH_E];
            if (threadIdx.x < POCT * 16) {
                const int k = threadIdx.x >> 4;
                int oi = 0;
                [&]<int... K>(std::integer_sequence<int, K...>) { ((K == k ? void(oi = TileLattice<K>::oct) : void()), ...); }(std::make_integer_sequence<int, POCT>{});
                reinterpret_cast<uint4 *>(T.perm[k])[threadIdx.x & 15] = __ldg(reinterpret_cast<const uint4 *>(S.perm[oi]) + (threadIdx.x & 15));
            }
            staged = z.seed;
        }
        // the zone's tiles, dealt to its chunks in turn
        const int64_t nch = (int64_t(z.nx) * z.nz + CHUNK - 1) / CHUNK;
        const int tx = (z.nx + PT - 1) / PT, tz = (z.nz + PT - 1) / PT;
        for (int64_t t = c0 / CHUNK; t < int64_t(tx) * tz; t += nch) {
            const int i0 = int(t % tx) * PT, j0 = int(t / tx) * PT, mx = min(PT, z.nx - i0), mz = min(PT, z.nz - j0);
            const int x0 = z.x0 + 32 * i0, z0 = z.z0 + 32 * j0;
            __syncthreads();                              // the previous tile is done, the octaves are in place
            tile_build(T, S.grad, 0, 4, 0, PPTS_T, x0, z0, mx, mz);
            __syncthreads();
            const int cx = threadIdx.x & 31, r0 = 4 * (threadIdx.x >> 5);       // a warp has four rows
            const unsigned rows = r0 < mz ? (1u << min(4, mz - r0)) - 1 : 0;
            unsigned hot = 0;                             // bit q: the cell in row r0 + q
            {
                const Sum4 a = tile_rows(T, 0, 2, cx, r0), b = tile_rows(T, 2, 4, cx, r0);
                #pragma unroll
                for (int q = 0; q < 4; q++) if (cx < mx && (rows >> q & 1) && !((a.v[q] + b.v[q]) * T.factor[0] < 0.55)) hot |= 1u << q;
            }
            if (__syncthreads_or(hot)) {
                tile_build(T, S.grad, 4, POCT, PPTS_T, PPTS, x0, z0, mx, mz);
                __syncthreads();
            }
            Sum4 c{{0, 0, 0, 0}}, e{{0, 0, 0, 0}};
            if (__any_sync(0xffffffffu, hot)) { c = tile_rows(T, 4, 10, cx, r0); e = tile_rows(T, 10, POCT, cx, r0); }
            #pragma unroll
            for (int q = 0; q < 4; q++)
                if (cx < mx && (rows >> q & 1)) {
                    const float prob = (hot >> q & 1) ? proxy_bin(w, c.v[q] * T.factor[1], e.v[q] * T.factor[2]) : 0.f;
                    out[z.off + int64_t(j0 + r0 + q) * z.nx + i0 + cx] = prob >= cut;
                }
        }
    });
}

// ---- component labelling of the bitmaps (the 8-connected components, centroids and interior starts of
// dsearch_desert.cpp:451-490).  Union-find over zone-local cell indices; a union links the larger root to
// the smaller one, so every component's root is its first cell in raster order, the order in which the
// reference's scan meets it.  Loops on the parent links stop after kLinkLimit steps and raise the error flag.
constexpr uint32_t kLinkLimit = 1u << 24;
// Root of x, shortening the path on the way (each visited node is pointed two levels up); parents are
// always smaller indices, so the stored value is still an ancestor whatever other threads do meanwhile.
__device__ __forceinline__ int32_t uf_find(int32_t *par, int32_t x, uint32_t *err) {
    int32_t cur = __ldcg(par + x);
    if (cur == x) return x;
    int32_t prev = x;
    for (uint32_t it = 0; it < kLinkLimit; it++) {
        const int32_t next = __ldcg(par + cur);
        if (next == cur) return cur;
        __stcg(par + prev, next);
        prev = cur; cur = next;
    }
    atomicOr(err, 1u);
    return cur;
}
__device__ __forceinline__ void uf_union(int32_t *par, int32_t a, int32_t b, uint32_t *err) {
    for (uint32_t it = 0; it < kLinkLimit; it++) {
        a = uf_find(par, a, err); b = uf_find(par, b, err);
        if (a == b) return;
        if (a < b) { const int32_t t = a; a = b; b = t; }
        const int32_t old = atomicCAS(par + a, a, b);
        if (old == a) return;
        a = old;
    }
    atomicOr(err, 1u);
}
__device__ __forceinline__ bool zone_bit(const uint8_t *b, const DZone &z, int x, int y) {
    return x >= 0 && y >= 0 && x < z.nx && y < z.nz && b[int64_t(y) * z.nx + x];
}
// All 8 neighbours set and the cell not on the zone's edge (the reference's interior test, :469-473).
__device__ __forceinline__ bool interior(const uint8_t *b, const DZone &z, int x, int y) {
    if (x <= 0 || y <= 0 || x >= z.nx - 1 || y >= z.nz - 1) return false;
    for (int dy = -1; dy <= 1; dy++)
        for (int dx = -1; dx <= 1; dx++) if (!b[int64_t(y + dy) * z.nx + x + dx]) return false;
    return true;
}
// Union-find inside one chunk, in shared memory (local indices; same rules as uf_find / uf_union).
__device__ __forceinline__ int lc_find(volatile int32_t *sp, int x) {
    for (;;) {
        const int p = sp[x];
        if (p == x) return x;
        const int g = sp[p];
        sp[x] = g;                                       // x is no root: its parent may move up to an ancestor
        x = g;
    }
}
__device__ __forceinline__ void lc_union(volatile int32_t *sp, int a, int b, uint32_t *err) {
    for (uint32_t it = 0; it < kLinkLimit; it++) {
        a = lc_find(sp, a); b = lc_find(sp, b);
        if (a == b) return;
        if (a < b) { const int t = a; a = b; b = t; }
        const int old = atomicCAS(const_cast<int32_t *>(sp) + a, a, b);
        if (old == a) return;
        a = old;
    }
    atomicOr(err, 1u);
}
// Per chunk: the union-find of the 8-connected pairs inside the chunk, in shared memory; every cell's parent
// in `par` becomes its chunk-local root (zone-local index), -1 for a clear cell.  Pairs reaching an earlier
// chunk are joined by k_cc_cross.  Each local root is its set's smallest index, as the global rule wants.
__global__ void __launch_bounds__(256) k_cc_local(const DZone *__restrict__ zones, const uint8_t *__restrict__ bits, int32_t *__restrict__ par,
                                                  uint32_t *err, ZoneWork wk) {
    __shared__ int32_t sp_mem[CHUNK];
    volatile int32_t *sp = sp_mem;
    each_chunk(zones, wk, [&](uint32_t, const DZone &z, int64_t c0, int64_t c1) {
        const uint8_t *b = bits + z.off;
        const int n = int(c1 - c0);
        __syncthreads();                                 // the previous chunk is done with sp
        for (int i = threadIdx.x; i < n; i += blockDim.x) sp[i] = b[c0 + i] ? i : -1;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            if (!b[c0 + i]) continue;
            const int64_t c = c0 + i;
            const int x = int(c % z.nx), y = int(c / z.nx);
            // the four neighbours that come earlier in raster order cover every 8-connected pair once
            const int64_t nb[4] = {c - 1, c - z.nx - 1, c - z.nx, c - z.nx + 1};
            const bool ok[4] = {zone_bit(b, z, x - 1, y), zone_bit(b, z, x - 1, y - 1), zone_bit(b, z, x, y - 1), zone_bit(b, z, x + 1, y - 1)};
            #pragma unroll
            for (int k = 0; k < 4; k++)
                if (ok[k] && nb[k] >= c0) lc_union(sp, i, int(nb[k] - c0), err);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            par[z.off + c0 + i] = b[c0 + i] ? int32_t(c0 + lc_find(sp, i)) : -1;
    });
}
// Pairs whose earlier cell lies in an earlier chunk (the chunk's first row and one cell), joined globally.
__global__ void __launch_bounds__(256) k_cc_cross(const DZone *__restrict__ zones, const uint8_t *__restrict__ bits, int32_t *__restrict__ par,
                                                  uint32_t *err, ZoneWork wk) {
    each_chunk(zones, wk, [&](uint32_t, const DZone &z, int64_t c0, int64_t c1) {
        const uint8_t *b = bits + z.off;
        int32_t *p = par + z.off;
        const int64_t e = min(c1, c0 + z.nx + 2);
        for (int64_t c = c0 + threadIdx.x; c < e; c += blockDim.x) {
            if (!b[c]) continue;
            const int x = int(c % z.nx), y = int(c / z.nx);
            const int64_t nb[4] = {c - 1, c - z.nx - 1, c - z.nx, c - z.nx + 1};
            const bool ok[4] = {zone_bit(b, z, x - 1, y), zone_bit(b, z, x - 1, y - 1), zone_bit(b, z, x, y - 1), zone_bit(b, z, x + 1, y - 1)};
            #pragma unroll
            for (int k = 0; k < 4; k++)
                if (ok[k] && nb[k] < c0) uf_union(p, int32_t(c), int32_t(nb[k]), err);
        }
    });
}
// Roots get a component id; every cell's parent becomes its root.
__global__ void __launch_bounds__(256) k_cc_roots(const DZone *__restrict__ zones, int32_t *__restrict__ par, int32_t *__restrict__ rid,
                                                  CompStat *__restrict__ cs, uint32_t *ctr, ZoneWork wk, uint32_t comp_cap) {
    each_chunk(zones, wk, [&](uint32_t zi, const DZone &z, int64_t c0, int64_t c1) {
        int32_t *p = par + z.off;
        for (int64_t c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
            if (p[c] < 0) continue;
            const int32_t r = uf_find(p, int32_t(c), ctr + 3);
            if (r == int32_t(c)) {
                const uint32_t id = atomicAdd(ctr, 1u);
                if (id >= comp_cap) { rid[z.off + c] = -1; atomicOr(ctr + 3, 2u); continue; }   // out of component records
                rid[z.off + c] = int32_t(id);
                CompStat &q = cs[id];
                q.zone = zi; q.first = uint32_t(c); q.cells = 0; q.inner = 0; q.minx = q.minz = 0x7fffffff; q.kid = -1;
                q.seg = 0; q.cur = 0; q.sx = 0; q.sz = 0;
            }
        }
    });
}
__global__ void __launch_bounds__(256) k_cc_flatten(const DZone *__restrict__ zones, int32_t *__restrict__ par, uint32_t *err, ZoneWork wk) {
    each_chunk(zones, wk, [&](uint32_t, const DZone &z, int64_t c0, int64_t c1) {
        int32_t *p = par + z.off;
        for (int64_t c = c0 + threadIdx.x; c < c1; c += blockDim.x)
            if (p[c] >= 0) p[c] = uf_find(p, int32_t(c), err);
    });
}
__global__ void __launch_bounds__(256) k_cc_stats(const DZone *__restrict__ zones, const uint8_t *__restrict__ bits, const int32_t *__restrict__ par,
                                                  const int32_t *__restrict__ rid, CompStat *__restrict__ cs, ZoneWork wk) {
    each_chunk(zones, wk, [&](uint32_t, const DZone &z, int64_t c0, int64_t c1) {
        const uint8_t *b = bits + z.off;
        for (int64_t c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
            const int32_t r = par[z.off + c];
            if (r < 0 || rid[z.off + r] < 0) continue;
            CompStat &q = cs[rid[z.off + r]];
            const int x = int(c % z.nx), y = int(c / z.nx);
            atomicAdd(&q.cells, 1u);
            atomicMin(&q.minx, x); atomicMin(&q.minz, y);
            atomicAdd(reinterpret_cast<unsigned long long *>(&q.sx), (unsigned long long)x);
            atomicAdd(reinterpret_cast<unsigned long long *>(&q.sz), (unsigned long long)y);
            if (interior(b, z, x, y)) atomicAdd(&q.inner, 1u);
        }
    });
}
// Components of at least min_cells cells are kept; each gets a segment for its interior keys.
__global__ void k_cc_keep(CompStat *__restrict__ cs, uint32_t min_cells, uint32_t *ctr, uint32_t comp_cap) {
    const uint32_t n = min(*ctr, comp_cap);
    for (uint32_t id = blockIdx.x * blockDim.x + threadIdx.x; id < n; id += gridDim.x * blockDim.x) {
        CompStat &q = cs[id];
        if (q.cells < min_cells) continue;
        q.kid = int32_t(atomicAdd(ctr + 1, 1u));
        q.seg = atomicAdd(ctr + 2, q.inner);
    }
}
// Interior cells of kept components as 96-bit keys (squared distance to the centroid, raster index), the
// order of the reference's sorted `inner` list; the arithmetic is the host's, operation by operation.
__global__ void __launch_bounds__(256) k_cc_keys(const DZone *__restrict__ zones, const uint8_t *__restrict__ bits, const int32_t *__restrict__ par,
                                                 const int32_t *__restrict__ rid, CompStat *__restrict__ cs, uint64_t *__restrict__ khi,
                                                 uint32_t *__restrict__ klo, ZoneWork wk) {
    each_chunk(zones, wk, [&](uint32_t, const DZone &z, int64_t c0, int64_t c1) {
        const uint8_t *b = bits + z.off;
        for (int64_t c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
            const int32_t r = par[z.off + c];
            if (r < 0 || rid[z.off + r] < 0) continue;
            CompStat &q = cs[rid[z.off + r]];
            if (q.kid < 0) continue;
            const int x = int(c % z.nx), y = int(c / z.nx);
            if (!interior(b, z, x, y)) continue;
            const double cx = double(q.sx) / double(q.cells), cz = double(q.sz) / double(q.cells);
            const double d = __dadd_rn(__dmul_rn(x - cx, x - cx), __dmul_rn(y - cz, y - cz));
            const uint32_t at = q.seg + atomicAdd(&q.cur, 1u);
            khi[at] = uint64_t(__double_as_longlong(d));       // d >= 0: the bit pattern orders like the value
            klo[at] = uint32_t(c);
        }
    });
}
// One block per kept component: the interior keys at ranks 0, n/3 and 2n/3.  The keys are unique (the raster
// index is part of them), so a key's rank is the number of smaller keys: up to SEL_DIRECT keys, each thread
// counts for its key over a shared-memory copy; above that, an exact radix selection over the 12 bytes of the
// key (all three ranks in each pass), warp k finding rank k's digit by a prefix sum over the histogram.
constexpr uint32_t SEL_DIRECT = 256;
__global__ void __launch_bounds__(256) k_cc_select(const CompStat *__restrict__ cs, const uint64_t *__restrict__ khi, const uint32_t *__restrict__ klo,
                                                   const uint32_t *ctr, dsg_component *__restrict__ rec, uint32_t comp_cap) {
    __shared__ uint32_t hist[3][256];
    __shared__ uint64_t pre_hi[3], s_kh[SEL_DIRECT];
    __shared__ uint32_t pre_lo[3], want[3], s_kl[SEL_DIRECT];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t ncomp = min(ctr[0], comp_cap);
    for (uint32_t id = blockIdx.x; id < ncomp; id += gridDim.x) {
        const CompStat q = cs[id];
        if (q.kid < 0) continue;
        dsg_component &o = rec[q.kid];
        const uint32_t n = q.inner;
        const uint32_t w0 = 0, w1 = n / 3, w2 = 2 * (n / 3) + ((2 * (n % 3)) / 3);     // floor(2n/3)
        if (threadIdx.x == 0) {
            o.zone = q.zone; o.first = int32_t(q.first); o.cells = q.cells; o.minx = q.minx; o.minz = q.minz; o.inner = n;
            for (int k = 0; k < 3; k++) { o.pick[k] = -1; pre_hi[k] = 0; pre_lo[k] = 0; }
            want[0] = w0; want[1] = w1; want[2] = w2;
        }
        __syncthreads();
        if (n == 0) { __syncthreads(); continue; }
        const uint64_t *kh = khi + q.seg;
        const uint32_t *kl = klo + q.seg;
        if (n <= SEL_DIRECT) {
            const uint32_t i = threadIdx.x;
            if (i < n) { s_kh[i] = kh[i]; s_kl[i] = kl[i]; }
            __syncthreads();
            if (i < n) {
                const uint64_t h = s_kh[i];
                const uint32_t l = s_kl[i];
                uint32_t r = 0;
                for (uint32_t j = 0; j < n; j++) r += (s_kh[j] < h) || (s_kh[j] == h && s_kl[j] < l);
                if (r == w0) o.pick[0] = int32_t(l);
                if (r == w1) o.pick[1] = int32_t(l);
                if (r == w2) o.pick[2] = int32_t(l);
            }
            __syncthreads();
            continue;
        }
        for (int d = 11; d >= 0; d--) {
            for (int i = threadIdx.x; i < 3 * 256; i += blockDim.x) (&hist[0][0])[i] = 0;
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
                const uint64_t h = kh[i];
                const uint32_t l = kl[i];
                const uint32_t dig = d >= 4 ? uint32_t(h >> (8 * (d - 4))) & 255u : (l >> (8 * d)) & 255u;
                #pragma unroll
                for (int k = 0; k < 3; k++) {
                    bool match;
                    if (d >= 4) match = d == 11 || (h >> (8 * (d - 4) + 8)) == (pre_hi[k] >> (8 * (d - 4) + 8));
                    else match = h == pre_hi[k] && (d == 3 || (l >> (8 * d + 8)) == (pre_lo[k] >> (8 * d + 8)));
                    if (match) atomicAdd(&hist[k][dig], 1u);
                }
            }
            __syncthreads();
            if (warp < 3) {                                     // the first digit whose cumulative count passes want
                const int k = warp;
                uint32_t c[8], sum = 0;
                #pragma unroll
                for (int j = 0; j < 8; j++) { c[j] = hist[k][lane * 8 + j]; sum += c[j]; }
                uint32_t incl = sum;
                #pragma unroll
                for (int o2 = 1; o2 < 32; o2 <<= 1) { const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o2); if (lane >= o2) incl += t; }
                const uint32_t wk = want[k], excl = incl - sum;
                const bool here = excl <= wk && wk < incl;          // the lane holding the digit (one lane at most)
                const uint32_t owner = __ballot_sync(0xffffffffu, here);
                // no lane holds it only if want >= the count (cannot happen); digit 255 then, as the scan would give
                const int src = owner ? __ffs(owner) - 1 : 31;
                uint32_t b = 255, below = 0;
                if (lane == src) {
                    uint32_t acc = excl;
                    b = uint32_t(lane * 8 + 7);
                    for (int j = 0; j < 8; j++) {
                        if (j == 7 || acc + c[j] > wk) { b = uint32_t(lane * 8 + j); break; }
                        acc += c[j];
                    }
                    below = acc;
                }
                b = __shfl_sync(0xffffffffu, b, src);
                below = __shfl_sync(0xffffffffu, below, src);
                if (lane == 0) {
                    want[k] = wk - below;
                    if (d >= 4) pre_hi[k] |= uint64_t(b) << (8 * (d - 4));
                    else pre_lo[k] |= b << (8 * d);
                }
            }
            __syncthreads();
        }
        if (threadIdx.x == 0)
            for (int k = 0; k < 3; k++) o.pick[k] = int32_t(pre_lo[k]);
        __syncthreads();
    }
}

// Component labelling of bitmaps already in `bits` (k_proxy's output): union-find, statistics, kept components
// (at least min_cells cells), interior keys and the three interior starts of each kept component into rec[kid].
// ctr = {components, kept, interior keys, error}, zeroed by the caller.
// comp_cap: records in cs and rec; more components raise bit 1 of the error flag (their cells are left out).
void label_components(const DZone *zones, dim3 grid, const ZoneWork &wk, const uint8_t *bits, int32_t *par, int32_t *rid, CompStat *cs,
                      uint64_t *khi, uint32_t *klo, dsg_component *rec, uint32_t *ctr, uint32_t min_cells, unsigned keep_blocks,
                      unsigned select_blocks, uint32_t comp_cap, cudaStream_t st) {
    k_cc_local<<<grid, 256, 0, st>>>(zones, bits, par, ctr + 3, wk);
    k_cc_cross<<<grid, 256, 0, st>>>(zones, bits, par, ctr + 3, wk);
    k_cc_roots<<<grid, 256, 0, st>>>(zones, par, rid, cs, ctr, wk, comp_cap);
    k_cc_flatten<<<grid, 256, 0, st>>>(zones, par, ctr + 3, wk);
    k_cc_stats<<<grid, 256, 0, st>>>(zones, bits, par, rid, cs, wk);
    k_cc_keep<<<(keep_blocks + 255) / 256, 256, 0, st>>>(cs, min_cells, ctr, comp_cap);
    k_cc_keys<<<grid, 256, 0, st>>>(zones, bits, par, rid, cs, khi, klo, wk);
    k_cc_select<<<select_blocks, 256, 0, st>>>(cs, khi, klo, ctr, rec, comp_cap);
}

struct State {
    std::mutex mu;
    cudaStream_t st = nullptr;
    SeedNoise *d_noise = nullptr; size_t seed_cap = 0;
    uint64_t *d_seeds = nullptr; size_t seeds_cap = 0;
    DZone *d_zones = nullptr; size_t zone_cap = 0;
    uint8_t *d_out = nullptr; size_t out_cap = 0;
    // component labelling (dsg_proxy_components): per cell, per component, per interior key; counters
    int32_t *d_par = nullptr, *d_rid = nullptr; size_t par_cap = 0, rid_cap = 0;
    CompStat *d_cs = nullptr; size_t cs_cap = 0;
    uint64_t *d_khi = nullptr; uint32_t *d_klo = nullptr; size_t khi_cap = 0, klo_cap = 0;
    dsg_component *d_rec = nullptr; size_t rec_cap = 0;
    uint32_t *d_ctr = nullptr, *h_ctr = nullptr;   // [0] components [1] kept [2] interior keys [3] error
};
State &S() { static State s; return s; }
template <class T> void grow(T *&p, size_t &cap, size_t need) {
    if (need <= cap) return;
    cudaFree(p); p = nullptr;
    const size_t c = std::max(need, cap * 2);
    DSG_CU(cudaMalloc(&p, c * sizeof(T)));
    cap = c;
}
}  // namespace

void proxy_set_cut(float cut) { g_cut = cut; }

int proxy_eval(const uint64_t *seeds, uint32_t nseeds, const uint32_t *zone_seed, const dsg_zone *zones, uint32_t nzones, uint8_t *bits) {
    State &g = S();
    std::lock_guard<std::mutex> l(g.mu);
    require_init();
    if (!g.st) {
        int lo, hi;
        DSG_CU(cudaDeviceGetStreamPriorityRange(&lo, &hi));
        DSG_CU(cudaStreamCreateWithPriority(&g.st, cudaStreamNonBlocking, hi));
    }
    std::vector<DZone> dz(nzones);
    int64_t off = 0, maxc = 0;
    for (uint32_t k = 0; k < nzones; k++) {
        const dsg_zone &z = zones[k];
        DSG_ARG(z.nx >= 0 && z.nz >= 0, "dsg_proxy: negative zone size");
        DSG_ARG(!zone_seed || zone_seed[k] < nseeds, "dsg_proxy: zone seed index out of range");
        dz[k] = {z.x0, z.z0, z.nx, z.nz, off, int32_t(zone_seed ? zone_seed[k] : 0), 0};
        off += int64_t(z.nx) * z.nz;
        maxc = std::max(maxc, int64_t(z.nx) * z.nz);
    }
    if (!off) return DSG_OK;
    DSG_ARG(maxc / CHUNK < 65535, "dsg_proxy: zone too large");
    grow(g.d_noise, g.seed_cap, nseeds);
    grow(g.d_seeds, g.seeds_cap, nseeds);
    grow(g.d_zones, g.zone_cap, nzones);
    grow(g.d_out, g.out_cap, size_t(off));
    DSG_CU(cudaMemcpyAsync(g.d_seeds, seeds, size_t(nseeds) * 8, cudaMemcpyHostToDevice, g.st));
    seed_noise_build(g.d_seeds, nseeds, g.d_noise, g.st);
    DSG_CU(cudaMemcpyAsync(g.d_zones, dz.data(), dz.size() * sizeof(DZone), cudaMemcpyHostToDevice, g.st));
    k_proxy<<<dim3(nzones, unsigned((maxc + CHUNK - 1) / CHUNK)), 256, 0, g.st>>>(g.d_noise, g.d_zones, world_dev(), g_cut, g.d_out, ZoneWork{});
    DSG_CU(cudaGetLastError());
    DSG_CU(cudaMemcpyAsync(bits, g.d_out, size_t(off), cudaMemcpyDeviceToHost, g.st));
    DSG_CU(cudaStreamSynchronize(g.st));
    return DSG_OK;
}

// Proxy bitmaps and their components in one pass on the device; only the kept components come back.
int proxy_components(const uint64_t *seeds, uint32_t nseeds, const uint32_t *zone_seed, const dsg_zone *zones, uint32_t nzones,
                     uint32_t min_cells, dsg_component *out, uint32_t cap, uint32_t *n_out, uint8_t *bits) {
    State &g = S();
    std::lock_guard<std::mutex> l(g.mu);
    require_init();
    *n_out = 0;
    if (!g.st) {
        int lo, hi;
        DSG_CU(cudaDeviceGetStreamPriorityRange(&lo, &hi));
        DSG_CU(cudaStreamCreateWithPriority(&g.st, cudaStreamNonBlocking, hi));
    }
    if (!g.d_ctr) {
        DSG_CU(cudaMalloc(&g.d_ctr, 4 * 4));
        DSG_CU(cudaMallocHost(&g.h_ctr, 4 * 4));
    }
    std::vector<DZone> dz(nzones);
    int64_t off = 0, maxc = 0;
    for (uint32_t k = 0; k < nzones; k++) {
        const dsg_zone &z = zones[k];
        DSG_ARG(z.nx >= 0 && z.nz >= 0, "dsg_proxy_components: negative zone size");
        DSG_ARG(int64_t(z.nx) * z.nz < (int64_t(1) << 31), "dsg_proxy_components: zone too large");
        DSG_ARG(zone_seed[k] < nseeds, "dsg_proxy_components: zone seed index out of range");
        dz[k] = {z.x0, z.z0, z.nx, z.nz, off, int32_t(zone_seed[k]), 0};
        off += int64_t(z.nx) * z.nz;
        maxc = std::max(maxc, int64_t(z.nx) * z.nz);
    }
    if (!off) return DSG_OK;
    DSG_ARG(maxc / CHUNK < 65535, "dsg_proxy_components: zone too large");
    grow(g.d_noise, g.seed_cap, nseeds);
    grow(g.d_seeds, g.seeds_cap, nseeds);
    grow(g.d_zones, g.zone_cap, nzones);
    grow(g.d_out, g.out_cap, size_t(off));
    grow(g.d_par, g.par_cap, size_t(off));
    grow(g.d_rid, g.rid_cap, size_t(off));
    grow(g.d_cs, g.cs_cap, size_t(off));             // at most one component per cell
    grow(g.d_khi, g.khi_cap, size_t(off));           // at most one interior key per cell
    grow(g.d_klo, g.klo_cap, size_t(off));
    grow(g.d_rec, g.rec_cap, size_t(off));
    cudaStream_t st = g.st;
    DSG_CU(cudaMemcpyAsync(g.d_seeds, seeds, size_t(nseeds) * 8, cudaMemcpyHostToDevice, st));
    seed_noise_build(g.d_seeds, nseeds, g.d_noise, st);
    DSG_CU(cudaMemcpyAsync(g.d_zones, dz.data(), dz.size() * sizeof(DZone), cudaMemcpyHostToDevice, st));
    DSG_CU(cudaMemsetAsync(g.d_ctr, 0, 4 * 4, st));
    const dim3 grid(nzones, unsigned((maxc + CHUNK - 1) / CHUNK));
    k_proxy<<<grid, 256, 0, st>>>(g.d_noise, g.d_zones, world_dev(), g_cut, g.d_out, ZoneWork{});
    label_components(g.d_zones, grid, ZoneWork{}, g.d_out, g.d_par, g.d_rid, g.d_cs, g.d_khi, g.d_klo, g.d_rec, g.d_ctr, min_cells,
                     unsigned(std::min<int64_t>(off, 1 << 20)), unsigned(std::min<int64_t>(off, 4 * 148)), uint32_t(std::min<int64_t>(off, 0x7fffffff)), st);
    DSG_CU(cudaGetLastError());
    if (bits) DSG_CU(cudaMemcpyAsync(bits, g.d_out, size_t(off), cudaMemcpyDeviceToHost, st));
    DSG_CU(cudaMemcpyAsync(g.h_ctr, g.d_ctr, 4 * 4, cudaMemcpyDeviceToHost, st));
    DSG_CU(cudaStreamSynchronize(st));
    if (g.h_ctr[3]) { set_error("dsg_proxy_components: component labelling did not converge"); return DSG_E_CUDA; }
    const uint32_t kept = g.h_ctr[1];
    *n_out = kept;
    std::vector<dsg_component> rec(kept);
    if (kept) {
        DSG_CU(cudaMemcpyAsync(rec.data(), g.d_rec, size_t(kept) * sizeof(dsg_component), cudaMemcpyDeviceToHost, st));
        DSG_CU(cudaStreamSynchronize(st));
    }
    std::sort(rec.begin(), rec.end(), [](const dsg_component &a, const dsg_component &b) { return a.zone != b.zone ? a.zone < b.zone : a.first < b.first; });
    std::copy(rec.begin(), rec.begin() + std::min(kept, cap), out);
    return kept > cap ? DSG_OVERFLOW : DSG_OK;
}
// Proxy bitmaps and components of zones built on the device (the device-resident searcher): zones[0, *nzones)
// with their cell offsets, and the chunk list chunk[0, *nchunk) over them; buffers sized for the capacities by
// the caller (par, rid, cs, khi, klo, rec: one entry per cell).  Enqueued on st; ctr as label_components.
void proxy_components_device(const SeedNoise *noise, const zones::DZone *zones, const ZoneWork &wk, uint32_t grid_blocks, uint8_t *bits,
                             int32_t *par, int32_t *rid, CompStat *cs, uint64_t *khi, uint32_t *klo, dsg_component *rec, uint32_t *ctr,
                             uint32_t min_cells, uint32_t comp_cap, cudaStream_t st) {
    DSG_CU(cudaMemsetAsync(ctr, 0, 4 * 4, st));
    k_proxy<<<grid_blocks, 256, 0, st>>>(noise, zones, world_dev(), g_cut, bits, wk);
    label_components(zones, dim3(grid_blocks), wk, bits, par, rid, cs, khi, klo, rec, ctr, min_cells, 1u << 20, 4 * 148, comp_cap, st);
    DSG_CU(cudaGetLastError());
}
}  // namespace dsg

extern "C" int dsg_proxy_components(const uint64_t *seeds, uint32_t nseeds, const uint32_t *zone_seed, const dsg_zone *zones, uint32_t nzones,
                                    uint32_t min_cells, dsg_component *out, uint32_t cap, uint32_t *n_out, uint8_t *bits) {
    return dsg::guarded([&] {
        DSG_ARG(n_out && (nzones == 0 || (seeds && zone_seed && zones)) && (cap == 0 || out), "dsg_proxy_components: null pointer");
        return dsg::proxy_components(seeds, nseeds, zone_seed, zones, nzones, min_cells, out, cap, n_out, bits);
    });
}

extern "C" int dsg_proxy(uint64_t seed, const dsg_zone *zones, uint32_t nzones, uint8_t *bits) {
    return dsg::guarded([&] {
        DSG_ARG(nzones == 0 || (zones && bits), "dsg_proxy: null pointer");
        return dsg::proxy_eval(&seed, 1, nullptr, zones, nzones, bits);
    });
}
extern "C" int dsg_proxy_batch(const uint64_t *seeds, uint32_t nseeds, const uint32_t *zone_seed, const dsg_zone *zones, uint32_t nzones,
                               uint8_t *bits) {
    return dsg::guarded([&] {
        DSG_ARG(nzones == 0 || (seeds && zone_seed && zones && bits), "dsg_proxy_batch: null pointer");
        return dsg::proxy_eval(seeds, nseeds, zone_seed, zones, nzones, bits);
    });
}
