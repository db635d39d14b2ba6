// FP64 climate sampling on the device: per-seed octave tables, Perlin octaves, two-sided noise channels,
// the Y=256 desert flood state, the hot-zone and proxy predicates.  Restates src/standalone.hpp:38-152,
// src/surface.hpp:74-134 and src/desert_proxy.hpp:13-31 operation by operation; the library is compiled
// with -fmad=false, so every product and sum rounds exactly as the reference's CPU code (built with
// -ffp-contract=off) rounds it, and biome IDs and flood areas come out identical.
#pragma once
#include "common.cuh"
#include "world.cuh"

namespace dsg {

// Channel order of the reference: temperature, humidity, continentalness, erosion, shift, weirdness.
enum { CH_T = 0, CH_H = 1, CH_C = 2, CH_E = 3, CH_S = 4, CH_W = 5 };
constexpr int NOCT = 46;                     // nonzero octaves over all channels, both sides

struct __align__(16) NOct { double ox, oy, oz, freq, amp, fy, vy; int32_t iy, pad; };
// All noise of one seed: octave k of channel ch, side s is oct[off[ch] + s * cnt[ch] + k].  Each permutation
// is stored twice over (perm[k][i] = perm[k][i & 255] for i < 512), so a lattice index masked once can be
// offset by a hash and a corner step without masking again.
// grad[h] holds Minecraft's gradient h (components 0 or +-1, the same for every seed; kept with the seed so that
// it sits in shared memory wherever the octaves do) as the two upper bytes of each component's high word, the
// only nonzero bytes of +-1.0 and 0.0: bytes 1-2 for x, 3-4 for y, 5-6 for z, bytes 0 and 7 zero.
struct __align__(16) SeedNoise {
    NOct oct[NOCT];
    uint2 grad[16];
    uint8_t perm[NOCT][512];
    double factor[6];
    int32_t off[6], cnt[6];
};

#ifdef __CUDACC__
__device__ __forceinline__ double fade_d(double t) { return t * t * t * (t * (t * 6. - 15.) + 10.); }
__device__ __forceinline__ double lerp_d(double t, double a, double b) { return a + t * (b - a); }
// The reference's grad(h, x, y, z) (standalone.hpp:62-83) is u + v, u and v two of +-x, +-y, +-z picked by h.
// Here it is gx*x + gy*y + gz*z with the components from G = SeedNoise::grad: each product is exactly +-x, +-y,
// +-z or a zero, so the two fused multiply-adds round once, on u + v, and give the same double (a zero's sign
// aside; every sum of octaves starts from +0, which drops it).  One 8-byte shared load and three byte permutes
// rebuild the components; three FP64 instructions replace the integer selects and sign flips of u + v.
__device__ __forceinline__ double grad_d(const uint2 *__restrict__ G, int h, double x, double y, double z) {
    const uint2 g = G[h & 15];
    const double gx = __hiloint2double(int(__byte_perm(g.x, g.y, 0x2100)), 0);
    const double gy = __hiloint2double(int(__byte_perm(g.x, g.y, 0x4300)), 0);
    const double gz = __hiloint2double(int(__byte_perm(g.x, g.y, 0x6500)), 0);
    return fma(gx, x, fma(gy, y, gz * z));
}
// One Perlin octave (standalone.hpp:62-83); P is the doubled permutation of the octave, G the gradients.
__device__ __forceinline__ double perlin(const NOct &o, const uint8_t *__restrict__ P, const uint2 *__restrict__ G, double x, double y, double z) {
    x += o.ox; z += o.oz;
    const double bx = floor(x), bz = floor(z);
    const int ix = int(bx) & 255, iz = int(bz) & 255;
    x -= bx; z -= bz;
    int jy = o.iy; double dy = o.fy, ty = o.vy;
    if (y != 0) { y += o.oy; const double by = floor(y); jy = int(by) & 255; dy = y - by; ty = fade_d(dy); }
    const int a0 = P[ix], a1 = P[ix + 1];
    const int b00 = P[a0 + jy], b01 = P[a0 + jy + 1];
    const int b10 = P[a1 + jy], b11 = P[a1 + jy + 1];
    const double tx = fade_d(x), tz = fade_d(z);
    const double lo = lerp_d(ty, lerp_d(tx, grad_d(G, P[b00 + iz], x, dy, z), grad_d(G, P[b10 + iz], x - 1, dy, z)),
                                 lerp_d(tx, grad_d(G, P[b01 + iz], x, dy - 1, z), grad_d(G, P[b11 + iz], x - 1, dy - 1, z)));
    const double hi = lerp_d(ty, lerp_d(tx, grad_d(G, P[b00 + iz + 1], x, dy, z - 1), grad_d(G, P[b10 + iz + 1], x - 1, dy, z - 1)),
                                 lerp_d(tx, grad_d(G, P[b01 + iz + 1], x, dy - 1, z - 1), grad_d(G, P[b11 + iz + 1], x - 1, dy - 1, z - 1)));
    return lerp_d(tz, lo, hi);
}
// Two-sided channel value (standalone.hpp:140-151): per-side sums, side B at 337/331 scale.
__device__ __forceinline__ double channel(const SeedNoise &S, int ch, double x, double y, double z) {
    const int off = S.off[ch], cnt = S.cnt[ch];
    double a0 = 0, a1 = 0;
    for (int j = 0; j < cnt; j++) {
        const NOct &o = S.oct[off + j];
        a0 += o.amp * perlin(o, S.perm[off + j], S.grad, x * o.freq, y * o.freq, z * o.freq);
    }
    const double s = 337. / 331.;
    const double px = x * s, py = y * s, pz = z * s;
    for (int j = 0; j < cnt; j++) {
        const NOct &o = S.oct[off + cnt + j];
        a1 += o.amp * perlin(o, S.perm[off + cnt + j], S.grad, px * o.freq, py * o.freq, pz * o.freq);
    }
    return (a0 + a1) * S.factor[ch];
}
// Octaves [lo, hi) of both sides in one accumulator (desert_proxy.hpp:13-23).
__device__ __forceinline__ double channel_low(const SeedNoise &S, int ch, double x, double z, int lo, int hi) {
    const int off = S.off[ch], cnt = S.cnt[ch];
    double s = 0;
    for (int side = 0; side < 2; side++) {
        const double sc = side ? 337. / 331. : 1.;
        for (int k = lo; k < hi && k < cnt; k++) {
            const int i = off + side * cnt + k;
            const NOct &o = S.oct[i];
            s += o.amp * perlin(o, S.perm[i], S.grad, x * sc * o.freq, 0, z * sc * o.freq);
        }
    }
    return s * S.factor[ch];
}
__device__ __forceinline__ int32_t q10k(float v) { return int32_t(10000.f * v); }
__device__ __forceinline__ float ridge_fold(float wv) { return -(fabsf(fabsf(wv) - 0.6666667f) - 0.33333334f) * 3.f; }
__device__ __forceinline__ int32_t depth_of(float spline) {
    const double off = double(spline + 0.015f);
    return q10k(float(1. - (64 * 4) / 128. - 83. / 160. + off));
}
__device__ __forceinline__ int32_t depth_q(const WorldDev &w, float c, float e, float wv) {
    const float v[4] = {c, e, ridge_fold(wv), wv};
    return depth_of(spline_eval(w, v));
}
// Desert flood state at quart (x, 64, z) (surface.hpp:98-124): 2 desert, 1 river bridged to desert, 0 other.
// In two parts so callers can batch the points the surface grid cannot decide: desert_state_begin returns the
// state, or -1 with the climate `p` that desert_state_finish completes (exact depth, then the exact search).
struct PendingState { int32_t q[6]; float c, e, w; int32_t stage; };
__device__ __forceinline__ int desert_state_decide(const WorldDev &w, float t, float c, float e, float wv, float h, PendingState &p) {
    int32_t q[6] = {q10k(t), q10k(h), q10k(c), q10k(e), -10000, q10k(wv)};
    auto pend = [&](int stage) {
        for (int k = 0; k < 6; k++) p.q[k] = q[k];
        p.c = c; p.e = e; p.w = wv; p.stage = stage;
        return -1;
    };
    int b = grid_lookup(w, q);
    if (b < 0) return pend(1);                     // first pick needs the exact search
    if (b == 2) return 2;
    if (b != 7 && b != 11) return 0;
    if (q[5] > 500 || q[5] < -500) return 0;
    q[5] = q[5] >= 0 ? 501 : -501;
    b = grid_lookup(w, q);
    if (b < 0) return pend(2);                     // second pick (bridged river) needs it
    return b == 2 ? 1 : 0;
}
// The octaves of a channel's two sides follow one another in SeedNoise; the channel order is T H C E shift W.
constexpr int kChanOff[7] = {0, 4, 8, 26, 34, 40, 46};
constexpr uint64_t octave_sides() {                // bit i: octave i belongs to side B
    uint64_t m = 0;
    for (int c = 0; c < 6; c++) for (int i = (kChanOff[c] + kChanOff[c + 1]) / 2; i < kChanOff[c + 1]; i++) m |= uint64_t(1) << i;
    return m;
}
constexpr uint64_t kSideB = octave_sides();
// ---------------------------------------------------------------- lattice points of a patch, shared by its cells
// Most climate octaves vary slowly: the 16 x 16 cells of a sub-block lie within two lattice cells along each axis, so
// the hashes and gradients of the 3 x 3 lattice columns around them serve every cell.  The block works them out once:
// per octave the lattice cell of the patch's corner (bx, bz) and per lattice column the gradient terms of its two y
// corners, (gx, gz, gy * dy), dy = fy and fy - 1 (the climate channels are sampled at y = 0).  A cell then needs no
// hashing: per corner two multiply-adds, fma(gx, x, fma(gz, z, gy * dy)).  One of the three components is zero, so the
// inner one is exact or the outer adds a zero, and the value is the reference's u + v rounded once, as in grad_d.
struct __align__(16) LatticePoint { double gx0, gz0, c0, gx1, gz1, c1; };
// Octaves 0..33 and 40..45 of SeedNoise (T, H, C, E, W) but C's three fastest of either side (14-16, 23-25; frequencies 2^-3
// to 2^-1), whose lattice cells are smaller than any patch.
constexpr int kPatchOct = 34;
struct __align__(16) PatchCache { double bx[kPatchOct], bz[kPatchOct]; LatticePoint pt[kPatchOct][9]; };
__device__ __forceinline__ int patch_slot(int i) {          // -1: not kept
    return i < 14 ? i : i < 17 ? -1 : i < 23 ? i - 3 : i < 26 ? -1 : i < 34 ? i - 6 : i - 12;
}
__device__ __forceinline__ int patch_octave(int slot) { return slot + (slot < 14 ? 0 : slot < 20 ? 3 : slot < 28 ? 6 : 12); }
// The table of the patch [x0, x0 + ext] x [z0, z0 + ext] (quarts, the warped coordinates included) by `nt` threads.  An
// octave whose patch spans more than about a lattice cell is left out (bx infinite: no cell is found inside).  So is one whose
// corner lies in lattice cell -1 or -2 along either axis.  A point of such a patch may lie in (-1, 1) and its difference from
// the corner in [1, 2), where doubles are coarser than the point's own: the last bits of its fraction would be lost.
// Everywhere else the difference is exact: from 0 it is the point itself, from any other corner the point is at least 1 in
// magnitude, so both are multiples of 2^-52.  The two cells are next to the origin of the octave's own noise.
__device__ __forceinline__ void patch_build(const SeedNoise &S, PatchCache &C, double x0, double z0, double ext, int t, int nt) {
    for (int k = t; k < kPatchOct * 9; k += nt) {
        const int slot = k / 9, j = k % 9, i = patch_octave(slot);
        const NOct &o = S.oct[i];
        const uint8_t *P = S.perm[i];
        const double s = (kSideB >> i & 1) ? 337. / 331. : 1.;
        const double bx = floor(x0 * s * o.freq + o.ox), bz = floor(z0 * s * o.freq + o.oz);
        const bool use = ext * s * o.freq < 1.25 && (bx < -2 || bx >= 0) && (bz < -2 || bz >= 0);
        if (j == 0) { C.bx[slot] = use ? bx : __longlong_as_double(0x7ff0000000000000ll); C.bz[slot] = bz; }
        if (!use) continue;
        const int ix = (int(bx) + j % 3) & 255, iz = (int(bz) + j / 3) & 255, a = P[ix] + o.iy;
        const int h0 = P[P[a & 255] + iz], h1 = P[P[(a + 1) & 255] + iz];
        C.pt[slot][j] = {grad_d(S.grad, h0, 1., 0., 0.), grad_d(S.grad, h0, 0., 0., 1.), grad_d(S.grad, h0, 0., o.fy, 0.),
                         grad_d(S.grad, h1, 1., 0., 0.), grad_d(S.grad, h1, 0., 0., 1.), grad_d(S.grad, h1, 0., o.fy - 1, 0.)};
    }
}
// perlin(o, P, G, x, 0, z) of octave slot `k` (-1: none), from the patch's table where the point lies in it.
__device__ __forceinline__ double perlin_patch(const NOct &o, const uint8_t *__restrict__ P, const uint2 *__restrict__ G, const PatchCache &C, int k, double x,
                                               double z) {
    const int kept = max(k, 0);
    double fx = (x + o.ox) - C.bx[kept], fz = (z + o.oz) - C.bz[kept];
    // both in [0, 2): compared as integers (a negative number's sign bit is the largest)
    if (k < 0 || uint32_t(__double2hiint(fx)) >= 0x40000000u || uint32_t(__double2hiint(fz)) >= 0x40000000u) return perlin(o, P, G, x, 0, z);
    const bool cx = __double2hiint(fx) >= 0x3ff00000, cz = __double2hiint(fz) >= 0x3ff00000;
    fx -= cx ? 1. : 0.; fz -= cz ? 1. : 0.;        // the fractions x - floor(x), z - floor(z): exact for the corners patch_build keeps
    const LatticePoint *q = &C.pt[k][(cz ? 3 : 0) + (cx ? 1 : 0)];
    const double tx = fade_d(fx), tz = fade_d(fz), ty = o.vy, ex = fx - 1;
    const auto row = [&](const LatticePoint &a, const LatticePoint &b, double dz) {
        return lerp_d(ty, lerp_d(tx, fma(a.gx0, fx, fma(a.gz0, dz, a.c0)), fma(b.gx0, ex, fma(b.gz0, dz, b.c0))),
                          lerp_d(tx, fma(a.gx1, fx, fma(a.gz1, dz, a.c1)), fma(b.gx1, ex, fma(b.gz1, dz, b.c1))));
    };
    const double lo = row(q[0], q[1], fz);
    return lerp_d(tz, lo, row(q[3], q[4], fz - 1));
}
// channel(S, ch, x, 0, z) for T, H, C, E, W through the patch's table.
__device__ __forceinline__ double channel_patch(const SeedNoise &S, const PatchCache &C, int ch, double x, double z) {
    const int off = S.off[ch], cnt = S.cnt[ch];
    double a0 = 0, a1 = 0;
    #pragma unroll 1
    for (int i = off; i < off + cnt; i++) {
        const NOct &o = S.oct[i];
        a0 += o.amp * perlin_patch(o, S.perm[i], S.grad, C, patch_slot(i), x * o.freq, z * o.freq);
    }
    const double px = x * (337. / 331.), pz = z * (337. / 331.);
    #pragma unroll 1
    for (int i = off + cnt; i < off + 2 * cnt; i++) {
        const NOct &o = S.oct[i];
        a1 += o.amp * perlin_patch(o, S.perm[i], S.grad, C, patch_slot(i), px * o.freq, pz * o.freq);
    }
    return (a0 + a1) * S.factor[ch];
}
// ---------------------------------------------------------------- the shift octaves on a sub-block's grid
// The two shift samples are taken at the cells themselves, (x, 0, z) and (z, x, 0): what depends on x alone or z alone is
// worked out once per column or row of the 16 x 16 cells.  A cell then skips the floors, fades and (at (x, 0, z)) the
// column hashes of the 12 octaves; the values are perlin's, expression by expression.
// Measured: a batch of 288 uneven floods (292 M cells evaluated, 830 rounds) 153.2 -> 150.5 ms, a burst of 120 service
// requests 73.0 -> 71.5 ms.  About a tenth of the source's operations for 2%: latency holds these rounds, not issue.
struct __align__(16) ShiftLines {
    double2 cx[6][16], rz[6][16], rx[6][16];       // (fraction, fade): columns along the octave's x, rows along its z and its x
    double cy[6][16];                              // columns along the octave's y: the fraction
    double2 z0[6];                                 // z = 0: (fraction, fade)
    uint32_t ch[6][16];                            // columns: P[P[ix + dx] + iy + dy], byte 2 dx + dy
    int32_t iz0[6];
    uint16_t ra[6][16];                            // rows: P[ix] | P[ix + 1] << 8
    uint8_t rzi[6][16], cyi[6][16];                // lattice rows; columns along y
};
// By threads t < 198: columns and rows of the cells at (x0 + step i, z0 + step j), i, j < 16.
__device__ __forceinline__ void shift_build(const SeedNoise &S, ShiftLines &L, int x0, int z0, int step, int t) {
    if (t >= 198) return;
    const int k = t < 192 ? t / 16 % 6 : t - 192, l = t & 15, i = kChanOff[CH_S] + k;
    const NOct &o = S.oct[i];
    const uint8_t *P = S.perm[i];
    const double s = k >= 3 ? 337. / 331. : 1.;
    const auto split = [](double v, int &at) { const double b = floor(v); at = int(b) & 255; return v - b; };
    int at;
    if (t < 96) {
        const double x = double(x0 + l * step) * s * o.freq, f = split(x + o.ox, at);
        const int a0 = P[at] + o.iy, a1 = P[at + 1] + o.iy;
        L.cx[k][l] = make_double2(f, fade_d(f));
        L.ch[k][l] = uint32_t(P[a0]) | uint32_t(P[a0 + 1]) << 8 | uint32_t(P[a1]) << 16 | uint32_t(P[a1 + 1]) << 24;
        L.cy[k][l] = split(x + o.oy, at);
        L.cyi[k][l] = uint8_t(at);
    } else if (t < 192) {
        const double z = double(z0 + l * step) * s * o.freq, f = split(z + o.oz, at);
        L.rz[k][l] = make_double2(f, fade_d(f));
        L.rzi[k][l] = uint8_t(at);
        const double g = split(z + o.ox, at);
        L.rx[k][l] = make_double2(g, fade_d(g));
        L.ra[k][l] = uint16_t(P[at] | P[at + 1] << 8);
    } else {
        const double f = split(o.oz, at);
        L.z0[k] = make_double2(f, fade_d(f));
        L.iz0[k] = at;
    }
}
// channel(S, CH_S, x, 0, z) (WHICH = 0) or channel(S, CH_S, z, x, 0) (1) of the cell in column c and row r.
template <int WHICH> __device__ __forceinline__ double shift_lines(const SeedNoise &S, const ShiftLines &L, int c, int r) {
    double a[2] = {0, 0};
    #pragma unroll
    for (int side = 0; side < 2; side++)
        #pragma unroll 1
        for (int k = 3 * side; k < 3 * side + 3; k++) {
            const NOct &o = S.oct[kChanOff[CH_S] + k];
            const uint8_t *P = S.perm[kChanOff[CH_S] + k];
            const double2 x = WHICH ? L.rx[k][r] : L.cx[k][c], z = WHICH ? L.z0[k] : L.rz[k][r];
            const double dy = WHICH ? L.cy[k][c] : o.fy, ty = WHICH ? fade_d(dy) : o.vy;
            int b00, b01, b10, b11;
            if (WHICH) {
                const int m = L.ra[k][r], j = L.cyi[k][c], a0 = (m & 255) + j, a1 = (m >> 8) + j;
                b00 = P[a0]; b01 = P[a0 + 1]; b10 = P[a1]; b11 = P[a1 + 1];
            } else {
                const uint32_t h = L.ch[k][c];
                b00 = h & 255; b01 = h >> 8 & 255; b10 = h >> 16 & 255; b11 = h >> 24;
            }
            P += WHICH ? L.iz0[k] : int(L.rzi[k][r]);
            const double ex = x.x - 1, ey = dy - 1, ez = z.x - 1;
            const double lo = lerp_d(ty, lerp_d(x.y, grad_d(S.grad, P[b00], x.x, dy, z.x), grad_d(S.grad, P[b10], ex, dy, z.x)),
                                         lerp_d(x.y, grad_d(S.grad, P[b01], x.x, ey, z.x), grad_d(S.grad, P[b11], ex, ey, z.x)));
            const double hi = lerp_d(ty, lerp_d(x.y, grad_d(S.grad, P[b00 + 1], x.x, dy, ez), grad_d(S.grad, P[b10 + 1], ex, dy, ez)),
                                         lerp_d(x.y, grad_d(S.grad, P[b01 + 1], x.x, ey, ez), grad_d(S.grad, P[b11 + 1], ex, ey, ez)));
            a[side] += o.amp * lerp_d(z.y, lo, hi);
        }
    return (a[0] + a[1]) * S.factor[CH_S];
}
// desert_state_begin of the cell in column `col` and row `row` of the sub-block, through its tables.
__device__ __forceinline__ int desert_state_begin_patch(const SeedNoise &S, const PatchCache &C, const ShiftLines &L, const WorldDev &w, int x, int z,
                                                        int col, int row, PendingState &p) {
    const double px = x + 4. * shift_lines<0>(S, L, col, row);
    const double pz = z + 4. * shift_lines<1>(S, L, col, row);
    float t = 0, c = 0, e = 0, wv = 0, h = 0;
    #pragma unroll 1
    for (int k = 0; k < 5; k++) {                  // one copy of the octave's code for the five channels
        const int ch = k == 0 ? CH_T : k == 1 ? CH_C : k == 2 ? CH_E : k == 3 ? CH_W : CH_H;
        const float v = float(channel_patch(S, C, ch, px, pz));
        if (k == 0) { t = v; if (q10k(t) < 5500) return 0; }
        else if (k == 1) c = v;
        else if (k == 2) e = v;
        else if (k == 3) wv = v;
        else h = v;
    }
    return desert_state_decide(w, t, c, e, wv, h, p);
}
__device__ __forceinline__ int desert_state_begin(const SeedNoise &S, const WorldDev &w, int x, int z, PendingState &p) {
    const double px = x + 4. * channel(S, CH_S, x, 0, z);
    const double pz = z + 4. * channel(S, CH_S, z, x, 0);
    const float t = float(channel(S, CH_T, px, 0, pz));
    if (q10k(t) < 5500) return 0;
    const float c = float(channel(S, CH_C, px, 0, pz)), e = float(channel(S, CH_E, px, 0, pz));
    const float wv = float(channel(S, CH_W, px, 0, pz)), h = float(channel(S, CH_H, px, 0, pz));
    return desert_state_decide(w, t, c, e, wv, h, p);
}
// The same by four lanes per point (the whole warp calls; lanes without a point pass any coordinates): the 52 octaves
// of a point are spread over the lanes four at a time, every lane adds the four terms in the order of the channel sums
// (per side from +0, then the sides), and lane 0 of the four decides: its result as desert_state_begin's, the others' 0.
__device__ __forceinline__ double octave_term(const SeedNoise &S, int i, double x, double y, double z) {
    const double s = (kSideB >> i & 1) ? 337. / 331. : 1.;      // x * 1. is x: side A is not scaled
    const NOct &o = S.oct[i];
    return o.amp * perlin(o, S.perm[i], S.grad, x * s * o.freq, y * s * o.freq, z * s * o.freq);
}
// Sum of the `n` octaves from off (side A's, then as many of side B), term k held by lane k & 3 of round k / 4.
struct SideSum {
    double acc = 0, a = 0;
    __device__ __forceinline__ bool add(double t, bool last_a, bool last_b) {       // true: the channel's sum is in a
        acc += t;
        if (last_a) { a = acc; acc = 0; }
        if (last_b) { a += acc; acc = 0; }
        return last_b;
    }
};
__device__ __forceinline__ int desert_state_begin4(const SeedNoise &S, const WorldDev &w, int x, int z, bool on, PendingState &p) {
    const int lane = threadIdx.x & 31, o = lane & 3, base = lane & 28;
    double v[2];                                   // the two shift samples: at (x, 0, z) and at (z, x, 0)
    {
        SideSum sum;
        #pragma unroll 1
        for (int r = 0; r < 3; r++) {
            const int k = 4 * r + o, second = k >= 6, i = kChanOff[CH_S] + (second ? k - 6 : k);
            const double t = octave_term(S, i, second ? z : x, second ? x : 0, second ? 0 : z);
            #pragma unroll
            for (int j = 0; j < 4; j++) {
                const int n = 4 * r + j;
                if (sum.add(__shfl_sync(0xffffffffu, t, base + j), n == 2 || n == 8, n == 5 || n == 11)) (n == 5 ? v[0] : v[1]) = sum.a * S.factor[CH_S];
            }
        }
    }
    const double px = x + 4. * v[0], pz = z + 4. * v[1];
    float t;
    {
        const double u = octave_term(S, kChanOff[CH_T] + o, px, 0, pz);
        const double a = __shfl_sync(0xffffffffu, u, base), b = __shfl_sync(0xffffffffu, u, base + 1);
        const double c = __shfl_sync(0xffffffffu, u, base + 2), d = __shfl_sync(0xffffffffu, u, base + 3);
        t = float(((0. + a + b) + (0. + c + d)) * S.factor[CH_T]);
    }
    const bool warm = on && q10k(t) >= 5500;
    if (!__any_sync(0xffffffffu, warm)) return 0;
    // C (18 octaves), E (8), W (6), H (4): nine rounds
    float c = 0, e = 0, wv = 0, h = 0;
    SideSum sum;
    constexpr uint64_t endA = 1ull << 8 | 1ull << 21 | 1ull << 28 | 1ull << 33, endB = 1ull << 17 | 1ull << 25 | 1ull << 31 | 1ull << 35;
    #pragma unroll 1
    for (int r = 0; r < 9; r++) {
        const int k = 4 * r + o;
        const int i = k < 18 ? kChanOff[CH_C] + k : k < 26 ? kChanOff[CH_E] + k - 18 : k < 32 ? kChanOff[CH_W] + k - 26 : kChanOff[CH_H] + k - 32;
        const double u = octave_term(S, i, px, 0, pz);
        #pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = 4 * r + j;
            if (sum.add(__shfl_sync(0xffffffffu, u, base + j), endA >> n & 1, endB >> n & 1)) {
                if (n == 17) c = float(sum.a * S.factor[CH_C]);
                else if (n == 25) e = float(sum.a * S.factor[CH_E]);
                else if (n == 31) wv = float(sum.a * S.factor[CH_W]);
                else h = float(sum.a * S.factor[CH_H]);
            }
        }
    }
    return warm && o == 0 ? desert_state_decide(w, t, c, e, wv, h, p) : 0;
}
__device__ inline int desert_state_finish(const WorldDev &w, const PendingState &p) {
    int32_t q[6];
    for (int k = 0; k < 6; k++) q[k] = p.q[k];
    q[4] = depth_q(w, p.c, p.e, p.w);
    if (p.stage == 2) return classify_exact(w, q) == 2 ? 1 : 0;
    int b = classify_exact(w, q);
    if (b == 2) return 2;
    if (b != 7 && b != 11) return 0;
    if (q[5] > 500 || q[5] < -500) return 0;
    q[5] = q[5] >= 0 ? 501 : -501;
    b = grid_lookup(w, q);
    if (b < 0) b = classify_exact(w, q);
    return b == 2 ? 1 : 0;
}
// desert_state_finish by a group of 8 lanes (the whole warp calls; `on`: the group has a point), T in shared memory.
__device__ __forceinline__ int desert_state_finish_group(const WorldDev &w, const ExactTab &T, const PendingState &p, bool on) {
    int32_t q[6];
    #pragma unroll
    for (int k = 0; k < 6; k++) q[k] = p.q[k];
    const GroupSearch first = classify_group_begin(w, T, q, on);
    q[4] = depth_of(spline_group(T.spline, p.c, p.e, ridge_fold(p.w), p.w));
    const int b = classify_group_end(w, q, on, first);
    // first stage: a river near W = 0 crosses to what lies beyond its bank
    const bool river = on && p.stage != 2 && (b == 7 || b == 11) && q[5] <= 500 && q[5] >= -500;
    int res = b == 2 ? (p.stage == 2 ? 1 : 2) : 0;
    if (__any_sync(0xffffffffu, river)) {
        q[5] = q[5] >= 0 ? 501 : -501;
        int b2 = river ? grid_lookup(w, q) : 0;
        const bool again = river && b2 < 0;
        if (__any_sync(0xffffffffu, again)) {
            const int b3 = classify_group_end(w, q, again, classify_group_begin(w, T, q, again));
            if (again) b2 = b3;
        }
        if (river) res = b2 == 2 ? 1 : 0;
    }
    return res;
}
__device__ inline int desert_state(const SeedNoise &S, const WorldDev &w, int x, int z) {
    PendingState p;
    const int v = desert_state_begin(S, w, x, z, p);
    return v >= 0 ? v : desert_state_finish(w, p);
}
// Hot-zone predicate: temperature at the unwarped point >= 0.55 (dsearch_desert.cpp:334).
__device__ __forceinline__ int hot_state(const SeedNoise &S, int x, int z) { return channel(S, CH_T, x, 0, z) >= 0.55 ? 2 : 0; }
// Low-octave proxy probability (desert_proxy.hpp:24-31): the bins of continentalness and erosion, where T >= 0.55.
__device__ __forceinline__ float proxy_bin(const WorldDev &w, double c, double e) {
    int i = int(floor((c + 0.8) / 0.05)), j = int(floor((e + 1.0) / 0.05));
    i = i < 0 ? 0 : (i > 39 ? 39 : i);
    j = j < 0 ? 0 : (j > 39 ? 39 : j);
    return w.prob[i * 40 + j];
}
__device__ __forceinline__ float proxy_prob(const SeedNoise &S, const WorldDev &w, int x, int z) {
    if (channel(S, CH_T, x, 0, z) < 0.55) return 0.f;
    return proxy_bin(w, channel_low(S, CH_C, x, z, 0, 3), channel_low(S, CH_E, x, z, 0, 2));
}
#endif

// Build the noise of `n` seeds into d_out (device), on `st`.  Defined in noise.cu.
void seed_noise_build(const uint64_t *d_seeds, uint32_t n, SeedNoise *d_out, cudaStream_t st);

}  // namespace dsg
