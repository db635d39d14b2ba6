// Amplitude kernels of the seed gate: the maximum over a periodic grid of a blurred Perlin octave, bit for bit the
// value of the reference's summation order, at a fraction of its work.
//
// The value the gate defines (per noise side) is the maximum over all cells of a chain of float operations: corner
// terms looked up by lattice hash and added in a fixed order, then a horizontal and a vertical chain of blur taps.
// Evaluating that chain at every cell costs 8 to 18 shared-memory gathers per cell, which is what bounded the
// kernels that did so.  Here every cell is first evaluated by a cheaper expression of the same real number, and the
// defining chain only where the maximum can be:
//
//  * Screen.  A corner term is linear in the hashed gradient, t = w wy(dy) (gx a_u b_v + gy (fy - dy) b_u b_v + gz b_u c_v),
//    with a, b, c per axis.  The hash of lattice point (x, z) is s[(c(dy, x) + z) mod 256], s = P & 15: along z
//    every lattice column is the same sequence, shifted by the column's hash.  So the whole z direction (corner
//    weights and blur) is applied once to the 256-entry sequence:  U_dy = w wy F[b; gx], V_dy = w wy ((fy - dy)
//    F[b; gy] + F[c; gz]).  A cell then needs, per lattice column, U and V of its two hashes (two 8-byte loads at
//    consecutive addresses across the warp: no bank conflicts), and the x direction: corner weights as fused
//    multiply-adds, the blur over a ring of samples in registers (256^2: symmetric pairs; 512^2: pending sums).
//  * Exact cells.  Screen and defining chain differ by at most E (below) at every cell, so the cell of the defining
//    chain's maximum has a screen value of at least (screen maximum) - 2 E.  The screen lists the cells within 2 E of
//    its running maximum (normally one), and the warp evaluates the defining chain there.  A seed whose screen
//    maxima cannot reach the threshold even with the error added is dropped before that.
//
// Error bound E.  All corner terms of a cell sum to at most w x 2 in magnitude (the interpolation weights sum to 1, a
// gradient has two components of magnitude 1 on offsets of at most 1) and the blur is an average, so M = 2 w = 1.91
// bounds every partial sum.  With u = 2^-24: the defining chain rounds a term at most 1 (table entry) + 18 (or 8)
// (sum) + 9 + 9 (or 15 + 15) (blur; twice that where products and sums round separately) + 1 (normaliser) times; the
// screen 1 + 11 (z taps) + 4 (U, V) + 1 (sum of the two hashes) + 6 (x corners) + 9 or 15 (blur) + 2 (tap
// roundings).  The largest total is 46 + 34 = 80 u M = 9.1e-6 (CPU form), 39 + 40 = 79 u M (full gate); E = 1.5e-5.
//
// What bounds them, on a B200 at 1,965 MHz, 2^26 seed indices (482,670 phase-passed seeds, 31,114 full-gate seeds):
// register operands and instruction issue.  Per cell and lane the 256^2 screen issues 20.9 instructions (13.5 of them
// on the FMA pipe) and reads 16 bytes of shared memory: issue 69% of active cycles, the FMA pipe busy in 62% (a two-wide
// instruction holds it for two; by instructions 50%), shared-memory wavefronts 59%.
// Before, every cell gathered its 18 (or 8) corner terms: the pre-gate took 161 ms (now 52), the full gate 43.6 (now
// 15.4), the sub-grid form 21.7 ms for 84,414 seeds (now 8.3).  Measured on the way: a multiply-add of three distinct
// registers takes 1.56 cycles per scheduler, of two and a constant 1.16, the two-wide one 3 (so two-wide forms serve
// only for sums and products of two operands, 2 cycles); with two-wide multiply-adds throughout 54.5 ms, pending sums
// instead of symmetric pairs 52.8, pending sums shifted through registers instead of rings 92 (the shifts became
// moves), a look at the cells every column instead of every third 53.5.  3 blocks (12 warps) per SM and 4 rows per lane: 2 rows
// 63.7, 8 rows 53.6, 4 blocks 52.5 (8% slower on a short range).
#pragma once
#include "common.cuh"
#include "gate_tuned.h"

namespace dsg {
namespace gate {

// Temperature octave -10 of one side, as the gate needs it (PerlinParams, gate.cuh:49).
struct __align__(16) Oct { uint8_t perm[256]; double ox, oz, fy, vy; int32_t iy, pad[3]; };
static_assert(sizeof(Oct) == 304, "Oct layout");

// 2 E.  A wider window lists more cells and drops fewer seeds, and the amplitudes are the same: the tests build it wider
// to fill the lists, which ordinary seeds do not.
#ifndef DSG_AMP_WINDOW
#define DSG_AMP_WINDOW 3e-5f
#endif
constexpr float AMP_E2 = DSG_AMP_WINDOW;
static_assert(AMP_E2 >= 3e-5f, "the error bound");
constexpr float AMP_FLOOR = 0.24f;                 // amplitudes below it are rare: no cell under it is listed at first
constexpr int AMP_CAP = 32;                        // listed cells per warp

// Blur taps, their normaliser and the octave's weight of a 256^2 gate (by value, in the kernel-parameter bank).
struct Taps256 { float k[9], norm; double w; };
struct Taps512 { float k[15], norm; double w; };

// ---------------------------------------------------------------- device math
// fade as the reference's GPU gate evaluates it: nvcc contracts t*6-15 and t*(..)+10 (gate.cuh:51).
__device__ __forceinline__ double fade_fused(double t) { return t * t * t * __fma_rn(t, __fma_rn(t, 6.0, -15.0), 10.0); }
__device__ __forceinline__ double fade_plain(double t) { return t * t * t * (t * (t * 6. - 15.) + 10.); }
// Minecraft's 16 gradients: two of (x, y, z) with signs; equal to gx*x + gy*y + gz*z for every nonzero value.
__device__ __forceinline__ double gradd(int h, double x, double y, double z) {
    h &= 15;
    const double u = h < 8 ? x : y;
    const double v = h < 4 ? y : ((h == 12 || h == 14) ? x : z);
    return ((h & 1) ? -u : u) + ((h & 2) ? -v : v);
}
// The same gradients as gx*x + gy*y + gz*z with their 0/+-1 components (the CPU code's gradient).  Component + 1
// of hash h sits in bits 2h, 2h + 1 of its word.
constexpr signed char kGradXYZ[16][3] = {{1, 1, 0}, {-1, 1, 0}, {1, -1, 0}, {-1, -1, 0}, {1, 0, 1}, {-1, 0, 1}, {1, 0, -1}, {-1, 0, -1},
                                         {0, 1, 1}, {0, -1, 1}, {0, 1, -1}, {0, -1, -1}, {1, 1, 0}, {0, -1, 1}, {-1, 1, 0}, {0, -1, -1}};
constexpr uint32_t grad_word(int axis) {
    uint32_t w = 0;
    for (int h = 0; h < 16; h++) w |= uint32_t(kGradXYZ[h][axis] + 1) << (2 * h);
    return w;
}
constexpr uint32_t kGX = grad_word(0), kGY = grad_word(1), kGZ = grad_word(2);
__device__ __forceinline__ int grad_comp(uint32_t word, int h) { return int((word >> (2 * h)) & 3u) - 1; }
__device__ __forceinline__ double grad_products(int h, double x, double y, double z) {
    return double(grad_comp(kGX, h)) * x + double(grad_comp(kGY, h)) * y + double(grad_comp(kGZ, h)) * z;
}

// Two floats in one 64-bit register: one instruction for two products or sums, each rounded as its scalar form.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { f2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ float warp_max(float v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ---------------------------------------------------------------- listed cells of a warp
struct CellList { uint32_t pos[AMP_CAP]; float val[AMP_CAP]; };
static_assert(AMP_CAP == 32, "list_cells clears a full list with a lane per entry");
// Running state of a warp's pass over its cells (warp-uniform): the maximum of the cells listed so far, the value
// from which cells are listed, the number listed.
struct Run { float best, lim; int n; };
template <int N> struct Cells { float v[N]; };
// The lane's N new cells (the first at `pos`, the next `dpos` apart) when one of the warp's exceeds lim: best becomes
// the warp's running maximum, lim rises to within 2 E of it, and the cells not below lim are listed.  A full list is
// first cleared of cells the maximum has left behind; should that not be enough, n becomes AMP_CAP + 1 and the
// caller evaluates every cell.  Rare (a handful of times per pass), so not inlined.
template <int N>
__device__ __noinline__ Run list_cells(Cells<N> c, uint32_t pos, uint32_t dpos, CellList *L, Run r, int lane) {
    float mx = c.v[0];
    #pragma unroll
    for (int q = 1; q < N; q++) mx = fmaxf(mx, c.v[q]);
    r.best = fmaxf(r.best, warp_max(mx));
    r.lim = fmaxf(r.lim, r.best - AMP_E2);
    #pragma unroll
    for (int q = 0; q < N; q++) {
        const bool on = c.v[q] >= r.lim;
        const uint32_t m = __ballot_sync(0xffffffffu, on);
        if (!m || r.n > AMP_CAP) continue;
        if (r.n + __popc(m) > AMP_CAP) {
            __syncwarp();
            const bool keep = lane < r.n && L->val[lane] >= r.lim;
            const uint32_t p = L->pos[lane]; const float x = L->val[lane];
            const uint32_t k = __ballot_sync(0xffffffffu, keep);
            __syncwarp();
            if (keep) { const int at = __popc(k & ((1u << lane) - 1)); L->pos[at] = p; L->val[at] = x; }
            r.n = __popc(k);
            __syncwarp();
        }
        if (r.n + __popc(m) > AMP_CAP) { r.n = AMP_CAP + 1; continue; }
        if (on) { const int at = r.n + __popc(m & ((1u << lane) - 1)); L->pos[at] = pos + q * dpos; L->val[at] = c.v[q]; }
        r.n += __popc(m);
    }
    __syncwarp();
    return r;
}

// Gradient components of the permutation's 256 entries as floats, three arrays (threads t of nt).
__device__ __forceinline__ void grad_rows(const uint8_t *__restrict__ P, float *__restrict__ gx, float *__restrict__ gy, float *__restrict__ gz, int t, int nt) {
    for (int e = t; e < 256; e += nt) {
        const int h = P[e] & 15;
        gx[e] = float(grad_comp(kGX, h)); gy[e] = float(grad_comp(kGY, h)); gz[e] = float(grad_comp(kGZ, h));
    }
}
// U and V of both y corners at sequence position e: NT taps from position e0.
template <int NT>
__device__ __forceinline__ void uv_entry(const float *__restrict__ gx, const float *__restrict__ gy, const float *__restrict__ gz,
                                         const float (&b)[NT], const float (&c)[NT], int e0, float w0, float w1, float fy, f2 &uv0, f2 &uv1) {
    float fx = 0.f, f_y = 0.f, fz = 0.f;
    #pragma unroll
    for (int t = 0; t < NT; t++) {
        const int i = (e0 + t) & 255;
        fx = __fmaf_rn(b[t], gx[i], fx); f_y = __fmaf_rn(b[t], gy[i], f_y); fz = __fmaf_rn(c[t], gz[i], fz);
    }
    uv0 = pack2(w0 * fx, w0 * __fmaf_rn(fy, f_y, fz));
    uv1 = pack2(w1 * fx, w1 * __fmaf_rn(fy - 1.f, f_y, fz));
}

// ---------------------------------------------------------------- 256^2 gates
// AMP_AA: the anti-aliased pre-gate (gate.cuh:198-346, stream_max<256,4,8,true>): 18 merged corner tables (four
// half-lattice parities averaged), fused blur chains.  AMP_CPU: the CPU search's sub-grid estimate
// (lowfield.hpp:60-102, what dsearch_desert.cpp:216-223 tests): 8 corners of one parity, unfused fade and blur.
// AMP_ONEPAR: the reference's legacy one-parity GPU pre-gate (tgate box=0, gate.cuh:236-313): the same grid with
// fused fade and blur chains and the device taps.
enum { AMP_AA = 0, AMP_CPU = 1, AMP_ONEPAR = 2 };

constexpr int PG_ZL = 4;                                        // grid rows per lane
constexpr int PG_WARPS = 8 / PG_ZL, PG_SIDE = 32 * PG_WARPS, PG_THREADS = 2 * PG_SIDE;   // warps, threads per side
constexpr int PG_GRP = 3;                                       // columns between two looks at the cells (divides 9)
template <int MODE> struct alignas(16) Side256 {
    static constexpr int NC = MODE == AMP_AA ? 3 : 2;          // lattice columns a cell's corners span
    static constexpr int NT = NC + 8;                          // z taps: corners and blur
    static constexpr int COLS = 267;                           // lattice columns streamed: 256 + 8 + NC - 1, rounded up to groups of PG_GRP
    static_assert(COLS >= 256 + 8 + NC - 1 && COLS % PG_GRP == 0, "columns");
    static constexpr int NTAB = MODE == AMP_AA ? 288 : 128;
    union {
        struct { f2 uv[2][512]; } a;                           // screen: [dy][position], positions 256.. repeat 0..
        struct { float tab[NTAB], smp[PG_WARPS][84]; } x;      // exact cells: corner tables, a cell's 81 samples per warp
    };
    uint32_t cw[272];                                          // 8 c(0, x) | 8 c(1, x) << 16 of lattice column ix0 + J
    alignas(16) uint8_t P[256];
    float bz[16], cz[16];
    CellList list[PG_WARPS];
};

// Corner tables of the defining chain, tab[e], as the reference computes them (gate.cuh:218-244, lowfield.hpp:65-73).
template <int MODE>
__device__ __forceinline__ void corner_tables256(const Oct &p, double w, float *__restrict__ tab, int t) {
    const double ox = p.ox, oz = p.oz, fy = p.fy, vy = p.vy;
    if (MODE == AMP_AA) {
        double fr[2][2]; int sh[2][2];
        #pragma unroll
        for (int ax = 0; ax < 2; ax++) {
            const double o = ax ? oz : ox;
            #pragma unroll
            for (int q = 0; q < 2; q++) { const double b = o + 0.5 * q; fr[ax][q] = b - floor(b); sh[ax][q] = int(floor(b) - floor(o)); }
        }
        for (int e = t; e < 288; e += PG_SIDE) {
            const int h = e & 15, dy = (e >> 4) & 1, uv = e >> 5, u = uv / 3, v = uv % 3;
            double acc = 0;
            #pragma unroll
            for (int px = 0; px < 2; px++)
                #pragma unroll
                for (int pz = 0; pz < 2; pz++) {
                    const int dx = u - sh[0][px], dz = v - sh[1][pz];
                    if (dx < 0 || dx > 1 || dz < 0 || dz > 1) continue;
                    const double fx = fr[0][px], fz = fr[1][pz], tx = fade_fused(fx), tz = fade_fused(fz);
                    const double wc = (dx ? tx : 1 - tx) * (dy ? vy : 1 - vy) * (dz ? tz : 1 - tz);
                    acc = __fma_rn(wc, gradd(h, fx - dx, fy - dy, fz - dz), acc);
                }
            tab[e] = float(0.25 * w * acc);
        }
    } else {
        constexpr bool CPU = MODE == AMP_CPU;
        const double fx = ox - floor(ox), fz = oz - floor(oz);
        const double tx = CPU ? fade_plain(fx) : fade_fused(fx), tz = CPU ? fade_plain(fz) : fade_fused(fz), ty = CPU ? fade_plain(fy) : vy;
        for (int e = t; e < 128; e += PG_SIDE) {
            const int c = e >> 4, h = e & 15, dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
            const double wc = (dx ? tx : 1 - tx) * (dy ? ty : 1 - ty) * (dz ? tz : 1 - tz);
            tab[e] = CPU ? float(w * wc * grad_products(h, fx - dx, fy - dy, fz - dz))
                         : float(1.0 * w * wc * gradd(h, fx - dx, fy - dy, fz - dz));
        }
    }
}
// The defining chain at cell (i, k): 81 samples by the lanes, 9 horizontal chains, one vertical chain.  All lanes
// return it.
template <int MODE>
__device__ __forceinline__ float exact_cell256(const Side256<MODE> &sd, float *__restrict__ smp, const Taps256 &tp, int iz0, int i, int k, int lane) {
    using A = Side256<MODE>;
    constexpr bool CPU = MODE == AMP_CPU;
    const auto acc = [](float a, float c, float v) { return CPU ? __fadd_rn(a, __fmul_rn(c, v)) : __fmaf_rn(c, v, a); };
    for (int n = lane; n < 81; n += 32) {
        const int col = i - 4 + n % 9, row = k - 4 + n / 9 + iz0;
        float s = 0.f;
        #pragma unroll
        for (int v = 0; v < A::NC; v++)                          // order v, dy, u (gate.cuh:274-281; corner order for 8)
            #pragma unroll
            for (int dy = 0; dy < 2; dy++)
                #pragma unroll
                for (int u = 0; u < A::NC; u++) {
                    const uint32_t c = sd.cw[(col + u) & 255] >> (dy ? 19 : 3);
                    const int h = sd.P[(c + uint32_t(row + v)) & 255u] & 15;
                    s = __fadd_rn(s, sd.x.tab[(MODE == AMP_AA ? (u * 3 + v) * 2 + dy : u + 2 * dy + 4 * v) * 16 + h]);
                }
        smp[n] = s;
    }
    __syncwarp();
    float hv = 0.f;
    if (lane < 9)
        #pragma unroll
        for (int d = 0; d < 9; d++) hv = acc(hv, tp.k[d], smp[lane * 9 + d]);
    float o = 0.f;
    #pragma unroll
    for (int d = 0; d < 9; d++) o = acc(o, tp.k[d], __shfl_sync(0xffffffffu, hv, d));
    __syncwarp();
    return CPU ? o : __fmul_rn(o, tp.norm);
}

// One CTA per seed; a warp holds PG_ZL grid rows per lane of one noise side (rows lane + 32 q), the columns stream.
// Survivors (amplitude sum >= thr; the sub-grid forms: not below thr) are appended; side_amp (may be null) gets both
// sides' maxima.
template <int MODE>
__global__ void __launch_bounds__(PG_THREADS, DSG_PG_MINBLOCKS)
k_amp256(const Oct *__restrict__ oct, const uint64_t *__restrict__ seeds, const uint32_t *__restrict__ n_in, uint32_t cap_in, double thr,
         const __grid_constant__ Taps256 tp, uint64_t *__restrict__ out_seed, uint32_t *__restrict__ out_idx, uint32_t *__restrict__ n_out,
         uint32_t cap_out, float *__restrict__ side_amp) {
    using A = Side256<MODE>;
    constexpr int NC = A::NC, NT = A::NT, ZL = PG_ZL, W = PG_WARPS;
    __shared__ A sides[2];
    __shared__ float sTop[2][2 * W], sAmp[2 * W];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, side = warp / W, wi = warp % W, t = threadIdx.x % PG_SIDE;
    A &sd = sides[side];
    const uint32_t n = min(*n_in, cap_in);
    const float floor0 = thr > 0.4 ? float(0.44 * thr) : AMP_FLOOR;
    const f2 kc = pack2(tp.k[4], tp.k[4]);                       // the taps are symmetric: k[8 - d] = k[d]
    int it = 0;
    for (uint32_t s = blockIdx.x; s < n; s += gridDim.x) {
        const Oct &p = oct[2 * size_t(s) + side];
        __syncthreads();                                         // the previous seed's cells are done with the shared arrays
        if (t < 16) reinterpret_cast<uint4 *>(sd.P)[t] = reinterpret_cast<const uint4 *>(p.perm)[t];
        const double ox = p.ox, oz = p.oz, fyd = p.fy, vyd = MODE == AMP_CPU ? fade_plain(p.fy) : p.vy;
        const int iy = p.iy, ix0 = int(floor(ox)), iz0 = int(floor(oz));
        // corner weights (b) and weights times offset (a along x, c along z) of the cell's lattice columns
        float a[NC], b[NC];
        {
            double db[2][3], da[2][3];
            #pragma unroll
            for (int ax = 0; ax < 2; ax++) {
                const double o = ax ? oz : ox, fl = floor(o);
                #pragma unroll
                for (int u = 0; u < 3; u++) { db[ax][u] = 0; da[ax][u] = 0; }
                #pragma unroll
                for (int q = 0; q < (MODE == AMP_AA ? 2 : 1); q++) {
                    const double h = o + 0.5 * q, f = h - floor(h), tt = MODE == AMP_CPU ? fade_plain(f) : fade_fused(f), sc = MODE == AMP_AA ? 0.5 : 1.0;
                    const bool sh = floor(h) > fl;
                    const double b0 = sc * (1 - tt), b1 = sc * tt, a0 = b0 * f, a1 = b1 * (f - 1);
                    db[ax][0] += sh ? 0 : b0; db[ax][1] += sh ? b0 : b1; db[ax][2] += sh ? b1 : 0;
                    da[ax][0] += sh ? 0 : a0; da[ax][1] += sh ? a0 : a1; da[ax][2] += sh ? a1 : 0;
                }
            }
            #pragma unroll
            for (int u = 0; u < NC; u++) { a[u] = float(da[0][u]); b[u] = float(db[0][u]); }
            if (t < NT) {
                double vb = 0, vc = 0;
                #pragma unroll
                for (int v = 0; v < NC; v++) {
                    const int d = t - v;
                    const double g = d >= 0 && d < 9 ? double(tp.k[d]) * double(tp.norm) : 0.0;
                    vb += db[1][v] * g; vc += da[1][v] * g;
                }
                sd.bz[t] = float(vb); sd.cz[t] = float(vc);
            }
        }
        __syncthreads();
        for (int j = t; j < A::COLS; j += PG_SIDE) {
            const int pc = sd.P[(ix0 + j) & 255] + iy;
            sd.cw[j] = uint32_t(sd.P[pc & 255]) << 3 | uint32_t(sd.P[(pc + 1) & 255]) << 19;
        }
        float *gx = reinterpret_cast<float *>(&sd.a.uv[0][256]), *gy = gx + 256, *gz = reinterpret_cast<float *>(&sd.a.uv[1][256]);
        grad_rows(sd.P, gx, gy, gz, t, PG_SIDE);
        __syncthreads();
        {
            float tb[NT], tc[NT];
            #pragma unroll
            for (int k = 0; k < NT; k++) { tb[k] = sd.bz[k]; tc[k] = sd.cz[k]; }
            const float w0 = float(tp.w * (1 - vyd)), w1 = float(tp.w * vyd), fy = float(fyd);
            #pragma unroll 1
            for (int e = t; e < 256; e += PG_SIDE) uv_entry<NT>(gx, gy, gz, tb, tc, e - 4 + iz0, w0, w1, fy, sd.a.uv[0][e], sd.a.uv[1][e]);
        }
        __syncthreads();                                         // the gradient rows are read; the repeats overwrite them
        for (int e = t; e < 512; e += PG_SIDE) sd.a.uv[e >> 8][(e & 255) + 256] = sd.a.uv[e >> 8][e & 255];
        __syncthreads();
        const int row0 = lane + 32 * ZL * wi;
        const char *uv0 = reinterpret_cast<const char *>(&sd.a.uv[0][row0]), *uv1 = reinterpret_cast<const char *>(&sd.a.uv[1][row0]);
        float start = floor0;
        for (;;) {
            Run r{-1e9f, start, 0};
            // acc[u]: the samples begun by the last columns; ring[J mod 9]: the last nine samples, two rows per register
            // pair (the columns are unrolled by nine, so the ring's slots are fixed registers)
            float acc[NC - 1][ZL];
            f2 ring[9][ZL / 2];
            #pragma unroll
            for (int q = 0; q < ZL; q++) {
                #pragma unroll
                for (int u = 0; u < NC - 1; u++) acc[u][q] = 0.f;
                #pragma unroll
                for (int j = 0; j < 9; j++) ring[j][q / 2] = 0;
            }
            #pragma unroll 1
            for (int J0 = 0; J0 < A::COLS; J0 += 9) {
                #pragma unroll
                for (int g = 0; g < 9; g += PG_GRP) {
                    if (g == A::COLS % 9 && J0 + g == A::COLS) break;
                    Cells<ZL> c[PG_GRP];
                    float mx;
                    #pragma unroll
                    for (int k = 0; k < PG_GRP; k++) {
                        const int ph = g + k;
                        const uint32_t w = sd.cw[J0 + ph];
                        const char *p0 = uv0 + (w & 0xffffu), *p1 = uv1 + (w >> 16);
                        float S[ZL];
                        #pragma unroll
                        for (int q = 0; q < ZL; q++) {
                            float U, V;
                            unpack2(add2(*reinterpret_cast<const f2 *>(p0 + 256 * q), *reinterpret_cast<const f2 *>(p1 + 256 * q)), U, V);
                            S[q] = __fmaf_rn(a[NC - 1], U, __fmaf_rn(b[NC - 1], V, acc[0][q]));
                            #pragma unroll
                            for (int u = 1; u < NC - 1; u++) acc[u - 1][q] = __fmaf_rn(a[NC - 1 - u], U, __fmaf_rn(b[NC - 1 - u], V, acc[u][q]));
                            acc[NC - 2][q] = __fmaf_rn(a[0], U, b[0] * V);
                        }
                        #pragma unroll
                        for (int q = 0; q < ZL / 2; q++) {
                            ring[ph][q] = pack2(S[2 * q], S[2 * q + 1]);
                            float o0, o1;
                            unpack2(mul2(kc, ring[(ph + 5) % 9][q]), o0, o1);
                            #pragma unroll
                            for (int d = 3; d >= 0; d--) {           // taps d and 8 - d: columns J - 8 + d and J - d
                                float x, y;
                                unpack2(add2(ring[(ph + 1 + d) % 9][q], ring[(ph + 9 - d) % 9][q]), x, y);
                                o0 = __fmaf_rn(tp.k[d], x, o0); o1 = __fmaf_rn(tp.k[d], y, o1);
                            }
                            c[k].v[2 * q] = o0; c[k].v[2 * q + 1] = o1;
                            mx = k == 0 && q == 0 ? fmaxf(o0, o1) : max3(mx, o0, o1);
                        }
                    }
                    if (__any_sync(0xffffffffu, mx > r.lim)) {
                        #pragma unroll
                        for (int k = 0; k < PG_GRP; k++) {
                            // column J completes sample column J - (NC - 1), the last tap of the cells at J - (NC - 1) - 4
                            const int J = J0 + g + k;
                            if (J >= 8 + NC - 1) r = list_cells<ZL>(c[k], uint32_t((J - (NC - 1) - 4) & 255) << 8 | uint32_t(row0), 32u, &sd.list[wi], r, lane);
                        }
                    }
                }
            }
            const float best = r.best;
            const int nl = r.n;
            const int par = it++ & 1;                            // two slots: the next pass writes the other one
            if (lane == 0) sTop[par][warp] = best;
            __syncthreads();
            float top[2] = {-1e9f, -1e9f};
            #pragma unroll
            for (int k = 0; k < 2 * W; k++) top[k / W] = fmaxf(top[k / W], sTop[par][k]);
            // a side whose maximum is under the floor (nothing listed) or so near it that cells within 2 E may be
            // missing is bounded by the floor; should that not drop the seed, both sides list without a floor
            const float ok = start + AMP_E2;
            if (double(fmaxf(top[0], ok)) + double(fmaxf(top[1], ok)) + double(AMP_E2) < thr) break;
            if (top[0] < ok || top[1] < ok) { start = -1e9f; continue; }
            corner_tables256<MODE>(p, tp.w, sd.x.tab, t);
            __syncthreads();
            const float cut = top[side] - AMP_E2;
            float m = -1e9f;
            const bool every = nl > AMP_CAP;                     // this warp's cells: columns x the rows of its lanes
            for (int c = 0; c < (every ? 256 * 32 * ZL : nl); c++) {
                if (!every && sd.list[wi].val[c] < cut) continue;
                const uint32_t pos = every ? uint32_t(c / (32 * ZL)) << 8 | uint32_t(c % (32 * ZL) + 32 * ZL * wi) : sd.list[wi].pos[c];
                m = fmaxf(m, exact_cell256<MODE>(sd, sd.x.smp[wi], tp, iz0, int(pos >> 8), int(pos & 255u), lane));
            }
            if (lane == 0) sAmp[warp] = m;
            __syncthreads();
            if (threadIdx.x == 0) {
                float ma = -1e9f, mb = -1e9f;
                #pragma unroll
                for (int k = 0; k < W; k++) { ma = fmaxf(ma, sAmp[k]); mb = fmaxf(mb, sAmp[W + k]); }
                const float amp = __fadd_rn(ma, mb);
                if (side_amp) { side_amp[2 * size_t(s)] = ma; side_amp[2 * size_t(s) + 1] = mb; }
                if (MODE == AMP_AA ? double(amp) >= thr : !(double(amp) < thr)) {
                    const uint32_t i = atomicAdd(n_out, 1u);
                    if (i < cap_out) { out_seed[i] = seeds[s]; if (out_idx) out_idx[i] = s; }
                }
            }
            break;
        }
    }
}

// ---------------------------------------------------------------- 512^2 full gate (gate.cuh stream_max<512,7,8,false>)
constexpr int FG_ZL = DSG_FG_ROWS;                              // grid rows per lane
constexpr int FG_WARPS = 8 / FG_ZL;                             // warps per (side, row parity)
constexpr int FG_COLS = 264;                                   // lattice columns streamed: 526 grid columns, 14 of them the blur's run-in
constexpr int FG_SIDE = 64 * FG_WARPS, FG_THREADS = 2 * FG_SIDE;
struct alignas(16) Side512 {
    union {
        struct { f2 uv[2][2][512]; } a;                         // screen: [row parity][dy][position]
        struct { float tab[512], smp[2 * FG_WARPS][232]; } x;   // exact cells: corner tables, a cell's 225 samples per warp
    };
    uint32_t cw[FG_COLS];
    alignas(16) uint8_t P[256];
    float bz[2][10], cz[2][10];                                 // [row parity]: taps on lattice rows -4 .. 5
    CellList list[2 * FG_WARPS];
};
// Corner tables per parity (gate.cuh:237-244), tab[(px*2+pz)*128 + c*16 + h].
__device__ __forceinline__ void corner_tables512(const Oct &p, double w, float *__restrict__ tab, int t) {
    for (int e = t; e < 512; e += FG_SIDE) {
        const int par = e >> 7, c = (e >> 4) & 7, h = e & 15, px = par >> 1, pz = par & 1;
        const double bx = px * 0.5 + p.ox, bz = pz * 0.5 + p.oz;
        const double fx = bx - floor(bx), fz = bz - floor(bz), tx = fade_fused(fx), tz = fade_fused(fz);
        const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
        const double wc = (dx ? tx : 1 - tx) * (dy ? p.vy : 1 - p.vy) * (dz ? tz : 1 - tz);
        tab[e] = float(1.0 * w * wc * gradd(h, fx - dx, p.fy - dy, fz - dz));
    }
}
// The defining chain at cell (i, r): 225 samples by the lanes, 15 horizontal chains, one vertical chain.
__device__ __forceinline__ float exact_cell512(const Side512 &sd, float *__restrict__ smp, const Taps512 &tp, int dx0, int iza, int izb, int i, int r,
                                               int lane) {
    for (int n = lane; n < 225; n += 32) {
        const int ci = (i - 7 + n % 15) & 511, cr = (r - 7 + n / 15) & 511, px = ci & 1, pz = cr & 1;
        const int col = (ci >> 1) + (px ? dx0 : 0), row = (cr >> 1) + (pz ? izb : iza);
        const float *T = sd.x.tab + (px * 2 + pz) * 128;
        float s = 0.f;
        #pragma unroll
        for (int c = 0; c < 8; c++) {
            const uint32_t hc = sd.cw[(col + (c & 1)) & 255] >> ((c & 2) ? 19 : 3);
            s = __fadd_rn(s, T[c * 16 + (sd.P[(hc + uint32_t(row + (c >> 2))) & 255u] & 15)]);
        }
        smp[n] = s;
    }
    __syncwarp();
    float hv = 0.f;
    if (lane < 15)
        #pragma unroll
        for (int d = 0; d < 15; d++) hv = __fmaf_rn(tp.k[d], smp[lane * 15 + d], hv);
    float o = 0.f;
    #pragma unroll
    for (int d = 0; d < 15; d++) o = __fmaf_rn(tp.k[d], __shfl_sync(0xffffffffu, hv, d), o);
    __syncwarp();
    return __fmul_rn(o, tp.norm);
}

// Maxima of a seed whose columns are split over CTAs (floats in unsigned order) and the CTAs that have added theirs; all
// zero between launches.
struct SplitMax { uint32_t top[2], arrived, pad; };
__device__ __forceinline__ uint32_t order_float(float v) { const uint32_t b = __float_as_uint(v); return b >> 31 ? ~b : b | 0x80000000u; }
__device__ __forceinline__ float unorder_float(uint32_t o) { return __uint_as_float(o >> 31 ? o & 0x7fffffffu : ~o); }
constexpr int FG_SPLIT = 4;
// One CTA per seed; a warp holds FG_ZL rows per lane of one side and row parity (rows 2 (lane + 32 q) + parity).
// A launch of few seeds takes the time of one (about 90 us, one SM's work).  While FG_SPLIT CTAs per seed fit the grid,
// each therefore takes a quarter of the columns (and the blur's run-in before them), evaluates its own exact cells,
// and the last to arrive decides: 47 seeds 100 -> 60 us.  split (may be null: never split) holds gridDim.x / FG_SPLIT entries.
__global__ void __launch_bounds__(FG_THREADS, DSG_FG_MINBLOCKS)
k_fullgate(const Oct *__restrict__ oct, const uint64_t *__restrict__ seeds, const uint32_t *__restrict__ idx, const uint32_t *__restrict__ n_in,
           uint32_t cap_in, float thr, const __grid_constant__ Taps512 tp, uint64_t *__restrict__ out_seed, float *__restrict__ out_amp,
           uint32_t *__restrict__ n_out, uint32_t cap_out, float *__restrict__ side_amp, SplitMax *__restrict__ split) {
    constexpr int W = 2 * FG_WARPS;                             // warps per side
    __shared__ __align__(16) Side512 sides[2];
    __shared__ float sTop[2][2 * W], sAmp[2 * W];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, side = warp / W, wi = warp % W, pz = wi / FG_WARPS, zh = wi % FG_WARPS;
    const int t = threadIdx.x % FG_SIDE;
    Side512 &sd = sides[side];
    const uint32_t n = min(*n_in, cap_in);
    const float floor0 = thr > 0.4f ? 0.44f * thr : AMP_FLOOR;
    int it = 0;
    const bool parts = split && n * FG_SPLIT <= gridDim.x;       // n is at most the survivor capacity: no overflow
    for (uint32_t unit = blockIdx.x; unit < (parts ? n * FG_SPLIT : n); unit += gridDim.x) {
        const uint32_t s = parts ? unit / FG_SPLIT : unit;
        // lattice columns: the run-in from jb, cells from jb + 7 to je - 1
        const int jb = parts ? 1 + int(unit % FG_SPLIT) * (256 / FG_SPLIT) : 1, je = parts ? jb + 7 + 256 / FG_SPLIT : FG_COLS;
        const Oct &p = oct[2 * size_t(idx ? idx[s] : s) + side];
        __syncthreads();                                         // the previous seed's cells are done with the shared arrays
        if (t < 16) reinterpret_cast<uint4 *>(sd.P)[t] = reinterpret_cast<const uint4 *>(p.perm)[t];
        const double ox = p.ox, oz = p.oz;
        const int iy = p.iy, ixa = int(floor(ox)), dx0 = int(floor(0.5 + ox)) - ixa, iza = int(floor(oz)), izb = int(floor(0.5 + oz)), dz0 = izb - iza;
        if (t >= 32 && t < 52) {
            // taps of row parity q on lattice row (t - 4): blur taps d times the corner weights of row q + d
            const int q = (t - 32) / 10, slot = (t - 32) % 10;
            double vb = 0, vc = 0, f[2], tz[2];
            #pragma unroll
            for (int h = 0; h < 2; h++) { const double b = 0.5 * h + oz; f[h] = b - floor(b); tz[h] = fade_fused(f[h]); }
            #pragma unroll
            for (int d = -7; d <= 7; d++) {
                const int pos = q + d, h = pos & 1, l = ((pos - h) >> 1) + (h ? dz0 : 0), dz = slot - 4 - l;
                if (dz != 0 && dz != 1) continue;
                const double wz = double(tp.k[d + 7]) * double(tp.norm) * (dz ? tz[h] : 1 - tz[h]);
                vb += wz; vc += wz * (f[h] - dz);
            }
            sd.bz[q][slot] = float(vb); sd.cz[q][slot] = float(vc);
        }
        // x corners of the two grid columns a lattice column completes: the first is parity 1 when that parity's
        // lattice index runs ahead (dx0), else parity 0
        float a[2][2], b[2][2];                                  // [first, second][corner]
        #pragma unroll
        for (int h = 0; h < 2; h++) {
            const int q = h ^ dx0;                               // the parity completed first (0) and second (1)
            const double o = 0.5 * q + ox, f = o - floor(o), tx = fade_fused(f);
            a[h][0] = float((1 - tx) * f); a[h][1] = float(tx * (f - 1)); b[h][0] = float(1 - tx); b[h][1] = float(tx);
        }
        __syncthreads();
        for (int j = t; j < FG_COLS; j += FG_SIDE) {
            const int pc = sd.P[(ixa + j) & 255] + iy;
            sd.cw[j] = uint32_t(sd.P[pc & 255]) << 3 | uint32_t(sd.P[(pc + 1) & 255]) << 19;
        }
        float *gx = reinterpret_cast<float *>(&sd.a.uv[0][0][256]), *gy = gx + 256, *gz = reinterpret_cast<float *>(&sd.a.uv[0][1][256]);
        grad_rows(sd.P, gx, gy, gz, t, FG_SIDE);
        __syncthreads();
        {
            const float w0 = float(tp.w * (1 - p.vy)), w1 = float(tp.w * p.vy), fy = float(p.fy);
            const int q = t / (FG_SIDE / 2);
            float tb[10], tc[10];
            #pragma unroll
            for (int k = 0; k < 10; k++) { tb[k] = sd.bz[q][k]; tc[k] = sd.cz[q][k]; }
            #pragma unroll 1
            for (int e = t % (FG_SIDE / 2); e < 256; e += FG_SIDE / 2)
                uv_entry<10>(gx, gy, gz, tb, tc, e - 4 + iza, w0, w1, fy, sd.a.uv[q][0][e], sd.a.uv[q][1][e]);
        }
        __syncthreads();
        for (int e = t; e < 1024; e += FG_SIDE) { f2 *u = sd.a.uv[e >> 9][(e >> 8) & 1]; u[(e & 255) + 256] = u[e & 255]; }
        __syncthreads();
        const int row0 = lane + 32 * FG_ZL * zh;
        const char *uv0 = reinterpret_cast<const char *>(&sd.a.uv[pz][0][row0]), *uv1 = reinterpret_cast<const char *>(&sd.a.uv[pz][1][row0]);
        float start = parts ? -1e9f : floor0;                    // a part cannot drop the seed: it lists without a floor
        for (;;) {
            Run r{-1e9f, start, 0};
            float acc[2][FG_ZL], pend[14][FG_ZL];                // pend: a ring, as in k_amp256, two steps per column
            #pragma unroll
            for (int q = 0; q < FG_ZL; q++)
                #pragma unroll
                for (int j = 0; j < 14; j++) pend[j][q] = 0.f;
            const auto column = [&](int J, float (&U)[FG_ZL], float (&V)[FG_ZL]) {
                const uint32_t w = sd.cw[J];
                const char *p0 = uv0 + (w & 0xffffu), *p1 = uv1 + (w >> 16);
                #pragma unroll
                for (int q = 0; q < FG_ZL; q++)
                    unpack2(add2(*reinterpret_cast<const f2 *>(p0 + 256 * q), *reinterpret_cast<const f2 *>(p1 + 256 * q)), U[q], V[q]);
            };
            {
                float U[FG_ZL], V[FG_ZL];
                column(jb - 1, U, V);
                #pragma unroll
                for (int h = 0; h < 2; h++)
                    #pragma unroll
                    for (int q = 0; q < FG_ZL; q++) acc[h][q] = __fmaf_rn(a[h][0], U[q], b[h][0] * V[q]);
            }
            #pragma unroll 1
            for (int J0 = jb; J0 < je; J0 += 7) {
                #pragma unroll
                for (int ph = 0; ph < 7; ph++) {
                    if ((ph == (FG_COLS - 1) % 7 || ph == (7 + 256 / FG_SPLIT) % 7) && J0 + ph == je) break;
                    float U[FG_ZL], V[FG_ZL];
                    column(J0 + ph, U, V);
                    // column J completes samples 2 J - 2 - dx0 and the next: two blur steps
                    #pragma unroll
                    for (int h = 0; h < 2; h++) {
                        Cells<FG_ZL> c;
                        #pragma unroll
                        for (int q = 0; q < FG_ZL; q++) {
                            const int at = 2 * ph + h;
                            const float S = __fmaf_rn(a[h][1], U[q], __fmaf_rn(b[h][1], V[q], acc[h][q]));
                            acc[h][q] = __fmaf_rn(a[h][0], U[q], b[h][0] * V[q]);
                            c.v[q] = __fmaf_rn(tp.k[14], S, pend[at][q]);
                            #pragma unroll
                            for (int j = 1; j < 14; j++) { float &t = pend[(at + j) % 14][q]; t = __fmaf_rn(tp.k[14 - j], S, t); }
                            pend[at][q] = tp.k[0] * S;
                        }
                        float mx = c.v[0];
                        #pragma unroll
                        for (int q = 1; q < FG_ZL; q++) mx = fmaxf(mx, c.v[q]);
                        if (__any_sync(0xffffffffu, mx > r.lim) && J0 + ph >= jb + 7)
                            r = list_cells<FG_ZL>(c, uint32_t((2 * (J0 + ph) - 9 - dx0 + h) & 511) << 9 | uint32_t(2 * row0 + pz), 64u, &sd.list[wi], r, lane);
                    }
                }
            }
            const float best = r.best;
            const int nl = r.n;
            const int par = it++ & 1;
            if (lane == 0) sTop[par][warp] = best;
            __syncthreads();
            float top[2] = {-1e9f, -1e9f};
            #pragma unroll
            for (int k = 0; k < 2 * W; k++) top[k / W] = fmaxf(top[k / W], sTop[par][k]);
            const float ok = start + AMP_E2;                     // as in k_amp256
            if (!parts && double(fmaxf(top[0], ok)) + double(fmaxf(top[1], ok)) + double(AMP_E2) < double(thr)) break;
            if (top[0] < ok || top[1] < ok) { start = -1e9f; continue; }
            corner_tables512(p, tp.w, sd.x.tab, t);
            __syncthreads();
            const float cut = top[side] - AMP_E2;
            float m = -1e9f;
            const bool every = nl > AMP_CAP;                     // this warp's cells: columns (a part: all of them) x the rows of its lanes
            for (int c = 0; c < (every ? 512 * 32 * FG_ZL : nl); c++) {
                if (!every && sd.list[wi].val[c] < cut) continue;
                const uint32_t pos = every ? uint32_t(c / (32 * FG_ZL)) << 9 | uint32_t(2 * (c % (32 * FG_ZL) + 32 * FG_ZL * zh) + pz) : sd.list[wi].pos[c];
                m = fmaxf(m, exact_cell512(sd, sd.x.smp[wi], tp, dx0, iza, izb, int(pos >> 9), int(pos & 511u), lane));
            }
            if (lane == 0) sAmp[warp] = m;
            __syncthreads();
            if (threadIdx.x == 0) {
                float ma = -1e9f, mb = -1e9f;
                #pragma unroll
                for (int k = 0; k < W; k++) { ma = fmaxf(ma, sAmp[k]); mb = fmaxf(mb, sAmp[W + k]); }
                if (parts) {
                    SplitMax &x = split[s];
                    atomicMax(&x.top[0], order_float(ma)); atomicMax(&x.top[1], order_float(mb));
                    __threadfence();
                    if (atomicAdd(&x.arrived, 1u) != FG_SPLIT - 1) break;
                    __threadfence();
                    ma = unorder_float(atomicExch(&x.top[0], 0u)); mb = unorder_float(atomicExch(&x.top[1], 0u));
                    x.arrived = 0;
                }
                const float amp = __fadd_rn(ma, mb);
                if (side_amp) { side_amp[2 * size_t(s)] = ma; side_amp[2 * size_t(s) + 1] = mb; }
                if (amp >= thr) {
                    const uint32_t i = atomicAdd(n_out, 1u);
                    if (i < cap_out) { out_seed[i] = seeds[s]; out_amp[i] = amp; }
                }
            }
            break;
        }
    }
}

}  // namespace gate
}  // namespace dsg
