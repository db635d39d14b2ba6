// Worldgen tables on the device (biome tree, parameter intervals, depth-0 surface grid, terrain spline,
// proxy probability table) and the lookups that use them: surface grid lookup, exact tree classify and the
// terrain-offset spline (src/surface.hpp:12-71, src/standalone.hpp:154-196).  Header-only device code,
// shared by every kernel that classifies climate points.
#pragma once
#include <cstdint>

namespace dsg {

struct SplineDev { int32_t axis, n; float value; float knot[12], slope[12]; int32_t kid[12]; };
// The same graph as a table of its inner nodes, for warps that evaluate it together from shared memory: per node the
// axis and knot count, the knots (ascending), slopes, and each knot's child: an inner node, or -1 and the leaf's value.
// Node 0 is the root; at most four levels of inner nodes.
constexpr int kSplineInner = 37, kSplineLevels = 4;
struct alignas(16) SplineTab {
    float knot[kSplineInner][12], slope[kSplineInner][12], leaf[kSplineInner][12];
    int32_t kid[kSplineInner][12];
    int32_t axis_n[40];                                  // axis | n << 8
};
// What a block keeps in shared memory for the exact searches: the spline, and the candidate grid's cuts per axis (T, H,
// C, E, W; padded with INT32_MAX) and its cells per axis.
struct alignas(16) ExactTab {
    SplineTab spline;
    int32_t cut[5][48];
    int32_t dim[8];
};
static_assert(sizeof(ExactTab) % 16 == 0, "ExactTab is copied in 16-byte words");

// Passed to kernels by value (it lives in the parameter constant bank); the large arrays are in HBM/L2.
struct WorldDev {
    const int16_t *cells;        // surface grid: biome id per grid cell, -1 = ambiguous (tree decides)
    const uint64_t *tree;        // biome tree nodes
    const int32_t *param;        // interval k = [param[2k], param[2k+1]]
    const int4 *nbox;            // box of node k, its six intervals unpacked: nbox[3k..3k+2] = lo[0..5], hi[0..5]
    const SplineDev *spl;        // terrain-offset spline graph (node 0 is the root)
    const ExactTab *exact;       // tables of the exact searches, for groups of lanes
    const float *prob;           // 40 x 40 proxy desert probability (row = C bin, column = E bin)
    const uint32_t *cand_off;    // candidate leaves of candidate-grid cell f: cand[cand_off[f] ..] (cand_n[f] of them)
    const uint16_t *cand;        // tree node indices, ascending within a cell
    const uint16_t *cand_n;
    int32_t ntree, nspl, nparam;
    int32_t strides[8];
    int32_t dim[5];              // grid cells per axis (T, H, C, E, W)
    int32_t ncut[5];             // cut planes per axis (= dim + 1)
    int32_t cut[5][32];          // sorted cut planes per axis
    int32_t cdim[5], nccut[5];   // candidate grid: the surface cuts and extra temperature cuts above the
    int32_t ccut[5][48];         //   surface grid
};
const WorldDev &world_dev();     // valid after dsg_init

#ifdef __CUDACC__
// Cell of q in the surface grid, axes T, H, C, E, W, each cell the half-open range [cut_k, cut_k+1): false when q
// lies outside the grid.  on_cut: a coordinate equals a cut plane.  (A climate value times 10,000 fits an int32:
// the octave amplitudes of every channel sum to less than 10.)
__device__ __forceinline__ bool grid_locate(const WorldDev &w, const int32_t *q, uint32_t &flat, bool &on_cut) {
    constexpr int AX[5] = {0, 1, 2, 3, 5};
    uint32_t f = 0;
    on_cut = false;
    #pragma unroll
    for (int a = 0; a < 5; a++) {
        const int32_t v = q[AX[a]];
        const int32_t *c = w.cut[a];
        const int nc = w.ncut[a];
        if (v < c[0] || v >= c[nc - 1]) return false;
        int lo = 0, hi = nc;                       // first cut > v (upper_bound)
        while (lo < hi) { const int mid = (lo + hi) >> 1; if (c[mid] <= v) lo = mid + 1; else hi = mid; }
        const int idx = lo - 1;
        on_cut |= v == c[idx];
        f = f * uint32_t(w.dim[a]) + uint32_t(idx);
    }
    flat = f;
    return true;
}
// Surface grid lookup (surface.hpp:58-70): the biome of the depth-0 surface box containing q, or -1 when q
// lies outside the grid, on a cut plane, or in a cell that is ambiguous.
__device__ __forceinline__ int grid_lookup(const WorldDev &w, const int32_t *q) {
    uint32_t f; bool on_cut;
    if (!grid_locate(w, q, f, on_cut) || on_cut) return -1;
    return w.cells[f];
}
__device__ __forceinline__ uint64_t box_dist(const WorldDev &w, int node, const int32_t *v) {
    const int4 a = __ldg(&w.nbox[3 * node]), b = __ldg(&w.nbox[3 * node + 1]), c = __ldg(&w.nbox[3 * node + 2]);
    const int32_t lo[6] = {a.x, a.y, a.z, a.w, b.x, b.y}, hi[6] = {b.z, b.w, c.x, c.y, c.z, c.w};
    uint64_t sum = 0;
    #pragma unroll
    for (int i = 0; i < 6; i++) {
        const uint32_t d = uint32_t(max(max(lo[i] - v[i], v[i] - hi[i]), 0));
        sum += uint64_t(d) * d;
    }
    return sum;
}
// Exact nearest-box search of the biome tree (standalone.hpp:182-196), with an explicit stack in place of
// the recursion.  Children are visited in order and pruned against the running best distance exactly as
// the recursive form does (the prune test is made when a child is reached, against the best distance at
// that moment).  A node's children's distances do not depend on the search state, so they are computed
// together when the node is entered: their box loads are independent and overlap, where visiting them one
// by one would wait on two dependent loads per child.
__device__ inline int tree_classify(const WorldDev &w, const int32_t *v) {
    struct Frame { int level, child0, stride, n, i; uint64_t d[6]; };
    Frame stk[8];
    int sp = 0, best = 0;
    uint64_t bestd = ~0ull, dnode = 0;
    // enter(node, level): leaf -> compare; inner -> push a frame with its children's distances
    int node = 0, level = 0;
    for (;;) {
        bool descended = false;
        const uint64_t e = __ldg(&w.tree[node]);
        if ((e >> 56) == 255) {
            if (dnode < bestd) { bestd = dnode; best = node; }
        } else if (sp < 8) {                       // tree depth is 6; the bound only guards the array
            int stride, lv = level;
            do { stride = w.strides[lv & 7]; lv++; } while (node + stride >= w.ntree && lv < 8);
            Frame &f = stk[sp++];
            f.level = lv; f.child0 = int(e >> 48); f.stride = stride; f.i = 0; f.n = 0;
            #pragma unroll
            for (int j = 0; j < 6; j++)
                if (f.child0 + j * stride < w.ntree) { f.d[j] = box_dist(w, f.child0 + j * stride, v); f.n = j + 1; }
        }
        // advance the innermost frame to its next child that passes the prune test
        while (sp > 0) {
            Frame &f = stk[sp - 1];
            bool found = false;
            while (f.i < f.n) {
                const int j = f.i++;
                if (f.d[j] < bestd) { node = f.child0 + j * f.stride; dnode = f.d[j]; level = f.level; found = true; break; }
            }
            if (found) { descended = true; break; }
            sp--;
        }
        if (!descended) break;
    }
    return int((__ldg(&w.tree[best]) >> 48) & 255);
}
// Cell of q in the candidate grid (half-open cells as in grid_locate); false outside it.
__device__ __forceinline__ bool cand_locate(const WorldDev &w, const int32_t *q, uint32_t &flat) {
    constexpr int AX[5] = {0, 1, 2, 3, 5};
    uint32_t f = 0;
    #pragma unroll
    for (int a = 0; a < 5; a++) {
        const int32_t v = q[AX[a]];
        const int32_t *c = w.ccut[a];
        const int nc = w.nccut[a];
        if (v < c[0] || v >= c[nc - 1]) return false;
        int lo = 0, hi = nc;
        while (lo < hi) { const int mid = (lo + hi) >> 1; if (c[mid] <= v) lo = mid + 1; else hi = mid; }
        f = f * uint32_t(w.cdim[a]) + uint32_t(lo - 1);
    }
    flat = f;
    return true;
}
// Exact nearest leaf (the reference's tree search, standalone.hpp:182-196): the (box distance, node index)
// minimum over the candidate leaves of the point's candidate-grid cell.  Below the root every box contains
// its children's boxes, so the pruned depth-first search returns exactly that minimum over all leaves; the
// candidates of a cell are every leaf that can attain it for some point of the cell and any depth
// (world_upload drops a leaf only when a leaf of the same depth interval is nearer everywhere in the cell, by
// bounds of the whole cell and by pairwise comparison).
// Points outside the candidate grid (rare: humidity beyond the surface boxes, T > 2, or C, E, W more than 1.0
// past them) take the tree search itself.
// Four candidates at a time: their boxes load together.
__device__ inline int classify_exact(const WorldDev &w, const int32_t *v) {
    uint32_t f;
    if (!cand_locate(w, v, f)) return tree_classify(w, v);
    uint64_t bestd = ~0ull;
    int best = 0;
    for (uint32_t k = __ldg(&w.cand_off[f]), e = k + __ldg(&w.cand_n[f]); k < e; k += 4) {
        int node[4];
        uint64_t d[4];
        #pragma unroll
        for (int i = 0; i < 4; i++) node[i] = __ldg(&w.cand[min(k + i, e - 1)]);
        #pragma unroll
        for (int i = 0; i < 4; i++) d[i] = box_dist(w, node[i], v);
        #pragma unroll
        for (int i = 0; i < 4; i++) if (d[i] < bestd) { bestd = d[i]; best = node[i]; }
    }
    return int((__ldg(&w.tree[best]) >> 48) & 255);
}
// Terrain-offset spline (standalone.hpp:154-169) with an explicit stack.  The float/double mix of the
// interpolation follows the reference expression by expression.
__device__ inline float spline_eval(const WorldDev &w, const float *v) {
    struct Frame { int node, lo, stage; float x, t, width, a; };
    Frame stk[8];
    int sp = 0;
    float ret = 0.f;
    int node = 0;
    for (;;) {
        // evaluate `node`: leaf values return immediately; inner nodes push a frame
        const SplineDev &s = w.spl[node];
        bool pushed = false;
        if (s.n == 0) ret = s.value;
        else {
            const float x = v[s.axis];
            int hi = 0;
            while (hi < s.n && x > s.knot[hi]) hi++;
            if (sp >= 8) { ret = s.value; }            // spline depth is 4; the bound only guards the array
            else if (hi == 0 || hi == s.n) {
                const int j = hi == 0 ? 0 : s.n - 1;
                stk[sp++] = {node, j, 0, x, 0.f, 0.f, 0.f};      // stage 0: extrapolate from child j
                node = s.kid[j]; pushed = true;
            } else {
                const int lo = hi - 1;
                const float width = __fsub_rn(s.knot[hi], s.knot[lo]);
                const float t = __fdiv_rn(__fsub_rn(x, s.knot[lo]), width);
                stk[sp++] = {node, lo, 1, x, t, width, 0.f};      // stage 1: need child lo, then child hi
                node = s.kid[lo]; pushed = true;
            }
        }
        if (pushed) continue;
        // unwind with ret = value of the node just evaluated
        bool next = false;
        while (sp > 0) {
            Frame &f = stk[sp - 1];
            const SplineDev &p = w.spl[f.node];
            if (f.stage == 0) {
                ret = __fadd_rn(ret, __fmul_rn(p.slope[f.lo], __fsub_rn(f.x, p.knot[f.lo])));
                sp--;
            } else if (f.stage == 1) {
                f.a = ret; f.stage = 2; node = p.kid[f.lo + 1]; next = true; break;
            } else {
                const float a = f.a, b = ret, t = f.t, width = f.width;
                const float dba = __fsub_rn(b, a);
                const float pp = __fsub_rn(__fmul_rn(p.slope[f.lo], width), dba);
                const float qq = __fadd_rn(__fmul_rn(-p.slope[f.lo + 1], width), dba);
                const double lin = __dadd_rn(double(a), __dmul_rn(double(t), __dsub_rn(double(b), double(a))));
                const double cur = __dadd_rn(double(pp), __dmul_rn(double(t), __dsub_rn(double(qq), double(pp))));
                ret = float(__dadd_rn(lin, __dmul_rn(double(__fmul_rn(t, __fsub_rn(1.f, t))), cur)));
                sp--;
            }
        }
        if (!next) break;
    }
    return ret;
}

// ---------------------------------------------------------------- eight lanes per point
// The two searches of a pending desert point by a group of 8 lanes (four points per warp; the whole warp calls, groups
// without a point with `on` false).  One thread evaluating the spline follows up to 15 inner nodes one after another,
// each a chain of dependent loads, a division and a double-precision combination (12,400 cycles on average, 76,000 at
// worst, where the lanes' paths diverged); the group takes the nodes of a level side by side, and no lane branches:
// four levels down, four up.
struct SplineStep { float t, width, slo, shi, ext, val; int mode; };      // mode 0: leaf (val), 1: extrapolation, 2: interpolation
__device__ __forceinline__ float spline_combine(const SplineStep &s, float a, float b) {
    const float dba = __fsub_rn(b, a);
    const float pp = __fsub_rn(__fmul_rn(s.slo, s.width), dba);
    const float qq = __fadd_rn(__fmul_rn(-s.shi, s.width), dba);
    const double lin = __dadd_rn(double(a), __dmul_rn(double(s.t), __dsub_rn(double(b), double(a))));
    const double cur = __dadd_rn(double(pp), __dmul_rn(double(s.t), __dsub_rn(double(qq), double(pp))));
    const float in = float(__dadd_rn(lin, __dmul_rn(double(__fmul_rn(s.t, __fsub_rn(1.f, s.t))), cur)));
    const float ex = __fadd_rn(a, __fmul_rn(s.slo, s.ext));
    return s.mode == 2 ? in : s.mode == 1 ? ex : s.val;
}
// Terrain offset at v (standalone.hpp:154-169, the expressions of spline_eval); T in shared memory.  Lane g of the group
// holds node g of each level; every lane returns the value.
__device__ __forceinline__ float spline_group(const SplineTab &T, float v0, float v1, float v2, float v3) {
    const int lane = threadIdx.x & 31, g = lane & 7, base = lane & 24;
    SplineStep st[kSplineLevels];
    int node = 0;                                        // inner node, or -1: leaf of value val
    float val = 0.f, la = 0.f, lb = 0.f;
    #pragma unroll
    for (int L = 0; L < kSplineLevels; L++) {
        const int k = max(node, 0), an = T.axis_n[k], n = an >> 8, axis = an & 255;
        const float x = axis == 0 ? v0 : axis == 1 ? v1 : axis == 2 ? v2 : v3;
        int hi = 0;
        #pragma unroll
        for (int j = 0; j < 3; j++) {
            const float4 q = reinterpret_cast<const float4 *>(T.knot[k])[j];
            hi += (4 * j < n && x > q.x) + (4 * j + 1 < n && x > q.y) + (4 * j + 2 < n && x > q.z) + (4 * j + 3 < n && x > q.w);
        }
        const bool ext = hi == 0 || hi == n;
        const int lo = ext ? (hi == 0 ? 0 : n - 1) : hi - 1, up = ext ? lo : hi;
        const float klo = T.knot[k][lo];
        SplineStep &s = st[L];
        s.mode = node < 0 ? 0 : ext ? 1 : 2;
        s.val = val;
        s.slo = T.slope[k][lo]; s.shi = T.slope[k][up];
        s.ext = __fsub_rn(x, klo);
        s.width = ext ? 1.f : __fsub_rn(T.knot[k][up], klo);
        s.t = __fdiv_rn(s.ext, s.width);
        const int ka = T.kid[k][lo], kb = T.kid[k][up];
        la = T.leaf[k][lo]; lb = T.leaf[k][up];
        if (L + 1 < kSplineLevels) {                     // lane g of the next level is child g & 1 of lane g / 2
            const int src = base + (g >> 1);
            const int na = __shfl_sync(0xffffffffu, ka, src), nb = __shfl_sync(0xffffffffu, kb, src);
            const float fa = __shfl_sync(0xffffffffu, la, src), fb = __shfl_sync(0xffffffffu, lb, src);
            node = (g & 1) ? nb : na; val = (g & 1) ? fb : fa;
        }
    }
    float r = spline_combine(st[kSplineLevels - 1], la, lb);
    #pragma unroll
    for (int L = kSplineLevels - 2; L >= 0; L--) {
        const float a = __shfl_sync(0xffffffffu, r, base + ((2 * g) & 7)), b = __shfl_sync(0xffffffffu, r, base + ((2 * g + 1) & 7));
        r = spline_combine(st[L], a, b);
    }
    return __shfl_sync(0xffffffffu, r, base);
}
// classify_exact by the group, in two parts, so that its chain of loads overlaps the spline that gives the depth (the
// candidate grid has no depth axis): classify_group_begin finds the point's cell (lane g counts axis g's cuts) and
// loads the lane's first candidate, classify_group_end adds the depth's share of the distances and takes the smallest
// (distance, node) of all candidates, eight at a time.
struct GroupSearch { uint32_t k, end; bool in; int node, biome, lo, hi; uint64_t dist; };
__device__ __forceinline__ void group_candidate(const WorldDev &w, const int32_t *v, GroupSearch &s) {
    s.node = __ldg(&w.cand[s.k]);
    const int4 a = __ldg(&w.nbox[3 * s.node]), b = __ldg(&w.nbox[3 * s.node + 1]), c = __ldg(&w.nbox[3 * s.node + 2]);
    s.biome = int((__ldg(&w.tree[s.node]) >> 48) & 255);
    const int32_t lo[6] = {a.x, a.y, a.z, a.w, b.x, b.y}, hi[6] = {b.z, b.w, c.x, c.y, c.z, c.w};
    s.dist = 0;
    #pragma unroll
    for (int i = 0; i < 6; i++) {
        if (i == 4) continue;
        const uint32_t d = uint32_t(max(max(lo[i] - v[i], v[i] - hi[i]), 0));
        s.dist += uint64_t(d) * d;
    }
    s.lo = lo[4]; s.hi = hi[4];
}
__device__ __forceinline__ GroupSearch classify_group_begin(const WorldDev &w, const ExactTab &T, const int32_t *v, bool on) {
    const int lane = threadIdx.x & 31, g = lane & 7, base = lane & 24, ax = min(g, 4);
    const int32_t x = ax == 0 ? v[0] : ax == 1 ? v[1] : ax == 2 ? v[2] : ax == 3 ? v[3] : v[5];
    int at = -1;
    #pragma unroll
    for (int j = 0; j < 12; j++) {
        const int4 c = reinterpret_cast<const int4 *>(T.cut[ax])[j];
        at += (c.x <= x) + (c.y <= x) + (c.z <= x) + (c.w <= x);
    }
    const unsigned bad = __ballot_sync(0xffffffffu, at < 0 || at >= T.dim[ax]) >> base & 0xffu;
    uint32_t f = 0;
    #pragma unroll
    for (int a = 0; a < 5; a++) f = f * uint32_t(T.dim[a]) + uint32_t(__shfl_sync(0xffffffffu, at, base + a));
    GroupSearch s{0, 0, on && !bad, 0, 0, 0, 0, 0};
    if (s.in) {
        const uint32_t k0 = __ldg(&w.cand_off[f]);
        s.end = k0 + __ldg(&w.cand_n[f]); s.k = k0 + g;
        if (s.k < s.end) group_candidate(w, v, s);
    }
    return s;
}
__device__ __forceinline__ int classify_group_end(const WorldDev &w, const int32_t *v, bool on, GroupSearch s) {
    const int lane = threadIdx.x & 31, g = lane & 7, base = lane & 24;
    unsigned long long key = ~0ull;                      // distance (below 2^35), node (below 2^16), biome (8 bits)
    while (s.in && s.k < s.end) {
        const uint32_t d = uint32_t(max(max(s.lo - v[4], v[4] - s.hi), 0));
        key = min(key, (unsigned long long)(s.dist + uint64_t(d) * d) << 24 | (unsigned long long)s.node << 8 | uint32_t(s.biome));
        s.k += 8;
        if (s.k < s.end) group_candidate(w, v, s);
    }
    int biome = 0;
    if (on && !s.in && g == 0) biome = tree_classify(w, v);
    __syncwarp();
    #pragma unroll
    for (int o = 4; o > 0; o >>= 1) key = min(key, __shfl_xor_sync(0xffffffffu, key, o));
    biome = __shfl_sync(0xffffffffu, biome, base);
    return s.in ? int(key & 255) : biome;
}
#endif

}  // namespace dsg
