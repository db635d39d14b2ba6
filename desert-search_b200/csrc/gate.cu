// Seed gate (stage S0) for sm_100a: y-phase filter -> anti-aliased 256^2 amplitude pre-gate -> full 512^2
// amplitude gate.  Restates src/gpu/gate.cuh (k_phase, k_init, k_amp2) with the same per-cell arithmetic
// (summation orders, fused multiply-adds of the blur chains, device expf taps), so amplitudes match the
// reference's GPU gate bit for bit, on a different schedule: the amplitude kernels (gate_amp.cuh) screen every
// cell with a cheaper expression of the same number and evaluate the reference's chain where the maximum can be.
// The whole batch (phase -> init -> pre-gate -> full gate) runs from device-side counts: no host sync
// between stages, so a batch can be captured in a CUDA graph.
#include "common.cuh"
#include "gate_amp.cuh"
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

namespace dsg {
namespace gate {

__device__ __forceinline__ double phase_of(uint64_t seed, double *fy = nullptr) {
    Xoro w = Xoro::seeded(seed);
    const uint64_t a = w.next(), b = w.next();
    Xoro c{a ^ kTempA, b ^ kTempB};
    double s = 0;
    #pragma unroll
    for (int side = 0; side < 2; side++) {
        const uint64_t fa = c.next(), fb = c.next();
        Xoro r{fa ^ kSalt10A, fb ^ kSalt10B};
        r.next();
        const double y = r.uniform() * 256.;
        const double f = y - floor(y);
        if (fy) fy[side] = f;
        s += fabs(f - .5);
    }
    return s;
}

// ---------------------------------------------------------------- kernels
// y-phase filter over seed indices [start, start + count): warp-aggregated append of passing seeds.
__global__ void __launch_bounds__(256) k_phase(uint64_t start, uint64_t count, double maxph, uint64_t *__restrict__ out,
                                                uint32_t *__restrict__ nout, uint32_t cap) {
    const int lane = threadIdx.x & 31;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t base = uint64_t(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u); base < count; base += stride) {
        const uint64_t k = base + lane;
        const uint64_t seed = fmix64(start + k);
        const bool pass = k < count && phase_of(seed) <= maxph;
        const uint32_t m = __ballot_sync(0xffffffffu, pass);
        if (m) {
            uint32_t at = 0;
            if (lane == __ffs(m) - 1) at = atomicAdd(nout, uint32_t(__popc(m)));
            at = __shfl_sync(0xffffffffu, at, __ffs(m) - 1);
            if (pass) {
                const uint32_t i = at + __popc(m & ((1u << lane) - 1));
                if (i < cap) out[i] = seed;
            }
        }
    }
}
__global__ void k_phase_list(const uint64_t *__restrict__ seeds, uint32_t n, double *__restrict__ ph, double *__restrict__ fy) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { double f[2]; ph[i] = phase_of(seeds[i], f); fy[2 * i] = f[0]; fy[2 * i + 1] = f[1]; }
}

// Temperature octave -10 of both sides of every listed seed (gate.cuh:59-70, k_init).
constexpr int OCT_THREADS = 64;
__global__ void __launch_bounds__(OCT_THREADS) k_octinit(const uint64_t *__restrict__ seeds, const uint32_t *__restrict__ n_in, uint32_t cap,
                                                  Oct *__restrict__ oct) {
    __shared__ uint8_t perm[256][OCT_THREADS];            // a column per thread
    const uint32_t n = min(*n_in, cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * n; i += gridDim.x * blockDim.x) {
        const uint64_t seed = seeds[i >> 1];
        const int side = int(i & 1);
        Xoro w = Xoro::seeded(seed);
        const uint64_t a = w.next(), b = w.next();
        Xoro c{a ^ kTempA, b ^ kTempB};
        uint64_t fa = c.next(), fb = c.next();
        if (side) { fa = c.next(); fb = c.next(); }
        Xoro r{fa ^ kSalt10A, fb ^ kSalt10B};
        const double ox = r.uniform() * 256, oy = r.uniform() * 256, oz = r.uniform() * 256;
        uint8_t *p = &perm[0][threadIdx.x];
        shuffle_column<OCT_THREADS>(r, p);
        Oct &o = oct[i];
        #pragma unroll 2
        for (int k = 0; k < 16; k++) reinterpret_cast<uint4 *>(o.perm)[k] = column_words<OCT_THREADS>(p, k);
        const double fl = floor(oy);
        o.ox = ox; o.oz = oz; o.fy = oy - fl; o.vy = fade_fused(oy - fl); o.iy = int(fl);
    }
}

__global__ void k_iota(uint32_t *a, uint32_t n) { const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; if (i < n) a[i] = i; }

// ---------------------------------------------------------------- host side
void gate_taps_device(float out[24]);                     // taps.cu
// The gate's constants from the device taps (9 for sigma 1, then 15 for sigma 2).
void gate_taps(const float raw[24], Taps256 &a, Taps512 &b) {
    float s9 = 0, s15 = 0;
    for (int i = 0; i < 9; i++) { a.k[i] = raw[i]; s9 += raw[i]; }
    for (int i = 0; i < 15; i++) { b.k[i] = raw[9 + i]; s15 += raw[9 + i]; }
    a.norm = 1.f / (s9 * s9); b.norm = 1.f / (s15 * s15);
    a.w = b.w = double(float(1.25 * (32.0 / 63.0) * 1.5));   // octave-0 temperature weight, final units (gate.cuh:47)
}

struct State {
    std::mutex mu;
    bool ready = false;
    Taps256 t256{};                                          // sigma 1, 9 device taps
    Taps512 t512{};                                          // sigma 2, 15 device taps
    float raw[24];
    cudaStream_t st = nullptr;
    // batch buffers
    uint64_t cap_batch = 0;
    uint32_t cap1 = 0, cap2 = 0, cap3 = 0;
    uint64_t *d_s1 = nullptr, *d_s2 = nullptr, *d_s3 = nullptr;
    uint32_t *d_idx2 = nullptr, *d_n = nullptr, *h_n = nullptr;
    float *d_a3 = nullptr;
    Oct *d_oct = nullptr;
    uint64_t *h_s3 = nullptr; float *h_a3 = nullptr;
    int pg_blocks = 0, fg_blocks = 0;
    SplitMax *d_split = nullptr;                             // the full gate's split seeds
};
State &S() { static State s; return s; }

void setup_locked(State &g) {
    if (g.ready) return;
    require_init();
    gate_taps_device(g.raw);
    gate_taps(g.raw, g.t256, g.t512);
    int lo, hi;
    DSG_CU(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    DSG_CU(cudaStreamCreateWithPriority(&g.st, cudaStreamNonBlocking, lo));   // the gate yields to scan/proxy/flood
    int occ = 0;
    DSG_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_amp256<AMP_AA>, PG_THREADS, 0));
    g.pg_blocks = std::max(1, occ) * device_info().sms;
    DSG_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fullgate, FG_THREADS, 0));
    g.fg_blocks = std::max(1, occ) * device_info().sms;
    DSG_CU(cudaMalloc(&g.d_split, size_t(g.fg_blocks / FG_SPLIT + 1) * sizeof(SplitMax)));
    DSG_CU(cudaMemsetAsync(g.d_split, 0, size_t(g.fg_blocks / FG_SPLIT + 1) * sizeof(SplitMax), g.st));
    DSG_CU(cudaStreamSynchronize(g.st));                     // the batches may run on other streams
    g.ready = true;
}
void ensure_buffers(State &g, uint64_t batch) {
    if (batch <= g.cap_batch) return;
    cudaFree(g.d_s1); cudaFree(g.d_s2); cudaFree(g.d_s3); cudaFree(g.d_idx2); cudaFree(g.d_a3); cudaFree(g.d_oct); cudaFree(g.d_n);
    cudaFreeHost(g.h_n); cudaFreeHost(g.h_s3); cudaFreeHost(g.h_a3);
    // caps as run_gate (gate.cuh:364) scaled to the batch: 1/16 of the indices, 1/4 of those, 1/16 of those
    g.cap1 = uint32_t(std::max<uint64_t>(1024, batch / 16));
    g.cap2 = std::max<uint32_t>(1024, g.cap1 / 4);
    g.cap3 = std::max<uint32_t>(1024, g.cap2 / 16);
    DSG_CU(cudaMalloc(&g.d_s1, size_t(g.cap1) * 8));
    DSG_CU(cudaMalloc(&g.d_oct, size_t(g.cap1) * 2 * sizeof(Oct)));
    DSG_CU(cudaMalloc(&g.d_s2, size_t(g.cap2) * 8));
    DSG_CU(cudaMalloc(&g.d_idx2, size_t(g.cap2) * 4));
    DSG_CU(cudaMalloc(&g.d_s3, size_t(g.cap3) * 8));
    DSG_CU(cudaMalloc(&g.d_a3, size_t(g.cap3) * 4));
    DSG_CU(cudaMalloc(&g.d_n, 4 * 4));
    DSG_CU(cudaMallocHost(&g.h_n, 4 * 4));
    DSG_CU(cudaMallocHost(&g.h_s3, size_t(g.cap3) * 8));
    DSG_CU(cudaMallocHost(&g.h_a3, size_t(g.cap3) * 4));
    g.cap_batch = batch;
}
// Enqueue one batch on `st` (no host synchronisation).
void enqueue_batch(State &g, cudaStream_t st, uint64_t start, uint64_t nb, const dsg_gate_cfg &c) {
    DSG_CU(cudaMemsetAsync(g.d_n, 0, 16, st));
    const unsigned pb = unsigned(std::min<uint64_t>((nb + 255) / 256, uint64_t(device_info().sms) * 64));
    k_phase<<<pb, 256, 0, st>>>(start, nb, double(c.maxph), g.d_s1, g.d_n, g.cap1);
    k_octinit<<<unsigned(device_info().sms) * 13, OCT_THREADS, 0, st>>>(g.d_s1, g.d_n, g.cap1, g.d_oct);
    k_amp256<AMP_AA><<<g.pg_blocks, PG_THREADS, 0, st>>>(g.d_oct, g.d_s1, g.d_n, g.cap1, c.pthr, g.t256, g.d_s2, g.d_idx2, g.d_n + 1, g.cap2, nullptr);
    k_fullgate<<<g.fg_blocks, FG_THREADS, 0, st>>>(g.d_oct, g.d_s2, g.d_idx2, g.d_n + 1, g.cap2, c.amp, g.t512, g.d_s3, g.d_a3, g.d_n + 2, g.cap3, nullptr, g.d_split);
    DSG_CU(cudaGetLastError());
}
// A gate with buffers of its own, for the device-resident searcher: batches of up to `batch` indices enqueued
// on the caller's stream.  survivors / counts point at its full-gate list and its counters {phase-passed,
// pre-gate passed, full-gate passed} (counts above the list capacities mean an overflow).
struct Lane { State g; };
Lane *lane_create(uint64_t batch) {
    Lane *l = new Lane;
    setup_locked(l->g);
    ensure_buffers(l->g, batch);
    return l;
}
void lane_enqueue(Lane *l, cudaStream_t st, uint64_t start, uint64_t nb, const dsg_gate_cfg &c) { enqueue_batch(l->g, st, start, nb, c); }
void lane_destroy(Lane *l) {
    if (!l) return;
    State &g = l->g;
    cudaFree(g.d_s1); cudaFree(g.d_s2); cudaFree(g.d_s3); cudaFree(g.d_idx2); cudaFree(g.d_a3); cudaFree(g.d_oct); cudaFree(g.d_n);
    cudaFreeHost(g.h_n); cudaFreeHost(g.h_s3); cudaFreeHost(g.h_a3);
    cudaFree(g.d_split);
    if (g.st) cudaStreamDestroy(g.st);
    delete l;
}
const uint64_t *lane_survivors(const Lane *l) { return l->g.d_s3; }
uint32_t *lane_counts(Lane *l) { return l->g.d_n; }
void lane_caps(const Lane *l, uint32_t caps[3]) { caps[0] = l->g.cap1; caps[1] = l->g.cap2; caps[2] = l->g.cap3; }
}  // namespace gate
}  // namespace dsg

using namespace dsg;
using namespace dsg::gate;

extern "C" int dsg_gate_taps(float taps[24]) {
    return guarded([&] {
        State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
        std::memcpy(taps, g.raw, sizeof g.raw);
        return DSG_OK;
    });
}

extern "C" int dsg_phase(const uint64_t *seeds, uint32_t n, double *phase, double *fy) {
    return guarded([&] {
        require_init();
        DSG_ARG(seeds && phase && fy, "dsg_phase: null pointer");
        if (!n) return DSG_OK;
        uint64_t *d_s; double *d_p, *d_f;
        DSG_CU(cudaMalloc(&d_s, size_t(n) * 8)); DSG_CU(cudaMalloc(&d_p, size_t(n) * 8)); DSG_CU(cudaMalloc(&d_f, size_t(n) * 16));
        DSG_CU(cudaMemcpy(d_s, seeds, size_t(n) * 8, cudaMemcpyHostToDevice));
        k_phase_list<<<(n + 255) / 256, 256>>>(d_s, n, d_p, d_f);
        DSG_CU(cudaGetLastError());
        DSG_CU(cudaMemcpy(phase, d_p, size_t(n) * 8, cudaMemcpyDeviceToHost));
        DSG_CU(cudaMemcpy(fy, d_f, size_t(n) * 16, cudaMemcpyDeviceToHost));
        cudaFree(d_s); cudaFree(d_p); cudaFree(d_f);
        return DSG_OK;
    });
}

extern "C" int dsg_gate_amps(const uint64_t *seeds, uint32_t n, float *pre, float *full) {
    return guarded([&] {
        DSG_ARG(seeds && pre && full, "dsg_gate_amps: null pointer");
        State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
        if (!n) return DSG_OK;
        uint64_t *d_s, *d_o; uint32_t *d_n, *d_i; float *d_pre, *d_full, *d_a; Oct *d_oct;
        DSG_CU(cudaMalloc(&d_s, size_t(n) * 8)); DSG_CU(cudaMalloc(&d_o, size_t(n) * 8)); DSG_CU(cudaMalloc(&d_i, size_t(n) * 4));
        DSG_CU(cudaMalloc(&d_n, 16)); DSG_CU(cudaMalloc(&d_pre, size_t(n) * 8)); DSG_CU(cudaMalloc(&d_full, size_t(n) * 8));
        DSG_CU(cudaMalloc(&d_a, size_t(n) * 4)); DSG_CU(cudaMalloc(&d_oct, size_t(n) * 2 * sizeof(Oct)));
        DSG_CU(cudaMemcpy(d_s, seeds, size_t(n) * 8, cudaMemcpyHostToDevice));
        const uint32_t hn[4] = {n, 0, n, 0};
        DSG_CU(cudaMemcpy(d_n, hn, 16, cudaMemcpyHostToDevice));
        k_octinit<<<(2 * n + OCT_THREADS - 1) / OCT_THREADS, OCT_THREADS>>>(d_s, d_n, n, d_oct);
        k_amp256<AMP_AA><<<g.pg_blocks, PG_THREADS>>>(d_oct, d_s, d_n, n, -1e30, g.t256, d_o, d_i, d_n + 1, n, d_pre);
        k_fullgate<<<g.fg_blocks, FG_THREADS>>>(d_oct, d_s, nullptr, d_n + 2, n, -1e30f, g.t512, d_o, d_a, d_n + 3, n, d_full, nullptr);
        DSG_CU(cudaGetLastError());
        DSG_CU(cudaMemcpy(pre, d_pre, size_t(n) * 8, cudaMemcpyDeviceToHost));
        DSG_CU(cudaMemcpy(full, d_full, size_t(n) * 8, cudaMemcpyDeviceToHost));
        cudaFree(d_s); cudaFree(d_o); cudaFree(d_i); cudaFree(d_n); cudaFree(d_pre); cudaFree(d_full); cudaFree(d_a); cudaFree(d_oct);
        return DSG_OK;
    });
}

extern "C" int dsg_gate_run(uint64_t start, uint64_t count, const dsg_gate_cfg *cfg, uint64_t *out_seed, float *out_amp, uint32_t cap,
                            uint32_t *n_out, uint64_t counts[4]) {
    return guarded([&] {
        DSG_ARG(cfg && n_out, "dsg_gate_run: null pointer");
        DSG_ARG(cap == 0 || (out_seed && out_amp), "dsg_gate_run: null output");
        State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
        const uint64_t B = cfg->batch ? cfg->batch : (1ull << 26);
        ensure_buffers(g, B);
        uint64_t tot[4] = {0, 0, 0, 0};
        uint32_t written = 0;
        bool overflow = false;
        std::vector<std::pair<uint64_t, float>> found;
        for (uint64_t base = 0; base < count; base += B) {
            const uint64_t nb = std::min(B, count - base);
            enqueue_batch(g, g.st, start + base, nb, *cfg);
            // the first survivors come with the counts: a short range needs no second round trip
            const uint32_t few = std::min(g.cap3, 1024u);
            DSG_CU(cudaMemcpyAsync(g.h_n, g.d_n, 16, cudaMemcpyDeviceToHost, g.st));
            DSG_CU(cudaMemcpyAsync(g.h_s3, g.d_s3, size_t(few) * 8, cudaMemcpyDeviceToHost, g.st));
            DSG_CU(cudaMemcpyAsync(g.h_a3, g.d_a3, size_t(few) * 4, cudaMemcpyDeviceToHost, g.st));
            DSG_CU(cudaStreamSynchronize(g.st));
            const uint32_t n1 = g.h_n[0], n2 = g.h_n[1], n3 = g.h_n[2];
            overflow |= n1 > g.cap1 || n2 > g.cap2 || n3 > g.cap3;
            const uint32_t k3 = std::min(n3, g.cap3);
            if (k3 > few) {
                DSG_CU(cudaMemcpyAsync(g.h_s3 + few, g.d_s3 + few, size_t(k3 - few) * 8, cudaMemcpyDeviceToHost, g.st));
                DSG_CU(cudaMemcpyAsync(g.h_a3 + few, g.d_a3 + few, size_t(k3 - few) * 4, cudaMemcpyDeviceToHost, g.st));
                DSG_CU(cudaStreamSynchronize(g.st));
            }
            found.clear();
            for (uint32_t i = 0; i < k3; i++) found.push_back({g.h_s3[i], g.h_a3[i]});
            std::sort(found.begin(), found.end());
            for (auto &f : found) {
                if (written < cap) { out_seed[written] = f.first; out_amp[written] = f.second; written++; }
                else overflow = true;
            }
            tot[0] += nb; tot[1] += n1; tot[2] += n2; tot[3] += n3;
        }
        *n_out = written;
        if (counts) std::memcpy(counts, tot, sizeof tot);
        return overflow ? DSG_OVERFLOW : DSG_OK;
    });
}

// ---- the CPU search's gate: y-phase, then the sub-grid pre-gate estimate (dsearch_desert.cpp:201-223)
namespace dsg { namespace gate {
// taps exp(-d^2/2) rounded to float and normalised by their double sum, on the host as the CPU code computes
// them (lowfield.hpp:86-89); w = factor x weight of the temperature octave -10 (1.25 x (32/63 x 1.5))
Taps256 sub_taps() {
    Taps256 t{};
    double s = 0;
    for (int d = -4; d <= 4; d++) s += t.k[d + 4] = float(std::exp(-0.5 * d * d));
    for (float &v : t.k) v = float(v / s);
    t.norm = 1.f;
    t.w = 1.25 * ((32.0 / 63.0) * 1.5);
    return t;
}
template <int MODE> int sub_blocks() {
    int occ = 0;
    DSG_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_amp256<MODE>, PG_THREADS, 0));
    return std::max(1, occ) * device_info().sms;
}
}}  // namespace dsg::gate

extern "C" int dsg_subgate_run(uint64_t start, uint64_t count, double maxph, double thr, uint64_t *out_seed, uint32_t cap, uint32_t *n_out,
                               uint64_t counts[3]) {
    return guarded([&] {
        DSG_ARG(n_out && (cap == 0 || out_seed), "dsg_subgate_run: null pointer");
        State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
        const uint64_t B = 1ull << 26;
        ensure_buffers(g, B);
        const Taps256 tp = sub_taps();
        const int blocks = sub_blocks<AMP_CPU>();
        uint64_t tot[3] = {0, 0, 0};
        uint32_t written = 0;
        bool overflow = false;
        std::vector<uint64_t> found;
        for (uint64_t base = 0; base < count; base += B) {
            const uint64_t nb = std::min(B, count - base);
            cudaStream_t st = g.st;
            DSG_CU(cudaMemsetAsync(g.d_n, 0, 16, st));
            const unsigned pb = unsigned(std::min<uint64_t>((nb + 255) / 256, uint64_t(device_info().sms) * 64));
            k_phase<<<pb, 256, 0, st>>>(start + base, nb, maxph, g.d_s1, g.d_n, g.cap1);
            k_octinit<<<unsigned(device_info().sms) * 13, OCT_THREADS, 0, st>>>(g.d_s1, g.d_n, g.cap1, g.d_oct);
            k_amp256<AMP_CPU><<<blocks, PG_THREADS, 0, st>>>(g.d_oct, g.d_s1, g.d_n, g.cap1, thr, tp, g.d_s2, nullptr, g.d_n + 1, g.cap2, nullptr);
            DSG_CU(cudaGetLastError());
            DSG_CU(cudaMemcpyAsync(g.h_n, g.d_n, 16, cudaMemcpyDeviceToHost, st));
            DSG_CU(cudaStreamSynchronize(st));
            const uint32_t n1 = g.h_n[0], n2 = g.h_n[1];
            overflow |= n1 > g.cap1 || n2 > g.cap2;
            const uint32_t k2 = std::min(n2, g.cap2);
            found.resize(k2);
            if (k2) {
                DSG_CU(cudaMemcpyAsync(found.data(), g.d_s2, size_t(k2) * 8, cudaMemcpyDeviceToHost, st));
                DSG_CU(cudaStreamSynchronize(st));
            }
            std::sort(found.begin(), found.end());
            for (uint64_t f : found) {
                if (written < cap) out_seed[written++] = f;
                else overflow = true;
            }
            tot[0] += nb; tot[1] += n1; tot[2] += n2;
        }
        *n_out = written;
        if (counts) std::memcpy(counts, tot, sizeof tot);
        return overflow ? DSG_OVERFLOW : DSG_OK;
    });
}

extern "C" int dsg_gate_onepar_run(uint64_t start, uint64_t count, const dsg_gate_cfg *cfg, float margin, uint64_t *out_seed, float *out_amp,
                                   uint32_t cap, uint32_t *n_out, uint64_t counts[4]) {
    return guarded([&] {
        DSG_ARG(cfg && n_out, "dsg_gate_onepar_run: null pointer");
        DSG_ARG(cap == 0 || (out_seed && out_amp), "dsg_gate_onepar_run: null output");
        State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
        const uint64_t B = cfg->batch ? cfg->batch : (1ull << 26);
        ensure_buffers(g, B);
        const double thr = double(cfg->amp - margin);         // float difference, as GateCfg.amp - GateCfg.margin
        const int blocks = sub_blocks<AMP_ONEPAR>();
        uint64_t tot[4] = {0, 0, 0, 0};
        uint32_t written = 0;
        bool overflow = false;
        std::vector<std::pair<uint64_t, float>> found;
        for (uint64_t base = 0; base < count; base += B) {
            const uint64_t nb = std::min(B, count - base);
            cudaStream_t st = g.st;
            DSG_CU(cudaMemsetAsync(g.d_n, 0, 16, st));
            const unsigned pb = unsigned(std::min<uint64_t>((nb + 255) / 256, uint64_t(device_info().sms) * 64));
            k_phase<<<pb, 256, 0, st>>>(start + base, nb, double(cfg->maxph), g.d_s1, g.d_n, g.cap1);
            k_octinit<<<unsigned(device_info().sms) * 13, OCT_THREADS, 0, st>>>(g.d_s1, g.d_n, g.cap1, g.d_oct);
            k_amp256<AMP_ONEPAR><<<blocks, PG_THREADS, 0, st>>>(g.d_oct, g.d_s1, g.d_n, g.cap1, thr, g.t256, g.d_s2, g.d_idx2, g.d_n + 1, g.cap2, nullptr);
            k_fullgate<<<g.fg_blocks, FG_THREADS, 0, st>>>(g.d_oct, g.d_s2, g.d_idx2, g.d_n + 1, g.cap2, cfg->amp, g.t512, g.d_s3, g.d_a3, g.d_n + 2,
                                                          g.cap3, nullptr, g.d_split);
            DSG_CU(cudaGetLastError());
            DSG_CU(cudaMemcpyAsync(g.h_n, g.d_n, 16, cudaMemcpyDeviceToHost, st));
            DSG_CU(cudaStreamSynchronize(st));
            const uint32_t n1 = g.h_n[0], n2 = g.h_n[1], n3 = g.h_n[2];
            overflow |= n1 > g.cap1 || n2 > g.cap2 || n3 > g.cap3;
            const uint32_t k3 = std::min(n3, g.cap3);
            if (k3) {
                DSG_CU(cudaMemcpyAsync(g.h_s3, g.d_s3, size_t(k3) * 8, cudaMemcpyDeviceToHost, st));
                DSG_CU(cudaMemcpyAsync(g.h_a3, g.d_a3, size_t(k3) * 4, cudaMemcpyDeviceToHost, st));
                DSG_CU(cudaStreamSynchronize(st));
            }
            found.clear();
            for (uint32_t i = 0; i < k3; i++) found.push_back({g.h_s3[i], g.h_a3[i]});
            std::sort(found.begin(), found.end());
            for (auto &f : found) {
                if (written < cap) { out_seed[written] = f.first; out_amp[written] = f.second; written++; }
                else overflow = true;
            }
            tot[0] += nb; tot[1] += n1; tot[2] += n2; tot[3] += n3;
        }
        *n_out = written;
        if (counts) std::memcpy(counts, tot, sizeof tot);
        return overflow ? DSG_OVERFLOW : DSG_OK;
    });
}

extern "C" int dsg_gate_onepar_amps(const uint64_t *seeds, uint32_t n, float *pre) {
    return guarded([&] {
        DSG_ARG(n == 0 || (seeds && pre), "dsg_gate_onepar_amps: null pointer");
        if (!n) return DSG_OK;
        State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
        uint64_t *d_s = nullptr; uint32_t *d_n = nullptr; Oct *d_oct = nullptr; float *d_e = nullptr; uint64_t *d_o = nullptr;
        try {
            DSG_CU(cudaMalloc(&d_s, size_t(n) * 8));
            DSG_CU(cudaMalloc(&d_n, 16));
            DSG_CU(cudaMalloc(&d_oct, size_t(n) * 2 * sizeof(Oct)));
            DSG_CU(cudaMalloc(&d_e, size_t(n) * 8));
            DSG_CU(cudaMalloc(&d_o, size_t(n) * 8));
            DSG_CU(cudaMemcpyAsync(d_s, seeds, size_t(n) * 8, cudaMemcpyHostToDevice, g.st));
            const uint32_t cnt[4] = {n, 0, 0, 0};
            DSG_CU(cudaMemcpyAsync(d_n, cnt, 16, cudaMemcpyHostToDevice, g.st));
            k_octinit<<<(2 * n + OCT_THREADS - 1) / OCT_THREADS, OCT_THREADS, 0, g.st>>>(d_s, d_n, n, d_oct);
            k_amp256<AMP_ONEPAR><<<sub_blocks<AMP_ONEPAR>(), PG_THREADS, 0, g.st>>>(d_oct, d_s, d_n, n, -1e30, g.t256, d_o, nullptr, d_n + 1, n, d_e);
            DSG_CU(cudaGetLastError());
            DSG_CU(cudaMemcpyAsync(pre, d_e, size_t(n) * 8, cudaMemcpyDeviceToHost, g.st));
            DSG_CU(cudaStreamSynchronize(g.st));
        } catch (...) { cudaFree(d_s); cudaFree(d_n); cudaFree(d_oct); cudaFree(d_e); cudaFree(d_o); throw; }
        cudaFree(d_s); cudaFree(d_n); cudaFree(d_oct); cudaFree(d_e); cudaFree(d_o);
        return DSG_OK;
    });
}

extern "C" int dsg_subgate_amps(const uint64_t *seeds, uint32_t n, float *est) {
    return guarded([&] {
        DSG_ARG(n == 0 || (seeds && est), "dsg_subgate_amps: null pointer");
        if (!n) return DSG_OK;
        State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
        uint64_t *d_s = nullptr; uint32_t *d_n = nullptr; Oct *d_oct = nullptr; float *d_e = nullptr; uint64_t *d_o = nullptr;
        try {
            DSG_CU(cudaMalloc(&d_s, size_t(n) * 8));
            DSG_CU(cudaMalloc(&d_n, 16));
            DSG_CU(cudaMalloc(&d_oct, size_t(n) * 2 * sizeof(Oct)));
            DSG_CU(cudaMalloc(&d_e, size_t(n) * 8));
            DSG_CU(cudaMalloc(&d_o, size_t(n) * 8));
            DSG_CU(cudaMemcpyAsync(d_s, seeds, size_t(n) * 8, cudaMemcpyHostToDevice, g.st));
            const uint32_t cnt[4] = {n, 0, 0, 0};
            DSG_CU(cudaMemcpyAsync(d_n, cnt, 16, cudaMemcpyHostToDevice, g.st));
            k_octinit<<<(2 * n + OCT_THREADS - 1) / OCT_THREADS, OCT_THREADS, 0, g.st>>>(d_s, d_n, n, d_oct);
            k_amp256<AMP_CPU><<<sub_blocks<AMP_CPU>(), PG_THREADS, 0, g.st>>>(d_oct, d_s, d_n, n, -1e30, sub_taps(), d_o, nullptr, d_n + 1, n, d_e);
            DSG_CU(cudaGetLastError());
            DSG_CU(cudaMemcpyAsync(est, d_e, size_t(n) * 8, cudaMemcpyDeviceToHost, g.st));
            DSG_CU(cudaStreamSynchronize(g.st));
        } catch (...) { cudaFree(d_s); cudaFree(d_n); cudaFree(d_oct); cudaFree(d_e); cudaFree(d_o); throw; }
        cudaFree(d_s); cudaFree(d_n); cudaFree(d_oct); cudaFree(d_e); cudaFree(d_o);
        return DSG_OK;
    });
}

// Device-resident form for benchmarks and the fused pipeline: enqueue one batch on `stream` and leave the
// counters {phase, pre, full} and survivors in device memory.
namespace dsg { namespace gate {
int run_device_batch(cudaStream_t st, uint64_t start, uint64_t nb, const dsg_gate_cfg &cfg, const uint32_t **d_counts,
                     const uint64_t **d_seeds, const float **d_amps) {
    State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
    ensure_buffers(g, nb);
    enqueue_batch(g, st, start, nb, cfg);
    *d_counts = g.d_n; *d_seeds = g.d_s3; *d_amps = g.d_a3;
    return DSG_OK;
}
}}

// Benchmark hook: `warmup` untimed batches, then `steps` timed batches of `per_step` seed indices each
// (fresh ranges), timed with CUDA events on the gate's own stream.  ms_kernel[0..3] = summed device time
// of the phase, octave-init, pre-gate and full-gate kernels; counts = summed {indices, phase, pre, full}.
extern "C" int dsg_gate_bench(uint64_t start, uint64_t per_step, uint32_t steps, uint32_t warmup, const dsg_gate_cfg *cfg,
                              float *ms_total, float ms_kernel[4], uint64_t counts[4]) {
    return guarded([&] {
        DSG_ARG(cfg && ms_total && ms_kernel && counts && per_step > 0, "dsg_gate_bench: bad arguments");
        State &g = S(); std::lock_guard<std::mutex> l(g.mu); setup_locked(g);
        ensure_buffers(g, per_step);
        const uint32_t total = warmup + steps;
        std::vector<cudaEvent_t> ev(size_t(steps) * 5 + 2);
        for (auto &e : ev) DSG_CU(cudaEventCreate(&e));
        uint32_t *h_cnt = nullptr;
        DSG_CU(cudaMallocHost(&h_cnt, size_t(total) * 16));
        const dsg_gate_cfg c = *cfg;
        const unsigned pb = unsigned(std::min<uint64_t>((per_step + 255) / 256, uint64_t(device_info().sms) * 64));
        for (uint32_t it = 0; it < total; it++) {
            const bool timed = it >= warmup;
            const uint32_t k = it - warmup;
            if (timed && k == 0) DSG_CU(cudaEventRecord(ev[0], g.st));
            DSG_CU(cudaMemsetAsync(g.d_n, 0, 16, g.st));
            if (timed) DSG_CU(cudaEventRecord(ev[2 + 5 * k], g.st));
            k_phase<<<pb, 256, 0, g.st>>>(start + uint64_t(it) * per_step, per_step, double(c.maxph), g.d_s1, g.d_n, g.cap1);
            if (timed) DSG_CU(cudaEventRecord(ev[3 + 5 * k], g.st));
            k_octinit<<<unsigned(device_info().sms) * 13, OCT_THREADS, 0, g.st>>>(g.d_s1, g.d_n, g.cap1, g.d_oct);
            if (timed) DSG_CU(cudaEventRecord(ev[4 + 5 * k], g.st));
            k_amp256<AMP_AA><<<g.pg_blocks, PG_THREADS, 0, g.st>>>(g.d_oct, g.d_s1, g.d_n, g.cap1, c.pthr, g.t256, g.d_s2, g.d_idx2, g.d_n + 1, g.cap2, nullptr);
            if (timed) DSG_CU(cudaEventRecord(ev[5 + 5 * k], g.st));
            k_fullgate<<<g.fg_blocks, FG_THREADS, 0, g.st>>>(g.d_oct, g.d_s2, g.d_idx2, g.d_n + 1, g.cap2, c.amp, g.t512, g.d_s3, g.d_a3, g.d_n + 2, g.cap3, nullptr, g.d_split);
            if (timed) DSG_CU(cudaEventRecord(ev[6 + 5 * k], g.st));
            DSG_CU(cudaGetLastError());
            DSG_CU(cudaMemcpyAsync(h_cnt + 4 * it, g.d_n, 16, cudaMemcpyDeviceToHost, g.st));
        }
        DSG_CU(cudaEventRecord(ev[1], g.st));
        DSG_CU(cudaStreamSynchronize(g.st));
        DSG_CU(cudaEventElapsedTime(ms_total, ev[0], ev[1]));
        for (int q = 0; q < 4; q++) ms_kernel[q] = 0;
        for (uint32_t k = 0; k < steps; k++)
            for (int q = 0; q < 4; q++) { float t; DSG_CU(cudaEventElapsedTime(&t, ev[2 + 5 * k + q], ev[3 + 5 * k + q])); ms_kernel[q] += t; }
        for (int q = 0; q < 4; q++) counts[q] = 0;
        for (uint32_t k = 0; k < steps; k++) {
            counts[0] += per_step;
            for (int q = 0; q < 3; q++) counts[1 + q] += h_cnt[4 * (warmup + k) + q];
        }
        cudaFreeHost(h_cnt);
        for (auto &e : ev) cudaEventDestroy(e);
        return DSG_OK;
    });
}

// Launch of the amplitude kernels on caller-provided buffers (used by the allocation-free entry point in
// gate_noalloc.cu).  counters[0..3] must hold {n, 0, n, 0} when the launches start.
namespace dsg { namespace gate {
void launch_amps_on(const uint64_t *d_seeds, uint32_t n, void *d_oct, uint32_t *d_counters, uint64_t *d_tmp_seeds, uint32_t *d_tmp_idx,
                    float *d_tmp_amp, float *d_pre, float *d_full, const float taps24[24], int pg_blocks, int fg_blocks, cudaStream_t st) {
    Taps256 t256; Taps512 t512;
    gate_taps(taps24, t256, t512);
    Oct *oct = static_cast<Oct *>(d_oct);
    k_octinit<<<(2 * n + OCT_THREADS - 1) / OCT_THREADS, OCT_THREADS, 0, st>>>(d_seeds, d_counters, n, oct);
    k_amp256<AMP_AA><<<pg_blocks, PG_THREADS, 0, st>>>(oct, d_seeds, d_counters, n, -1e30, t256, d_tmp_seeds, d_tmp_idx, d_counters + 1, n, d_pre);
    k_fullgate<<<fg_blocks, FG_THREADS, 0, st>>>(oct, d_seeds, nullptr, d_counters + 2, n, -1e30f, t512, d_tmp_seeds, d_tmp_amp, d_counters + 3, n, d_full, nullptr);
}
size_t oct_bytes() { return sizeof(Oct); }
int pregate_blocks_per_sm() { int occ = 0; cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_amp256<AMP_AA>, PG_THREADS, 0); return occ; }
int fullgate_blocks_per_sm() { int occ = 0; cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fullgate, FG_THREADS, 0); return occ; }
}}

// ---------------------------------------------------------------- the gate in double precision
// The same two amplitude stages with every step in double: corner tables without the rounding to float, cell
// sums, blur taps exp(-d^2 / (2 sigma^2)) and their sum, the two fused multiply-add blur passes, the division
// by the squared tap sum, the maximum.  The FP64 yardstick of the FP32 gate (the reference's gate is FP32;
// this is the same algorithm at double width), used where a seed's FP32 amplitude lies within the proven
// error margin of a threshold.  Few seeds take this path, so it favours plainness over speed: one block per
// (seed, side) and row, the grids in global scratch.
namespace dsg { namespace gate {
constexpr int G64_PRE = 256, G64_FULL = 512;
__device__ __forceinline__ double weight64() { return 1.25 * (32.0 / 63.0) * 1.5; }
// Corner tables of one (seed, side): tpre[288] (merged parity terms of the anti-aliased grid, gate.cuh:218-235)
// and tfull[512] ([px*2+pz][corner][hash], gate.cuh:236-244).
__global__ void __launch_bounds__(512) k_g64_tables(const Oct *__restrict__ oct, double *__restrict__ tpre, double *__restrict__ tfull) {
    const Oct &p = oct[blockIdx.x];
    const int e = threadIdx.x;
    if (e < 288) {
        const int h = e & 15, dy = (e >> 4) & 1, uv = e >> 5, u = uv / 3, v = uv % 3;
        double fr[2][2]; int sh[2][2];
        for (int ax = 0; ax < 2; ax++) {
            const double o = ax ? p.oz : p.ox;
            for (int q = 0; q < 2; q++) { const double b = o + 0.5 * q; fr[ax][q] = b - floor(b); sh[ax][q] = int(floor(b) - floor(o)); }
        }
        double acc = 0;
        for (int px = 0; px < 2; px++)
            for (int pz = 0; pz < 2; pz++) {
                const int dx = u - sh[0][px], dz = v - sh[1][pz];
                if (dx < 0 || dx > 1 || dz < 0 || dz > 1) continue;
                const double fx = fr[0][px], fz = fr[1][pz], tx = fade_fused(fx), tz = fade_fused(fz);
                const double wc = __dmul_rn(__dmul_rn(dx ? tx : 1 - tx, dy ? p.vy : 1 - p.vy), dz ? tz : 1 - tz);
                acc = __fma_rn(wc, gradd(h, fx - dx, p.fy - dy, fz - dz), acc);
            }
        tpre[size_t(blockIdx.x) * 288 + e] = __dmul_rn(__dmul_rn(0.25, weight64()), acc);
    }
    {
        const int h = e & 15, c = (e >> 4) & 7, pp = e >> 7, px = pp >> 1, pz = pp & 1;
        const double bx = px * 0.5 + p.ox, bz = pz * 0.5 + p.oz;
        const double fx = bx - floor(bx), fz = bz - floor(bz);
        const double tx = fade_fused(fx), tz = fade_fused(fz), ty = p.vy;
        const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
        const double wc = __dmul_rn(__dmul_rn(dx ? tx : 1 - tx, dy ? ty : 1 - ty), dz ? tz : 1 - tz);
        tfull[size_t(blockIdx.x) * 512 + e] = __dmul_rn(__dmul_rn(weight64(), wc), gradd(h, fx - dx, p.fy - dy, fz - dz));
    }
}
// Cell sums of row blockIdx.x of (seed, side) blockIdx.y: G = 256 (pre-gate) or 512 (full gate).
template <int G>
__global__ void __launch_bounds__(256) k_g64_cells(const Oct *__restrict__ oct, const double *__restrict__ tab, double *__restrict__ S) {
    const Oct &p = oct[blockIdx.y];
    const int r = blockIdx.x;
    const double *T = tab + size_t(blockIdx.y) * (G == G64_PRE ? 288 : 512);
    double *row = S + (size_t(blockIdx.y) * G + r) * G;
    for (int i = threadIdx.x; i < G; i += blockDim.x) {
        double acc = 0;
        if (G == G64_PRE) {
            const int ix0 = int(floor(p.ox)), iz0 = int(floor(p.oz));
            for (int v = 0; v < 3; v++)
                for (int dy = 0; dy < 2; dy++)
                    for (int u = 0; u < 3; u++) {
                        const int col = p.perm[(p.perm[(i + u + ix0) & 255] + p.iy + dy) & 255];
                        acc = __dadd_rn(acc, T[((u * 3 + v) * 2 + dy) * 16 + (p.perm[(col + r + v + iz0) & 255] & 15)]);
                    }
        } else {
            const int pz = r & 1, iz = (r >> 1) + int(floor(pz * 0.5 + p.oz));
            const int px = i & 1, ix = (i >> 1) + int(floor(px * 0.5 + p.ox));
            for (int c = 0; c < 8; c++) {
                const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
                const int col = p.perm[(p.perm[(ix + dx) & 255] + p.iy + dy) & 255];
                acc = __dadd_rn(acc, T[((px * 2 + pz) * 8 + c) * 16 + (p.perm[(col + iz + dz) & 255] & 15)]);
            }
        }
        row[i] = acc;
    }
}
// Blur taps in double and their sum (lowfield-style Gaussian, unnormalised as the gate's).
template <int R>
__device__ __forceinline__ double taps64(double sig, double (&k)[2 * R + 1]) {
    double ks = 0;
    for (int d = -R; d <= R; d++) { k[d + R] = exp(-0.5 * d * d / (sig * sig)); ks += k[d + R]; }
    return ks;
}
template <int G, int R>
__global__ void __launch_bounds__(256) k_g64_hblur(const double *__restrict__ S, double *__restrict__ H, double sig) {
    double k[2 * R + 1];
    taps64<R>(sig, k);
    const size_t base = (size_t(blockIdx.y) * G + blockIdx.x) * G;
    for (int i = threadIdx.x; i < G; i += blockDim.x) {
        double s = 0;
        for (int d = 0; d <= 2 * R; d++) s = __fma_rn(k[d], S[base + ((i + d - R) & (G - 1))], s);
        H[base + i] = s;
    }
}
__device__ __forceinline__ unsigned long long order64(double v) {    // unsigned order of doubles
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double unorder64(unsigned long long o) {
    return __longlong_as_double((long long)((o >> 63) ? (o & 0x7fffffffffffffffull) : ~o));
}
template <int G, int R>
__global__ void __launch_bounds__(256) k_g64_vmax(const double *__restrict__ H, double sig, unsigned long long *__restrict__ best) {
    __shared__ unsigned long long bm;
    double k[2 * R + 1];
    const double ks = taps64<R>(sig, k);
    if (threadIdx.x == 0) bm = 0;
    __syncthreads();
    const int o = blockIdx.x;
    const size_t base = size_t(blockIdx.y) * G * G;
    unsigned long long m = 0;
    for (int i = threadIdx.x; i < G; i += blockDim.x) {
        double s = 0;
        for (int d = 0; d <= 2 * R; d++) s = __fma_rn(k[d], H[base + size_t((o - R + d) & (G - 1)) * G + i], s);
        m = max(m, order64(__ddiv_rn(s, __dmul_rn(ks, ks))));
    }
    atomicMax(&bm, m);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&best[blockIdx.y], bm);
}
__global__ void k_g64_out(const unsigned long long *__restrict__ best, uint32_t n2, double *__restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n2) out[i] = unorder64(best[i]);
}

// FP64 side amplitudes pre[2i + s], full[2i + s] of n seeds (device pointers), on st, with scratch it allocates.
void amps_fp64(const uint64_t *d_seeds, uint32_t n, double *d_pre, double *d_full, cudaStream_t st) {
    constexpr uint32_t CH = 32;                              // seeds per chunk: ~300 MB of grids
    Oct *oct; uint32_t *cnt; double *tpre, *tfull, *S, *H; unsigned long long *best;
    DSG_CU(cudaMalloc(&oct, size_t(CH) * 2 * sizeof(Oct)));
    DSG_CU(cudaMalloc(&cnt, 4));
    DSG_CU(cudaMalloc(&tpre, size_t(CH) * 2 * 288 * 8)); DSG_CU(cudaMalloc(&tfull, size_t(CH) * 2 * 512 * 8));
    DSG_CU(cudaMalloc(&S, size_t(CH) * 2 * G64_FULL * G64_FULL * 8)); DSG_CU(cudaMalloc(&H, size_t(CH) * 2 * G64_FULL * G64_FULL * 8));
    DSG_CU(cudaMalloc(&best, size_t(CH) * 2 * 8));
    for (uint32_t b = 0; b < n; b += CH) {
        const uint32_t m = std::min(CH, n - b);
        DSG_CU(cudaMemcpyAsync(cnt, &m, 4, cudaMemcpyHostToDevice, st));
        k_octinit<<<(2 * m + OCT_THREADS - 1) / OCT_THREADS, OCT_THREADS, 0, st>>>(d_seeds + b, cnt, m, oct);
        k_g64_tables<<<2 * m, 512, 0, st>>>(oct, tpre, tfull);
        DSG_CU(cudaMemsetAsync(best, 0, size_t(2 * m) * 8, st));
        k_g64_cells<G64_PRE><<<dim3(G64_PRE, 2 * m), 256, 0, st>>>(oct, tpre, S);
        k_g64_hblur<G64_PRE, 4><<<dim3(G64_PRE, 2 * m), 256, 0, st>>>(S, H, 1.0);
        k_g64_vmax<G64_PRE, 4><<<dim3(G64_PRE, 2 * m), 256, 0, st>>>(H, 1.0, best);
        k_g64_out<<<(2 * m + 127) / 128, 128, 0, st>>>(best, 2 * m, d_pre + 2 * size_t(b));
        DSG_CU(cudaMemsetAsync(best, 0, size_t(2 * m) * 8, st));
        k_g64_cells<G64_FULL><<<dim3(G64_FULL, 2 * m), 256, 0, st>>>(oct, tfull, S);
        k_g64_hblur<G64_FULL, 7><<<dim3(G64_FULL, 2 * m), 256, 0, st>>>(S, H, 2.0);
        k_g64_vmax<G64_FULL, 7><<<dim3(G64_FULL, 2 * m), 256, 0, st>>>(H, 2.0, best);
        k_g64_out<<<(2 * m + 127) / 128, 128, 0, st>>>(best, 2 * m, d_full + 2 * size_t(b));
        DSG_CU(cudaGetLastError());
        DSG_CU(cudaStreamSynchronize(st));                   // the chunk's scratch is reused by the next
    }
    cudaFree(oct); cudaFree(cnt); cudaFree(tpre); cudaFree(tfull); cudaFree(S); cudaFree(H); cudaFree(best);
}
}}  // namespace dsg::gate

extern "C" int dsg_gate_amps_fp64(const uint64_t *seeds, uint32_t n, double *pre, double *full) {
    return guarded([&] {
        DSG_ARG(n == 0 || (seeds && pre && full), "dsg_gate_amps_fp64: null pointer");
        require_init();
        if (!n) return DSG_OK;
        uint64_t *d_s; double *d_p, *d_f;
        cudaStream_t st;
        DSG_CU(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        DSG_CU(cudaMalloc(&d_s, size_t(n) * 8)); DSG_CU(cudaMalloc(&d_p, size_t(n) * 16)); DSG_CU(cudaMalloc(&d_f, size_t(n) * 16));
        DSG_CU(cudaMemcpyAsync(d_s, seeds, size_t(n) * 8, cudaMemcpyHostToDevice, st));
        gate::amps_fp64(d_s, n, d_p, d_f, st);
        DSG_CU(cudaMemcpyAsync(pre, d_p, size_t(n) * 16, cudaMemcpyDeviceToHost, st));
        DSG_CU(cudaMemcpyAsync(full, d_f, size_t(n) * 16, cudaMemcpyDeviceToHost, st));
        DSG_CU(cudaStreamSynchronize(st));
        cudaFree(d_s); cudaFree(d_p); cudaFree(d_f); cudaStreamDestroy(st);
        return DSG_OK;
    });
}

// The gate decided in double precision at the price of the FP32 gate: the FP32 gate screens at thresholds
// lowered by `margin`, so every seed the FP64 gate passes survives the screen as long as the FP32 amplitudes
// are within `margin` of the FP64 ones; survivors whose FP32 amplitudes clear both thresholds by the margin
// pass as they are, and the rest are decided by the FP64 amplitudes.
extern "C" int dsg_gate_run_fp64(uint64_t start, uint64_t count, double maxph, double pthr, double amp, double margin, uint64_t *out_seed,
                                 uint32_t cap, uint32_t *n_out, uint64_t counts[6]) {
    uint64_t tot[6] = {0, 0, 0, 0, 0, 0};
    const int rc0 = guarded([&] {
        DSG_ARG(n_out && (cap == 0 || out_seed), "dsg_gate_run_fp64: null pointer");
        DSG_ARG(margin >= 0 && margin < 0.1, "dsg_gate_run_fp64: margin must be in [0, 0.1)");
        return DSG_OK;
    });
    if (rc0 != DSG_OK) return rc0;
    *n_out = 0;
    const dsg_gate_cfg screen{float(maxph), float(pthr - margin), float(amp - margin), 0};
    const uint64_t B = 1ull << 26;
    std::vector<uint64_t> s(1u << 20); std::vector<float> a(1u << 20);
    bool over = false;
    for (uint64_t base = 0; base < count; base += B) {
        const uint64_t nb = std::min(B, count - base);
        uint32_t n = 0; uint64_t c[4];
        const int rc = dsg_gate_run(start + base, nb, &screen, s.data(), a.data(), uint32_t(s.size()), &n, c);
        if (rc < 0) return rc;
        if (rc == DSG_OVERFLOW) over = true;
        tot[0] += c[0]; tot[1] += c[1]; tot[2] += n;
        if (!n) continue;
        std::vector<float> pre(2 * size_t(n)), full(2 * size_t(n));
        int rc2 = dsg_gate_amps(s.data(), n, pre.data(), full.data());
        if (rc2 < 0) return rc2;
        std::vector<uint64_t> unsure;
        std::vector<char> keep(n, 0);
        for (uint32_t i = 0; i < n; i++) {
            const double p32 = double(0.f + pre[2 * i] + pre[2 * i + 1]), f32 = double(0.f + full[2 * i] + full[2 * i + 1]);
            if (p32 >= pthr + margin && f32 >= amp + margin) keep[i] = 1;
            else unsure.push_back(s[i]);
        }
        tot[3] += n - unsure.size(); tot[4] += unsure.size();
        std::vector<double> p64(2 * unsure.size()), f64(2 * unsure.size());
        if (!unsure.empty()) {
            rc2 = dsg_gate_amps_fp64(unsure.data(), uint32_t(unsure.size()), p64.data(), f64.data());
            if (rc2 < 0) return rc2;
        }
        for (uint32_t i = 0, u = 0; i < n; i++) {
            if (!keep[i]) { keep[i] = p64[2 * u] + p64[2 * u + 1] >= pthr && f64[2 * u] + f64[2 * u + 1] >= amp; u++; }
            if (!keep[i]) continue;
            tot[5]++;
            if (*n_out < cap) out_seed[(*n_out)++] = s[i];
            else over = true;
        }
    }
    if (counts) std::memcpy(counts, tot, sizeof tot);
    if (over) { dsg::set_error("dsg_gate_run_fp64: more survivors than capacity"); return DSG_OVERFLOW; }
    return DSG_OK;
}
