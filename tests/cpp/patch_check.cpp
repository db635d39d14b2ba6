// The patch form of the climate octaves (noise.cuh: patch_build, perlin_patch, channel_patch) against perlin and channel
// themselves, double for double, on random octave tables.  Patches lie where the fraction is most easily lost: with their
// corner just below a lattice line near 0, where v = x freq + o changes sign and doubles are finest, with offsets from
// far below one lattice cell up to 256, along x, along z and along both; and at random places of the world.
// Prints "ok <samples> <octave patches kept away from line 0>, of <all of them>", or the first difference.
#include "device_on_host.h"
#include "noise.cuh"
#include <random>

using namespace dsg;

static SeedNoise S;
static PatchCache C;
static std::mt19937_64 rng(20240607);
static double unit() { return double(rng() >> 11) * 0x1p-53; }

// Random permutations and offsets; frequencies, amplitudes and gradients as k_seed_noise stores them (offsets on its grid of 2^-45).
static void make_noise(double most) {
    static const int cnt[6] = {2, 2, 9, 4, 3, 3}, off[6] = {0, 4, 8, 26, 34, 40}, first[6] = {-10, -8, -9, -9, -3, -7};
    for (int ch = 0; ch < 6; ch++) {
        S.off[ch] = off[ch]; S.cnt[ch] = cnt[ch]; S.factor[ch] = 1.25;
        for (int k = 0; k < 2 * cnt[ch]; k++) {
            const int i = off[ch] + k, j = k % cnt[ch];
            NOct &o = S.oct[i];
            const auto offset = [&] { return std::floor(unit() * most * 0x1p45) * 0x1p-45; };
            o.ox = offset(); o.oy = unit() * 256; o.oz = offset();
            o.freq = std::ldexp(1.0, first[ch] + (ch == CH_T ? 2 * j : j));
            o.amp = std::ldexp(1.0, -j) * (0.5 + unit());
            o.iy = int(o.oy); o.fy = o.oy - o.iy; o.vy = fade_d(o.fy); o.pad = 0;
            uint8_t p[256];
            for (int e = 0; e < 256; e++) p[e] = uint8_t(e);
            std::shuffle(p, p + 256, rng);
            for (int e = 0; e < 512; e++) S.perm[i][e] = p[e & 255];
        }
    }
    for (int h = 0; h < 16; h++) {
        const int ui = h < 8 ? 0 : 1, vi = h < 4 ? 1 : ((h == 12 || h == 14) ? 0 : 2);
        uint64_t packed = 0;
        for (int c = 0; c < 3; c++) {
            const double g = (ui == c ? ((h & 1) ? -1. : 1.) : 0.) + (vi == c ? ((h & 2) ? -1. : 1.) : 0.);
            packed |= uint64_t(uint32_t(__double2hiint(g)) >> 16) << (8 + 16 * c);
        }
        S.grad[h] = make_uint2(uint32_t(packed), uint32_t(packed >> 32));
    }
}
static bool same(double a, double b) { return std::bit_cast<uint64_t>(a) == std::bit_cast<uint64_t>(b) || (a == 0 && b == 0); }

int main() {
    long samples = 0, kept = 0, plain = 0;
    // the patch at (x0, z0): every octave at points of it, and the five channels
    const auto check = [&](double x0, double z0, double ext, bool world) {
        for (int t = 0; t < 256; t++) patch_build(S, C, x0, z0, ext, t, 256);
        for (int n = 0; n < 24; n++) {
            const double px = x0 + unit() * ext, pz = z0 + unit() * ext;
            for (int k = 0; k < kPatchOct; k++) {
                const int i = patch_octave(k);
                const NOct &o = S.oct[i];
                const double s = (kSideB >> i & 1) ? 337. / 331. : 1., x = px * s * o.freq, z = pz * s * o.freq;
                const double got = perlin_patch(o, S.perm[i], S.grad, C, k, x, z), want = perlin(o, S.perm[i], S.grad, x, 0, z);
                samples++;
                if (!same(got, want)) {
                    printf("octave %d (freq %g, offsets %.17g %.17g) at %.17g %.17g, patch corner %.17g %.17g: %.17g, perlin %.17g\n", i, o.freq,
                           o.ox, o.oz, px, pz, x0, z0, got, want);
                    exit(1);
                }
            }
            for (int ch : {CH_T, CH_H, CH_C, CH_E, CH_W})
                if (!same(channel_patch(S, C, ch, px, pz), channel(S, ch, px, 0, pz))) { printf("channel %d differs\n", ch); exit(1); }
        }
        if (world)
            for (int k = 0; k < kPatchOct; k++) {
                const NOct &o = S.oct[patch_octave(k)];
                if (ext * (337. / 331.) * o.freq >= 1.25) continue;
                plain++; kept += std::isfinite(C.bx[k]);
            }
    };
    for (int rep = 0; rep < 400; rep++) {
        make_noise(rep % 4 == 0 ? 256. : rep % 4 == 1 ? 1. : rep % 4 == 2 ? 0x1p-8 : 0x1p-30);
        for (int m = 0; m < 12; m++) {
            const int i = patch_octave(int(rng() % kPatchOct)), line = int(rng() % 6) - 3, step = 1 + int(rng() % 3);
            const NOct &o = S.oct[i];
            const double s = (kSideB >> i & 1) ? 337. / 331. : 1., ext = 15 * step + 4, far = std::floor((unit() - 0.5) * 15e6);
            // whole quarts, as the sub-blocks', the line somewhere inside the patch
            const double lx = std::floor((line - o.ox) / (s * o.freq) - unit() * ext), lz = std::floor((line - o.oz) / (s * o.freq) - unit() * ext);
            check(m % 3 == 1 ? far : lx, m % 3 == 0 ? far : lz, ext, false);
        }
        check(std::floor((unit() - 0.5) * 15e6), std::floor((unit() - 0.5) * 15e6), 19, rep % 4 == 0);
    }
    printf("ok %ld %ld %ld\n", samples, kept, plain);
}
