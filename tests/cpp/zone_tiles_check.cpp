// Which zones go by tiles (zones.cuh, tiled): every lattice column under a tile has its place in the tile's table.  The
// positions as k_proxy takes them (32-bit quart coordinates, which wrap), the widths as its tables are sized: the span of 31
// steps in whole lattice cells, one more, and the far corner.  And no zone is kept from its tiles but a strip or one that wraps.
// Prints "ok <zones by tiles> <others>", or the first zone that breaks a rule.
#include "device_on_host.h"
#include "zones.cuh"
#include <random>

using dsg::zones::DZone;

// Largest place of a column of the axis' tiles in a table row, over the octave at 2^-log2f; -1: a column before the first.
static int64_t reach(int32_t first, int32_t n, int log2f, bool side, double off) {
    int64_t most = 0;
    for (int32_t i0 = 0; i0 < n; i0 += 32) {
        const auto pos = [&](int c) {
            const int32_t x = int32_t(uint32_t(first) + 32u * uint32_t(i0 + c));
            return std::floor(double(x) * (side ? 337. / 331. : 1.) * std::ldexp(1.0, -log2f) + off);
        };
        for (int c = 0; c < min(32, n - i0); c++) {
            const double d = pos(c) - pos(0);
            if (d < 0) return -1;
            most = max(most, int64_t(d));
        }
    }
    return most;
}

int main() {
    std::mt19937_64 rng(7);
    const auto between = [&](int64_t lo, int64_t hi) { return int64_t(lo + int64_t(rng() % uint64_t(hi - lo + 1))); };
    long tiles = 0, others = 0;
    for (int rep = 0; rep < 60000; rep++) {
        DZone z{};
        const int64_t ends[4] = {0, 7'500'000, INT32_MAX, INT32_MIN};
        const int64_t x = ends[rep % 4] + between(-40000, 40000), zz = ends[rep / 4 % 4] + between(-40000, 40000);
        z.x0 = int32_t(std::clamp<int64_t>(x, INT32_MIN, INT32_MAX)); z.z0 = int32_t(std::clamp<int64_t>(zz, INT32_MIN, INT32_MAX));
        z.nx = int32_t(between(1, rep % 3 ? 70 : 1500)); z.nz = int32_t(between(1, rep % 5 ? 70 : 1500));
        const bool by_tiles = dsg::zones::tiled(z);
        (by_tiles ? tiles : others)++;
        const int64_t lx = int64_t(z.x0) + 32 * int64_t(z.nx - 1), lz = int64_t(z.z0) + 32 * int64_t(z.nz - 1);
        if (!by_tiles && z.nx >= 8 && z.nz >= 8 && lx <= INT32_MAX && lz <= INT32_MAX) {
            printf("not by tiles: %d %d %d %d\n", z.x0, z.z0, z.nx, z.nz);
            return 1;
        }
        if (!by_tiles) continue;
        for (int log2f = 7; log2f <= 10; log2f++)
            for (int side = 0; side < 2; side++) {
                const int width = int(31 * 32 * 337.0 / 331.0 / double(1 << log2f)) + 3;
                const double off = double(rng() >> 11) * 0x1p-53 * 256;
                for (int axis = 0; axis < 2; axis++) {
                    const int64_t at = reach(axis ? z.z0 : z.x0, axis ? z.nz : z.nx, log2f, side, off);
                    if (at < 0 || at + 1 >= width) {
                        printf("zone %d %d %d %d: place %lld of %d lattice columns (frequency 2^-%d)\n", z.x0, z.z0, z.nx, z.nz, (long long)at, width, log2f);
                        return 1;
                    }
                }
            }
    }
    printf("ok %ld %ld\n", tiles, others);
}
