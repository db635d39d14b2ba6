"""Exact floods in large rounds where the noise of a temperature octave has its own origin: lattice lines -1, 0 and 1 along x or z
pass through the window, so a sub-block's patch straddles them and doubles are finest there.  Against the oracle, enough
copies in one batch that its rounds are large, and each flood alone."""
import numpy as np
import pytest

import libs

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1


class Rng:
    """The worlds' generator (xoroshiro128++)."""

    def __init__(self, s0, s1):
        self.s = [s0, s1]

    def next(self):
        s0, s1 = self.s
        rot = lambda v, k: ((v << k) | (v >> (64 - k))) & M64
        out, t = (rot((s0 + s1) & M64, 17) + s0) & M64, s1 ^ s0
        self.s = [rot(s0, 49) ^ t ^ ((t << 21) & M64), rot(t, 28)]
        return out

    def uniform(self):
        return (self.next() >> 11) * 2.0 ** -53


def offsets(seed):
    """(x, z) offsets of the slowest temperature octave (frequency 2^-10), sides A and B."""
    s = seed ^ 0x6a09e667f3bcc909
    w = Rng(libs.mix(s), libs.mix(s + 0x9e3779b97f4a7c15))
    a, b = w.next(), w.next()
    c = Rng(a ^ 0x5c7e6b29735f0d7f, b ^ 0xf7d86f1bbc734988)
    out = []
    for _ in range(2):
        fa, fb = c.next(), c.next()
        r = Rng(fa ^ 0x36d326eed40efeb2, fb ^ 0x5be9ce18223c636a)
        x, _, z = (r.uniform() * 256 for _ in range(3))
        out.append((x, z))
    return out


def starts(dsg, n):
    rng = np.random.default_rng(41)
    out = []
    while len(out) < n:
        seeds = [int(v) for v in rng.integers(-(1 << 63), (1 << 63) - 1, 64, dtype=np.int64).view(np.uint64)]
        xz = rng.integers(-7_000_000, 7_000_000, (64, 16, 2)).astype(np.int32)
        for i, s in enumerate(seeds):
            axis, side, line = i & 1, (i >> 1) & 1, (-1, 0, 1)[i % 3]
            scale = 337 / 331 if side else 1.0
            xz[i, :, axis] = np.floor((line - offsets(s)[side][axis]) * 1024 / scale).astype(np.int32) + rng.integers(-9, 10, 16)
        st = dsg.query(np.array(seeds, dtype=np.uint64), np.repeat(np.arange(64, dtype=np.uint32), 16), 6, xz.reshape(-1, 2)).reshape(64, 16)
        for i in range(64):
            k = np.nonzero(st[i] == 2)[0]
            if len(k):
                out.append((seeds[i], int(xz[i, k[0], 0]), int(xz[i, k[0], 1])))
    return out[:n]


@pytest.mark.parametrize("step,half", [(1, 48), (3, 30)])
def test_floods_across_lattice_lines(dsg, step, half):
    ss = starts(dsg, 24)
    want = [libs.orc().flood(s, x, z, step, half, False, 0) for s, x, z in ss]
    assert sum(a[0] > 50 for a in want) >= 12
    assert [dsg.flood(s, x, z, step, half, False) for s, x, z in ss] == want
    got = dsg.flood_batch([dsg.flood_req(s, x, z, step, half, False) for _ in range(30) for s, x, z in ss])
    assert got == want * 30
