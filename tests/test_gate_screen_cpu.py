"""The two evaluations of the gate's amplitude kernels (csrc/gate_amp.cuh) restated in numpy, in float32 and in the
kernels' operation order: the screen (z direction applied once to the permutation's sequence, then the x direction)
and the defining chain (corner terms by hash, blur along x, blur along z).  At every cell they differ by at most
E = 1.5e-5, the bound derived from the operation counts in the header, on random octaves and at the edges of the
offsets (lattice points, half points, just below either)."""
import numpy as np
import pytest

E = 1.5e-5
GRAD = np.array([[1, 1, 0], [-1, 1, 0], [1, -1, 0], [-1, -1, 0], [1, 0, 1], [-1, 0, 1], [1, 0, -1], [-1, 0, -1],
                 [0, 1, 1], [0, -1, 1], [0, 1, -1], [0, -1, -1], [1, 1, 0], [0, -1, 1], [-1, 1, 0], [0, -1, -1]], dtype=np.float64)
F = np.float32
WEIGHT = 1.25 * (32 / 63) * 1.5


def fade(t):
    return t * t * t * (t * (t * 6 - 15) + 10)


def fma(a, b, c):
    return (np.float64(a) * np.float64(b) + np.float64(c)).astype(F)


def taps(r, sigma):
    k = np.exp(-0.5 * (np.arange(-r, r + 1) / sigma) ** 2).astype(F)
    s = F(0)
    for v in k:
        s = F(s + v)
    return k, F(1) / (s * s)


def octave(seed, edge):
    rng = np.random.default_rng(seed)
    ox, oy, oz = rng.random(3) * 256
    near = [0.0, 0.5, np.nextafter(0.5, 0), np.nextafter(1.0, 0), 255.0, 254.5]
    if edge is not None:
        ox, oz = np.floor(ox) + near[edge[0] % 6] % 1, np.floor(oz) + near[edge[1] % 6] % 1
    return rng.permutation(256), ox, oy, oz


def column_hashes(perm, x, y):
    return perm[(perm[x & 255] + y) & 255]


def axis_terms(o, half, merged):
    """(lattice offset, weight, weight * distance) of the corners of the axis' sample at parity `half`."""
    out = []
    for q in ((0, 1) if merged else (half,)):
        b = o + 0.5 * q
        f, t, sc = b - np.floor(b), fade(b - np.floor(b)), 0.5 if merged else 1.0
        for d in (0, 1):
            w = sc * (t if d else 1 - t)
            out.append((int(np.floor(b) - np.floor(o)) + d, w, w * (f - d)))
    return out


def gather(terms, n):
    b, c = np.zeros(n), np.zeros(n)
    for at, w, wd in terms:
        b[at] += w; c[at] += wd
    return b, c


def chain(perm, ox, oy, oz, form):
    """The defining chain's grid (side x side float32)."""
    fy, vy, iy = oy - np.floor(oy), fade(oy - np.floor(oy)), int(np.floor(oy))
    full = form == "full"
    n, r = (512, 7) if full else (256, 4)
    k, norm = taps(r, 2.0 if full else 1.0)
    i = np.arange(n)
    S = np.zeros((n, n), F)                                # [z][x]
    wy = (1 - vy, vy)
    if form == "aa":
        tx, tz = axis_terms(ox, 0, True), axis_terms(oz, 0, True)
        for v in range(3):
            for dy in range(2):
                for u in range(3):
                    T = np.zeros(16)
                    for au, wx, wdx in tx:
                        for av, wz, wdz in tz:
                            if au == u and av == v:
                                T += wy[dy] * (GRAD[:, 0] * wdx * wz + GRAD[:, 1] * (fy - dy) * wx * wz + GRAD[:, 2] * wx * wdz)
                    col = column_hashes(perm, i + u + int(np.floor(ox)), iy + dy)
                    h = perm[(col[None, :] + (i + v + int(np.floor(oz)))[:, None]) & 255] & 15
                    S = (S + (WEIGHT * T).astype(F)[h]).astype(F)
    else:
        par = i & 1 if full else 0 * i
        cell = i >> 1 if full else i
        bx, bz = ox + 0.5 * par, oz + 0.5 * par
        fx, fz = bx - np.floor(bx), bz - np.floor(bz)
        for c in range(8):
            dx, dy, dz = c & 1, (c >> 1) & 1, c >> 2
            col = column_hashes(perm, cell + np.floor(bx).astype(int) + dx, iy + dy)
            h = perm[(col[None, :] + (cell + np.floor(bz).astype(int) + dz)[:, None]) & 255] & 15
            wx, wz = (fade(fx) if dx else 1 - fade(fx))[None, :], (fade(fz) if dz else 1 - fade(fz))[:, None]
            T = WEIGHT * wx * wy[dy] * wz * (GRAD[:, 0][h] * (fx - dx)[None, :] + GRAD[:, 1][h] * (fy - dy) + GRAD[:, 2][h] * (fz - dz)[:, None])
            S = (S + T.astype(F)).astype(F)
    for ax in (1, 0):
        acc = np.zeros_like(S)
        for d in range(-r, r + 1):
            x = np.roll(S, -d, ax)
            acc = (acc + (k[d + r] * x).astype(F)).astype(F) if form == "cpu" else fma(k[d + r], x, acc)
        S = acc
    return (S * norm).astype(F)


def screen(perm, ox, oy, oz, form):
    fy, vy, iy = oy - np.floor(oy), fade(oy - np.floor(oy)), int(np.floor(oy))
    full = form == "full"
    r = 7 if full else 4
    k, norm = taps(r, 2.0 if full else 1.0)
    s = GRAD[perm & 15].astype(F)                          # (256, 3)
    ix0, iz0 = int(np.floor(ox)), int(np.floor(oz))
    e = np.arange(256)
    out = np.zeros((512, 512) if full else (256, 256), F)
    for q in range(2 if full else 1):                      # row parity
        # z taps on lattice rows -r' .. of a row of this parity
        lo, nt = -4, 10 if full else 11
        b, c = np.zeros(nt), np.zeros(nt)
        for d in range(-r, r + 1):
            pos = q + d
            h, cell = (pos & 1, pos >> 1) if full else (0, pos)
            for at, w, wd in axis_terms(oz, h, form == "aa"):
                g = np.float64(k[d + r]) * np.float64(norm)
                b[cell + at - lo] += g * w; c[cell + at - lo] += g * wd
        b, c = b.astype(F), c.astype(F)
        fx, f_y, fz = (np.zeros(256, F) for _ in range(3))
        for t in range(nt):
            g = s[(e + lo + iz0 + t) & 255]
            fx, f_y, fz = fma(b[t], g[:, 0], fx), fma(b[t], g[:, 1], f_y), fma(c[t], g[:, 2], fz)
        w = [F(WEIGHT * (1 - vy)), F(WEIGHT * vy)]
        U = [(w[dy] * fx).astype(F) for dy in (0, 1)]
        V = [(w[dy] * fma(F(fy) - F(dy), f_y, fz)).astype(F) for dy in (0, 1)]
        col = [column_hashes(perm, ix0 + e, iy + dy) for dy in (0, 1)]
        u = (U[0][(col[0][None, :] + e[:, None]) & 255] + U[1][(col[1][None, :] + e[:, None]) & 255]).astype(F)
        v = (V[0][(col[0][None, :] + e[:, None]) & 255] + V[1][(col[1][None, :] + e[:, None]) & 255]).astype(F)
        if full:
            S = np.zeros((256, 512), F)
            for p in (0, 1):
                acc = np.zeros((256, 256), F)
                for at, wx, wdx in axis_terms(ox, p, False):
                    acc = fma(F(wdx), np.roll(u, -at, 1), fma(F(wx), np.roll(v, -at, 1), acc))
                S[:, p::2] = acc
        else:
            n = 3 if form == "aa" else 2
            bx, ax = gather(axis_terms(ox, 0, form == "aa"), 3)
            S = np.zeros((256, 256), F)
            for t in range(n):
                S = fma(F(ax[t]), np.roll(u, -t, 1), fma(F(bx[t]), np.roll(v, -t, 1), S))
        o = (k[r] * S).astype(F)
        if full:                                           # pending sums, taps in order
            o = np.zeros_like(S)
            for d in range(-r, r + 1):
                o = fma(k[d + r], np.roll(S, -d, 1), o)
        else:                                              # symmetric pairs, nearest first
            for d in range(1, r + 1):
                o = fma(k[r - d], (np.roll(S, -d, 1) + np.roll(S, d, 1)).astype(F), o)
        if full:
            out[q::2] = o
        else:
            out = o
    return out


@pytest.mark.parametrize("form", ["aa", "cpu", "onepar", "full"])
@pytest.mark.parametrize("seed,edge", [(0, None), (1, None), (2, (0, 1)), (3, (1, 0)), (4, (2, 3)), (5, (3, 2)), (6, (4, 5))])
def test_screen_is_within_its_bound_of_the_defining_chain(form, seed, edge):
    o = octave(seed, edge)
    a, b = chain(*o, form), screen(*o, form)
    assert np.abs(a).max() > 0.1
    assert np.abs(a.astype(np.float64) - b).max() <= E
