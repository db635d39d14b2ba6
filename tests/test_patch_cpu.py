"""The patch form of a Perlin octave (noise.cuh, perlin_patch), restated in numpy: the fraction from the patch's lattice
corner is x - floor(x) exactly, and the corner term gx x + (gz z + gy dy) is the reference's u + v, double for double
(a product with 0 or +-1 is exact, so plain numpy rounds where the fused form does)."""
import numpy as np

GRAD = np.array([[1, 1, 0], [-1, 1, 0], [1, -1, 0], [-1, -1, 0], [1, 0, 1], [-1, 0, 1], [1, 0, -1], [-1, 0, -1],
                 [0, 1, 1], [0, -1, 1], [0, 1, -1], [0, -1, -1], [1, 1, 0], [0, -1, 1], [-1, 1, 0], [0, -1, -1]], dtype=np.float64)


def uv(h, x, y, z):
    u = x if h < 8 else y
    v = y if h < 4 else (x if h in (12, 14) else z)
    return (-u if h & 1 else u) + (-v if h & 2 else v)


def test_corner_terms():
    rng = np.random.default_rng(0)
    x, y, z = (np.r_[rng.random(4000), 0.0, 1 - 2.0 ** -53, 2.0 ** -40] for _ in range(3))
    for h in range(16):
        gx, gy, gz = GRAD[h]
        for dx in (0, 1):
            for dy in (0, 1):
                for dz in (0, 1):
                    a = gx * (x - dx) + (gz * (z - dz) + gy * (y - dy))
                    assert np.array_equal(a, uv(h, x - dx, y - dy, z - dz))


def test_fractions_from_the_corner():
    rng = np.random.default_rng(1)
    for freq in 2.0 ** -np.arange(1, 11):
        for s in (1.0, 337 / 331):
            o = rng.random(2000) * 256
            x0 = rng.integers(-7_500_000, 7_500_000, 2000).astype(np.float64)
            x = x0 + rng.random(2000) * 18
            b = np.floor(x0 * s * freq + o)
            v = x * s * freq + o
            f = v - b
            ins = (f >= 0) & (f < 2)
            cell = f >= 1
            assert np.array_equal((f - cell)[ins], (v - np.floor(v))[ins])
            assert np.array_equal((b + cell)[ins], np.floor(v)[ins])
            if 19 * s * freq < 1.25:
                assert ins.mean() > 0.7


def test_patch_covers_its_cells():
    """An octave kept in the table (extent below 1.25 lattice cells) has every lattice column of an inside point in 3 x 3."""
    f = np.array([0.0, 0.5, 1.0, 1.5, np.nextafter(2.0, 0)])
    cell = (f >= 1).astype(int)
    assert ((cell >= 0) & (cell + 1 <= 2)).all()
