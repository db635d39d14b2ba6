"""Large rounds of exact floods take the shift octaves from tables of a sub-block's columns and rows.  Floods across the
origin, where a column or row at coordinate 0 meets the octave at y = 0 or z = 0, and across negative coordinates, against
the oracle: enough copies in one batch that its rounds are large."""
import numpy as np
import pytest

import libs

pytestmark = pytest.mark.gpu


def starts(dsg, n):
    rng = np.random.default_rng(23)
    out = []
    while len(out) < n:
        seeds = rng.integers(-(1 << 63), (1 << 63) - 1, 256, dtype=np.int64).view(np.uint64)
        xz = rng.integers(-9, 10, (256, 2)).astype(np.int32)
        st = dsg.query(seeds, np.arange(256, dtype=np.uint32), 6, xz)
        out += [(int(seeds[i]), int(xz[i, 0]), int(xz[i, 1])) for i in np.nonzero(st == 2)[0]]
    return out[:n]


@pytest.mark.parametrize("step,half", [(1, 40), (1, 17), (3, 30), (17, 25), (100, 20)])
def test_floods_across_the_origin(dsg, step, half):
    ss = starts(dsg, 10)
    want = [libs.orc().flood(s, x, z, step, half, True, 0) for s, x, z in ss]
    assert any(a[0] > 50 for a in want) or step > 3
    got = dsg.flood_batch([dsg.flood_req(s, x, z, step, half, True) for _ in range(60) for s, x, z in ss])
    assert got == want * 60
