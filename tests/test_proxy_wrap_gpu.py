"""Proxy zones that reach past 2^31 quarts: their coordinates wrap, as 32-bit numbers do, and each cell is the cell of that place.
Against zones of one cell (never by tiles) at the wrapped coordinates, and against the oracle."""
import json
import os

import numpy as np
import pytest

import libs

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1
FINDS = json.load(open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "finds.json")))
TOP = (1 << 31) - 1


def wrapped(v):
    return (v + (1 << 31)) % (1 << 32) - (1 << 31)


@pytest.mark.parametrize("x0,z0,nx,nz", [(TOP, -4000, 40, 33), (-4000, TOP - 31, 33, 40), (TOP - 32 * 20, TOP - 32 * 9, 64, 70), (TOP - 32 * 31, 0, 32, 32),
                                         (TOP - 32 * 31 + 1, 0, 32, 32), (-(1 << 31), -(1 << 31), 70, 41)])
def test_zones_that_wrap(dsg, x0, z0, nx, nz):
    for f in FINDS[:2]:
        got = dsg.proxy(f["seed"], [(x0, z0, nx, nz)])[0]
        cols = dsg.proxy(f["seed"], [(wrapped(x0 + 32 * i), wrapped(z0 + 32 * j), 1, 1) for j in range(nz) for i in range(nx)])
        assert np.array_equal(got, np.array([int(m[0, 0]) for m in cols], dtype=np.uint8).reshape(nz, nx))
        rows = [libs.orc_proxy_zone(f["seed"] & M64, wrapped(x0 + 32 * i), wrapped(z0 + 32 * j), 1, 1, 0.35)[0, 0] for j in (0, nz - 1) for i in range(nx)]
        assert np.array_equal(got[[0, nz - 1]].ravel(), np.array(rows))
        comps, maps = dsg.proxy_components([f["seed"]], [0], [(x0, z0, nx, nz)])
        assert np.array_equal(maps[0], got) and sum(c["cells"] for c in comps) == int(got.sum())
