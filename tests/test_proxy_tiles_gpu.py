"""Proxy bitmaps over tiles of 32 x 32 cells (and strips, which are not tiled): sizes at and beside the tile's edges, zones of
one call with different seeds and shapes, coordinates of both signs and out to the world border, against the oracle
cell for cell."""
import json
import os

import numpy as np
import pytest

import libs

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
M64 = (1 << 64) - 1
FINDS = json.load(open(os.path.join(G, "finds.json")))


def centred(f, nx, nz):
    return ((f["x"] >> 2) // 32 * 32 - 32 * (nx // 2), (f["z"] >> 2) // 32 * 32 - 32 * (nz // 2), nx, nz)


@pytest.mark.parametrize("nx,nz", [(1, 1), (1, 300), (300, 1), (7, 40), (40, 7), (8, 8), (9, 33), (31, 31), (32, 32), (33, 32), (32, 33), (63, 65), (64, 64), (200, 95)])
def test_sizes(dsg, nx, nz):
    seen = 0
    for f in FINDS[:3]:
        z = centred(f, nx, nz)
        got = dsg.proxy(f["seed"], [z])[0]
        want = libs.orc_proxy_zone(f["seed"] & M64, *z, 0.35)
        assert np.array_equal(got, want)
        seen += int(want.sum())
    assert seen > 0


@pytest.mark.parametrize("x0,z0", [(-7_500_000, -7_500_000), (7_490_000, -7_490_000), (-40, 7_480_000), (0, 0), (13, -27)])
def test_places(dsg, x0, z0):
    """Origins off the step-32 grid, at the corners of the world and across its centre."""
    for f in FINDS[3:6]:
        z = (x0, z0, 70, 41)
        assert np.array_equal(dsg.proxy(f["seed"], [z])[0], libs.orc_proxy_zone(f["seed"] & M64, *z, 0.35))


def test_zones_of_several_seeds_in_one_call(dsg):
    seeds, owner, zones = [], [], []
    for k, f in enumerate(FINDS[:6]):
        seeds.append(f["seed"])
        for nx, nz in [(5, 90), (64, 37), (100, 100), (8, 33)]:
            owner.append(k); zones.append(centred(f, nx, nz))
    _, maps = dsg.proxy_components(seeds, owner, zones, min_cells=1)
    for k, z, m in zip(owner, zones, maps):
        assert np.array_equal(m, libs.orc_proxy_zone(seeds[k] & M64, *z, 0.35))
