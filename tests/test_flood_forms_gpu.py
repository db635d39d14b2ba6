"""The two forms of the flood evaluation give one result: a round of few sub-blocks (a single flood: four lanes per cell,
eight lanes per pending point) and a round of many (a large batch: one lane per cell, the patch's lattice points shared).
Every DenseArea field against the oracle, on sites whose rounds exercise both, at the steps where a sub-block spans
less than one lattice cell, a few and many, and at window sizes that cut sub-blocks and tiles."""
import json
import os

import numpy as np
import pytest

import libs

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
M64 = (1 << 64) - 1


def sites(dsg, n):
    """Desert starts: verified finds, then random worlds."""
    finds = json.load(open(os.path.join(G, "finds.json")))[:n // 2]
    out = [(f["seed"] & M64, f["x"] >> 2, f["z"] >> 2) for f in finds]
    rng = np.random.default_rng(11)
    while len(out) < n:
        seeds = rng.integers(-(1 << 63), (1 << 63) - 1, 64, dtype=np.int64).view(np.uint64)
        xz = (rng.integers(-30_000_000, 30_000_001, (64 * 64, 2)) >> 2).astype(np.int32)
        st = dsg.query(seeds, np.repeat(np.arange(64, dtype=np.uint32), 64), 6, xz).reshape(64, 64)
        for i in range(64):
            k = np.nonzero(st[i] == 2)[0]
            if len(k) and len(out) < n:
                out.append((int(seeds[i]), int(xz[i * 64 + k[0], 0]), int(xz[i * 64 + k[0], 1])))
    return out


@pytest.mark.parametrize("step,half,conn8", [(1, 150, False), (1, 7, True), (1, 33, False), (3, 100, True), (8, 120, False), (64, 90, True)])
def test_single_and_batched_floods_equal_the_oracle(dsg, step, half, conn8):
    ss = sites(dsg, 12)
    want = [libs.orc().flood(s, x, z, step, half, conn8, 0) for s, x, z in ss]
    assert [dsg.flood(s, x, z, step, half, conn8) for s, x, z in ss] == want
    many = 60                                              # 720 floods: rounds beyond what the split form takes
    got = dsg.flood_batch([dsg.flood_req(s, x, z, step, half, conn8) for _ in range(many) for s, x, z in ss])
    assert got == want * many


def test_world_border(dsg):
    """Cells beyond |x|, |z| = 7,499,996 quarts are outside: the same in both forms, wherever a start there is passable."""
    rng = np.random.default_rng(3)
    reqs, want = [], []
    for s, _, _ in sites(dsg, 12):
        xz = np.stack([rng.integers(-7499990, 7499990, 512), np.where(rng.random(512) < 0.5, -1, 1) * 7499980], 1).astype(np.int32)
        st = dsg.query(np.array([s], dtype=np.uint64), np.zeros(512, dtype=np.uint32), 6, xz)
        for k in np.nonzero(st == 2)[0][:3]:
            a = libs.orc().flood(s, int(xz[k, 0]), int(xz[k, 1]), 1, 60, False, 0)
            assert dsg.flood(s, int(xz[k, 0]), int(xz[k, 1]), 1, 60, False) == a
            reqs.append(dsg.flood_req(s, int(xz[k, 0]), int(xz[k, 1]), 1, 60, False)); want.append(a)
    assert len(reqs) > 0 and any(a[7] for a in want)
    n = -(-600 // len(reqs))
    assert dsg.flood_batch(reqs * n) == want * n


def test_predicates_mixed_in_one_round(dsg):
    """Hot, proxy and desert floods together, few (split rounds hold all three) and many."""
    ss = sites(dsg, 6)
    reqs = [dsg.flood_req(s, x, z, 16, 60, True, pred, 0.35) for s, x, z in ss for pred in (0, 1, 2)]
    want = [libs.orc().flood(s, x, z, 16, 60, True, pred, 0.35) for s, x, z in ss for pred in (0, 2, 4)]      # the oracle's codes
    for k in (1, 3, len(reqs)):
        assert dsg.flood_batch(reqs[:k]) == want[:k]
    assert dsg.flood_batch(reqs * 30) == want * 30


@pytest.mark.parametrize("step,half,conn8", [(256, 40, True), (128, 63, True), (64, 15, False), (1, 50, False), (256, 3, True)])
def test_hot_floods_alone(dsg, step, half, conn8):
    """Batches of hot-zone floods alone have a kernel of their own: one flood, a few, many, several seeds a block."""
    ss = sites(dsg, 12)
    want = [libs.orc().flood(s, x, z, step, half, conn8, 2) for s, x, z in ss]
    reqs = [dsg.flood_req(s, x, z, step, half, conn8, 1) for s, x, z in ss]
    assert [dsg.flood_batch([r])[0] for r in reqs] == want
    assert dsg.flood_batch(reqs) == want
    assert dsg.flood_batch(reqs * 200) == want * 200
    assert any(a[0] > 1 for a in want)


def test_hot_floods_at_the_border(dsg):
    rng = np.random.default_rng(5)
    reqs, want = [], []
    for s, _, _ in sites(dsg, 8):
        for x, z in [(7499900, int(rng.integers(-7e6, 7e6))), (int(rng.integers(-7e6, 7e6)), -7499900)]:
            reqs.append(dsg.flood_req(s, x, z, 64, 30, True, 1)); want.append(libs.orc().flood(s, x, z, 64, 30, True, 2))
    assert dsg.flood_batch(reqs) == want and any(a[7] for a in want)
