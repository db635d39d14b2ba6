"""The gate's cell lists when they fill (csrc/gate_amp.cuh, list_cells): a full list is cleared of cells that the running maximum has left
behind, and where that is not enough the warp evaluates the defining chain at every cell.  Ordinary seeds list a cell or two, so
the library is built with a wider listing window here: the same amplitudes, bit for bit, from every form of the gate.
That the lists do fill is shown on the screen's own values, restated on the CPU."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

import libs
import tune_gate
from test_flood_lines_gpu import Rng
from test_gate_screen_cpu import screen

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
START, COUNT = 10**12, 30000

CHILD = """
import sys, numpy as np, dsgpu
dsgpu.init(0, 0.35)
seeds = np.load(sys.argv[1])
pre, full = dsgpu.gate_amps(seeds)
got, amps, counts, rc = dsgpu.gate_run(int(sys.argv[3]), int(sys.argv[4]))
assert rc == 0
np.savez(sys.argv[2], pre=pre, full=full, onepar=dsgpu.gate_onepar_amps(seeds), sub=dsgpu.subgate_amps(seeds), got=got, amps=amps, counts=counts)
"""


def octaves(seed):
    """The gate's octave of both sides: permutation and offsets."""
    s = seed ^ 0x6a09e667f3bcc909
    w = Rng(libs.mix(s), libs.mix(s + 0x9e3779b97f4a7c15))
    a, b = w.next(), w.next()
    c = Rng(a ^ 0x5c7e6b29735f0d7f, b ^ 0xf7d86f1bbc734988)
    out = []
    for _ in range(2):
        fa, fb = c.next(), c.next()
        r = Rng(fa ^ 0x36d326eed40efeb2, fb ^ 0x5be9ce18223c636a)
        off = [r.uniform() * 256 for _ in range(3)]
        p = list(range(256))
        for k in range(256):
            n = 256 - k
            m = (r.next() & 0xffffffff) * n
            while (m & 0xffffffff) < (1 << 32) % n:
                m = (r.next() & 0xffffffff) * n
            j = k + (m >> 32)
            p[k], p[j] = p[j], p[k]
        out.append((np.array(p), *off))
    return out


def walk(columns, window):
    """A warp's list over its columns of screen values, without a floor: was it cleared, was it full all the same."""
    best, lim, vals, cleared = -1e9, -1e9, [], False
    for col in columns:
        best = max(best, col.max())
        lim = max(lim, best - window)
        for v in col.reshape(-1, 32):
            m = v[v >= lim]
            if len(vals) + len(m) > 32:
                cleared, vals = True, [x for x in vals if x >= lim]
            if len(vals) + len(m) > 32:
                return cleared, True
            vals += list(m)
    return cleared, False


def fill(seeds, window, form):
    """The lists of the seeds whose gate lists without a floor (a side within the window of the floor), by `walk`."""
    out = []
    for s in seeds:
        grids = [screen(*o, form) for o in octaves(int(s))]
        if min(g.max() for g in grids) > 0.24 + window - 1e-4:
            continue
        for g in grids:
            if form == "aa":
                warps = [g[128 * w: 128 * w + 128].T for w in (0, 1)]
                at = 4
            else:
                warps, at = [g[pz::2][128 * zh: 128 * zh + 128].T for pz in (0, 1) for zh in (0, 1)], 7
            out += [walk(np.roll(w, -at, 0), window) for w in warps]
    return out


@pytest.fixture(scope="module")
def seeds():
    s = np.array([libs.mix(START + k) for k in range(1 << 13)], dtype=np.uint64)
    ph, _ = libs.orc().phase(s)
    return s[ph <= 0.06][:40]


@pytest.mark.parametrize("window", [0.03, 0.1])
def test_full_lists_give_the_same_amplitudes(dsg, seeds, tmp_path, window):
    if not shutil.which("nvcc") or not os.path.exists(os.path.join(tune_gate.BUILD, "search.o")):
        pytest.skip("needs nvcc and make's objects")
    for form in ("aa", "full"):
        lists = fill(seeds, window, form)
        assert any(full if window > 0.05 else cleared and not full for cleared, full in lists)
    obj, lib = str(tmp_path / "gate.o"), str(tmp_path / "libdsgpu.so")
    subprocess.check_call(["nvcc"] + tune_gate.FLAGS + tune_gate.ARCH + [f"-DDSG_AMP_WINDOW={window}f", "-c", os.path.join(ROOT, "desert-search_b200", "csrc", "gate.cu"), "-o", obj])
    objs = [os.path.join(tune_gate.BUILD, f) for f in sorted(os.listdir(tune_gate.BUILD)) if f.endswith(".o") and f not in ("gate.o", "orc_blob.o")]
    subprocess.check_call(["nvcc"] + tune_gate.ARCH + ["-shared", "-o", lib, obj] + objs + ["-lcudart_static", "-lpthread", "-ldl", "-lrt"])
    np.save(tmp_path / "seeds.npy", seeds)
    subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "seeds.npy"), str(tmp_path / "out.npz"), str(START), str(COUNT)], check=True, timeout=300,
                   env=dict(os.environ, DSGPU_LIB=lib, PYTHONPATH=os.path.join(ROOT, "desert-search_b200")))
    got = np.load(tmp_path / "out.npz")
    pre, full = libs.orc_gate(seeds, True, *dsg.gate_taps())
    assert np.array_equal(got["pre"], pre) and np.array_equal(got["full"], full)
    assert np.array_equal(got["sub"], libs.orc_subgate(seeds))
    assert np.array_equal(got["onepar"], dsg.gate_onepar_amps(seeds))
    # a short range: the full gate's columns are split over blocks
    s, a, counts = libs.orc_gate_range(START, COUNT)
    assert len(s) > 0 and np.array_equal(got["got"], s) and np.array_equal(got["amps"], a)
    assert [int(c) for c in got["counts"]] == [int(c) for c in counts]
