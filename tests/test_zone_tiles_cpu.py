"""A proxy zone goes by tiles only where every lattice column under a tile has its place in the tile's table (csrc/zones.cuh, tiled): not
where its coordinates wrap, which the library accepts.  The rule itself, compiled by the host compiler (cpp/zone_tiles_check.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_zones_by_tiles_stay_in_their_tables(tmp_path):
    exe = str(tmp_path / "zone_tiles_check")
    subprocess.check_call(["g++", "-O2", "-march=x86-64-v3", "-ffp-contract=off", "-std=c++20", "-I/usr/local/cuda/include", "-I" + os.path.join(ROOT, "include"),
                           "-I" + os.path.join(ROOT, "tests", "cpp"), "-I" + os.path.join(ROOT, "desert-search_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "zone_tiles_check.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
    _, tiles, others = out.stdout.split()
    assert int(tiles) > 10000 and int(others) > 10000
