"""The climate octaves from a patch's lattice points (csrc/noise.cuh, patch_build and perlin_patch) are the octave's own
doubles wherever the patch lies.  The device functions themselves, compiled by the host compiler (cpp/patch_check.cpp): patches whose
corner lies just below a lattice line near 0, where a fraction taken from the corner would lose its last bits, and patches all
over the world.  Away from line 0 nearly every octave has to stay in the table."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_patch_octaves_are_the_octaves(tmp_path):
    exe = str(tmp_path / "patch_check")
    subprocess.check_call(["g++", "-O2", "-march=x86-64-v3", "-ffp-contract=off", "-std=c++20", "-I/usr/local/cuda/include", "-I" + os.path.join(ROOT, "include"),
                           "-I" + os.path.join(ROOT, "tests", "cpp"), "-I" + os.path.join(ROOT, "desert-search_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "patch_check.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
    _, samples, kept, plain = out.stdout.split()
    assert int(samples) > 1_000_000
    assert int(kept) >= 0.99 * int(plain)
