"""The arithmetic of the unit-box walk (voxviz_b200/csrc: fixed_div.h,
walknode.h, lod_bound.h, dxt.h) against what it stands for, on the host: quotients by
a ray's direction equal IEEE division, node records equal the words they are
made from, the quick LOD test never clears a level that stops, and a DXT5
texel decoded alone equals its block's.  The
kernels' bit-exact parity rests on these."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_walk_arithmetic(tmp_path):
    exe = tmp_path / "walk_arith_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", str(ROOT / "tests" / "walk_arith_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    counts = [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    assert len(counts) == 4 and all(bad == 0 for _, bad in counts)
    assert counts[0][0] == 20000000 and counts[1][0] > 2000000 and counts[2][0] > 100000, counts
