"""The LOD certificates (voxviz_b200/csrc/lod_bound.h) clear no level for a
camera beyond the distances that their bounds are shown for, also where its
squared distance overflows binary32."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_far_cameras_clear_nothing(tmp_path):
    exe = tmp_path / "lod_far_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", str(ROOT / "tests" / "lod_far_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[0]) > 5000
