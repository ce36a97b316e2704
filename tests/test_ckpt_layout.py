"""The layout of checkpoint buffers (voxviz_b200/csrc/ckpt_layout.h) for every
number of record slots a caller may ask for, on the host, and the library's
sizes by it."""
import subprocess
from pathlib import Path

import voxviz_b200 as vv

ROOT = Path(__file__).resolve().parents[1]


def test_layout(tmp_path):
    exe = tmp_path / "ckpt_layout_check"
    subprocess.run(["g++", "-O2", "-std=c++17", str(ROOT / "tests" / "ckpt_layout_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[0]) == 135


def test_sizes():
    for w, h, per_ray in ((1, 1, 1), (63, 47, 16), (2, 1, 1 << 30), (1, 1, (1 << 31) - 1)):
        assert vv.Context.ckpt_bytes(w, h, per_ray) == (8 * w * h + 15) // 16 * 16 + 48 * w * h * per_ray
