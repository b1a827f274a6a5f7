"""The ray walk's division by a cell size with its reciprocal at hand
(csrc/cell_div.h) rounds like the division, at ends of the mantissa too."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_division_by_reciprocal_is_the_division(tmp_path):
    exe = tmp_path / "cell_div_host"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'f-rep-voxel-rendering_b200/csrc'}",
                    f"-I{ROOT / 'include'}", str(ROOT / "tests/cpp/cell_div_host.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), "3000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
