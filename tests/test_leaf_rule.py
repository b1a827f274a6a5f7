"""The rule between the two last-level passes (csrc/leaf_rule.h) takes the one
that measured faster, over launches of every kind, and the host leaves the pass
over micro-ops out of launches that are too small for it."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

# transcendental, root words, node words, nodes, grid, us word by word, us as micro-ops
MEASURED = [
    (1, 46, 30, 24274, "16 8 4", 77, 142), (1, 47, 47, 15584, "16 4 4", 56, 101),
    (0, 19, 19, 43056, "16 4 4", 58, 101), (1, 26, 25, 36536, "16 8 4", 69, 105),
    (0, 499, 40, 13760, "16 8 4", 46, 67), (0, 223, 21, 24527, "16 8 4", 50, 67),
    (0, 499, 39, 55059, "16 16 4", 101, 128), (0, 1904, 44, 31325, "32 8 4", 75, 93),
    (0, 3094, 60, 215754, "16 16 4", 431, 351), (0, 7807, 135, 446362, "16 16 4", 1846, 1320),
    (0, 12390, 128, 765104, "16 16 4", 3051, 1947), (0, 12390, 195, 44047, "16 4 4", 306, 359),
    (0, 19, 19, 714544, "16 16 4", 509, 402), (0, 19, 19, 178824, "16 8 4", 151, 175),
    (1, 49, 42, 245621, "16 16 4", 790, 1035),
    (1, 49, 40, 3830873, "16 4 4 4 4", 11065, 12118), (1, 239, 43, 2191931, "24 8 4", 7322, 6611),
    (0, 7710, 101, 1722936, "32 16 4", 5387, 2697), (0, 8054, 158, 71624, "12 8 8", 2282, 1504),
    (0, 570, 40, 23873, "16 16 8", 241, 208), (0, 570, 42, 3345, "12 8 8", 52, 58), (0, 374, 37, 24989, "16 16 4", 58, 83),
    (0, 12390, 849, 1881, "16 4", 292, 244), (0, 217, 43, 60, "16 4", 28, 30),
    (0, 12390, 849, 1881, "16 8", 374, 661), (0, 499, 79, 320, "16 8", 50, 120),
    (0, 499, 45, 941, "32 8", 30, 58), (0, 19, 19, 8936, "32 8", 56, 77),
    (0, 223, 21, 97951, "16 16 8", 523, 304), (0, 12390, 128, 765104, "16 16 8", 14678, 9738),
    (1, 46, 30, 24274, "16 8 8", 736, 404), (0, 19, 19, 714544, "16 16 8", 2394, 2450),
    (1, 26, 25, 146120, "16 16 8", 906, 955), (0, 3094, 237, 939, "16 16", 298, 284),
    (0, 27962, 1681, 1538, "16 16", 2862, 4200), (0, 7807, 1566, 288, "8 32", 3931, 3212),
    (0, 27962, 4757, 312, "8 32", 12849, 17388),
]


def _rule(tmp_path, cases):
    exe = tmp_path / "leaf_rule_host"
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{ROOT / 'f-rep-voxel-rendering_b200/csrc'}",
                    str(ROOT / "tests/cpp/leaf_rule_host.cpp"), "-o", str(exe)], check=True)
    lines = [f"{t} {r} {w} {n} {len(g.split())} {g}" for t, r, w, n, g, *_ in cases]
    out = subprocess.run([str(exe)], input="\n".join(lines), capture_output=True, text=True, check=True).stdout
    return [(int(a), float(b)) for a, b in (line.split() for line in out.splitlines())]


def test_the_faster_pass_is_picked(tmp_path):
    for case, (micro, _) in zip(MEASURED, _rule(tmp_path, MEASURED)):
        plain, ops = case[5:]
        assert micro == (ops < plain), case


def test_small_grids_are_left_to_the_point_pass(tmp_path):
    grids = {"16 4": 0, "16 4 4": 0, "16 8 4": 0, "16 8": 0, "32 8": 0, "16 16 4": 1, "16 16 8": 1, "16 8 8": 1, "8 32": 1,
             "16 4 4 4 4": 1}
    cases = [(0, 100, 50, 1000, g) for g in grids]
    for g, (_, load) in zip(grids, _rule(tmp_path, cases)):
        assert (load >= 1.0) == bool(grids[g]), g
