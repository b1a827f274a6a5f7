"""The last-level pass's micro-ops (csrc/micro_ops.h) on the host: every tape
form that the library takes (compiled scenes, the reference's demo shapes,
imported wide tapes with reused, repeated, unread and uninitialised-free
slots), shortened at random, gives the bits of plain interpretation; marks are stripped from copied pools word for word. And the loop's
generated header is its generator's output, with a case for every dispatch
index that the decoder makes."""
from __future__ import annotations

import importlib.util
import subprocess
from pathlib import Path

import numpy as np

import frep
from frep import scenes

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "f-rep-voxel-rendering_b200" / "csrc"


def random_tape(rng, n, slots):
    """Instructions over a small slot file: inputs, constants and results are
    read any number of times, in either operand or both; unread ones occur."""
    words, known = [], [0, 1, 2, 3]
    for i in range(n):
        op = int(rng.choice([0, 0, 0, 3, 4, 5, 3, 4, 5, 7, 8, 7, 8, 10, 11, 12, 6, 1]))
        out = 0 if i == n - 1 else int(rng.integers(0, slots))
        if op == 0:
            bits = int(np.float32(rng.uniform(-2, 2)).view(np.uint32))
            w = op | out << 16 | bits << 32
        else:
            pick = lambda: int(words[-1] >> 16 & 0xFFFF) if words and rng.random() < 0.5 else int(rng.choice(known))
            w = op | out << 16 | pick() << 32 | pick() << 48
        words.append(w)
        if out not in known:
            known.append(out)
    return np.array(words, np.uint64)


def test_decoded_tapes_match_plain_interpretation(tmp_path):
    rng = np.random.default_rng(3)
    tapes = [frep.Tape(scenes.random_csg(n, seed=n).shape).wide() for n in (4, 9, 33, 80)]
    tapes += [frep.Tape(f(2)).wide() for f in scenes.DEMO_SHAPES.values()]
    tapes += [frep.Tape(scenes.spheres_union(70).shape, const_reload=r).wide() for r in (0, 0xFFFFFFFF)]
    tapes.append(frep.Tape(scenes.stress_gyroid(8).shape).wide())
    tapes += [random_tape(rng, int(rng.integers(1, 300)), int(rng.integers(5, 32))) for _ in range(200)]
    data = tmp_path / "tapes.bin"
    with open(data, "wb") as f:
        for t in tapes:
            f.write(np.uint64(len(t)).tobytes() + np.ascontiguousarray(t, np.uint64).tobytes())
    exe = tmp_path / "micro_host"
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", f"-I{CSRC}", str(ROOT / "tests/cpp/micro_host.cpp"),
                    str(CSRC / "micro_ops.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(data)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
    n, words, ops = (int(v) for v in r.stdout.replace(",", "").split()[0:5:2])
    assert n == len(tapes) and 0 < ops < words


def _gen():
    spec = importlib.util.spec_from_file_location("gen_leaf_dispatch", CSRC / "gen_leaf_dispatch.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_leaf_loop_table():
    g = _gen()
    assert (CSRC / "leaf_dispatch.cuh").read_text() == g.text()
    for k in g.WIDTHS:
        lines = g.gen(k)
        tab = next(l for l in lines if ".branchtargets" in l)
        targets = tab.split(".branchtargets", 1)[1].strip(" ;").split(", ")
        assert len(targets) == 512
        for t in set(targets):
            assert sum(1 for l in lines if l == t + ":") == 1, t
        for idx, t in enumerate(targets):
            ka, kb, op = idx & 3, idx >> 2 & 3, idx >> 4 & 15
            name = {v: n for n, v in g.OPS.items()}.get(op)
            src = "SFI?"[ka] + "SFI?"[kb]
            inline = (name in g.BINARY and src in g.SOURCES and not (name in g.COMMUTATIVE and src in ("SF", "IS", "IF"))
                      or name in g.UNARY and (src == "FS" or src == "SS" and name != "SQRT") or name == "CONST" and src == "SS")
            assert (t != "$FRL_EXIT") == inline, (idx, t)
