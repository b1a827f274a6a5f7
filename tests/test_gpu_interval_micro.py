"""The interval passes over micro-ops (interval_micro.cuh) where a bound is not
finite: divisions by intervals that hold 0, products and exponentials that
overflow, an infinite and a NaN constant, an infinite tape time. Such cells run
the exact path, and masks, topology and shortened tapes equal the oracle's in
both roundings, with one and two cells per lane and with item pruning."""
from __future__ import annotations

import importlib.util
from pathlib import Path

import numpy as np
import pytest

import frep
from frep import csg, scenes
from frep.csg import Exp, Max, Min, Sqrt, T, X, Y, Z

CSRC = Path(__file__).resolve().parents[1] / "f-rep-voxel-rendering_b200" / "csrc"


def _const_tape(value):
    """min(max(x, c) - 0.3, y * y - 0.5) with the constant c = value."""
    c = int(np.float32(value).view(np.uint32))
    w = [(0 | 4 << 16 | c << 32), (8 | 4 << 16 | 0 << 32 | 4 << 48),
         (0 | 5 << 16 | int(np.float32(0.3).view(np.uint32)) << 32), (4 | 4 << 16 | 4 << 32 | 5 << 48),
         (5 | 6 << 16 | 1 << 32 | 1 << 48), (0 | 5 << 16 | int(np.float32(0.5).view(np.uint32)) << 32),
         (4 | 6 << 16 | 6 << 32 | 5 << 48), (7 | 0 << 16 | 4 << 32 | 6 << 48)]
    return frep.Tape.from_wide(np.array(w, np.uint64))


def _ball():
    return X() * X() + Y() * Y() + Z() * Z() - 0.8


SHAPES = {
    "div": (lambda: Min(1.0 / X() - 2.0, Max(_ball(), Y() / Z() - 0.5)), 0.0),
    "overflow": (lambda: Max(_ball(), Min(X() * 3e38 * (Y() * 3e38) * Z(), Z() - 0.2)), 0.0),
    "exp": (lambda: Max(_ball(), Min(Exp(X() * 200.0) - Exp(Y() * 200.0), Z())), 0.0),
    "sqrt": (lambda: Max(Sqrt(_ball()) - 0.4, Min(X() * X() * 3e38 * 10.0 - Y(), Z())), 0.0),
    "time": (lambda: Min(_ball(), Max(X() * T() - Y(), Z() - 0.1)), float("inf")),
    "inf": (lambda: _const_tape(np.inf), 0.0),
    "-inf": (lambda: _const_tape(-np.inf), 0.0),
    "nan": (lambda: _const_tape(np.nan), 0.0),
    "finite": (lambda: Max(_ball(), Min(X() * Y() - 0.1, Z())), 0.5),
}


@pytest.mark.gpu
@pytest.mark.parametrize("rounding", [0, 1])
@pytest.mark.parametrize("name", list(SHAPES))
def test_cells_with_infinite_bounds_equal_the_oracle(name, rounding):
    from parity import compare_trees, oracle_tree
    ctx = frep.Context(0, hbm_budget_bytes=8 << 30)
    make, time = SHAPES[name]
    shape = make()
    tape = shape if isinstance(shape, frep.Tape) else frep.Tape(shape)
    storages, oracles = [], []
    for dims in ([16, 4], [4, 8, 4]):
        sc = scenes.Scene(name, tape, dims, (-1.5, -1.5, -1.5), 3.0, None, 64, 64)
        # (pools large enough for item pruning at the second level)
        vs = frep.VoxelStorage(dims, sc.low_vertex, sc.world_size, rounding=rounding, node_words=1 << 26,
                               tape_words=1 << 26).init(ctx, tape)
        frep.Voxelizer(ctx, vs).voxelize(time)
        oracles.append(oracle_tree(sc, tape, rounding=rounding, tape_time=time))
        assert compare_trees(vs.export(), oracles[-1]) == [], dims
        storages.append(vs)
    batch = frep.Batch(ctx, storages)  # two cells per lane at the root
    batch.voxelize([time] * 2)
    for vs, orc in zip(storages, oracles):
        assert compare_trees(vs.export(), orc) == []
    batch.close()


def test_interval_micro_table():
    spec = importlib.util.spec_from_file_location("gen_interval_micro", CSRC / "gen_interval_micro.py")
    g = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(g)
    assert (CSRC / "interval_micro.cuh").read_text() == g.text()
    for rnd in (0, 1):
        for cells in (1, 2):
            lines = g.gen(rnd, cells)
            tab = next(l for l in lines if ".branchtargets" in l)
            targets = tab.split(".branchtargets", 1)[1].strip(" ;").split(", ")
            assert len(targets) == 512
            for t in set(targets):
                assert sum(1 for l in lines if l == t + ":") == 1, t
            labels = {l[:-1] for l in lines if l.endswith(":") and l.count("_") == 3}
            assert labels == set(targets) - {"$FIM_EXIT"}
