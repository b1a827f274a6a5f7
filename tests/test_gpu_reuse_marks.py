"""Reuse compares instructions, not the readers that the root tape had: two
tapes whose nodes' tapes are the same words below the root, though in one of
them the far branch reads a value of the near one, share those nodes."""
from __future__ import annotations

import numpy as np
import pytest

import frep
from frep import scenes
from parity import compare_trees, oracle_tree

pytestmark = pytest.mark.gpu

CONST, ADD, SUB, MUL, MIN = 0, 3, 4, 5, 7


def _op(op, out, a, b):
    return op | out << 16 | a << 32 | b << 48


def _const(out, value):
    return CONST | out << 16 | int(np.float32(value).view(np.uint32)) << 32


def _tape(shared):
    """min(x^2 + y^2 - 0.5, far): far = x^2 + x + 10 (reads x^2) or x + x + 20;
    both above the cylinder in every cell of the root."""
    w = [_op(MUL, 4, 0, 0), _op(MUL, 5, 1, 1), _op(ADD, 5, 4, 5), _const(6, 0.5), _op(SUB, 5, 5, 6),
         _op(ADD, 4, 4, 0) if shared else _op(ADD, 4, 0, 0), _const(6, -10.0 if shared else -20.0), _op(SUB, 4, 4, 6),
         _op(MIN, 0, 5, 4)]
    return frep.Tape.from_wide(np.array(w, np.uint64))


@pytest.mark.parametrize("first", [True, False])
def test_nodes_with_the_same_words_are_copied(first):
    ctx = frep.Context(0, hbm_budget_bytes=8 << 30)
    sc = scenes.Scene("cylinder", None, [16, 8, 4], (-1.5, -1.5, -1.5), 3.0, None, 64, 64)
    trees, tapes = [], [_tape(first), _tape(not first)]
    for tape in tapes:
        vs = frep.VoxelStorage(sc.grid_dims, sc.low_vertex, sc.world_size).init(ctx, tape)
        frep.Voxelizer(ctx, vs).voxelize(0.0, reuse=trees[0] if trees else None)
        assert compare_trees(vs.export(), oracle_tree(sc, tape)) == []
        trees.append(vs)
    work = [vs.work() for vs in trees]
    assert work[0][1] > 0 and work[0][2] > 0
    assert work[1][0] > 0 and work[1][1:] == [0, 0]
    for vs in trees:
        vs.cleanup()
    ctx.close()
