"""Item pruning looks for SIN / COS / EXP in a node's tape only where the tree's
root tape has one, which the header says per voxelization: a batch whose trees
change between algebraic and transcendental tapes, and a
shape whose shortened tapes have lost the sine in some nodes and kept it in
others, equal the oracle each time."""
from __future__ import annotations

import pytest

import frep
from frep import scenes
from frep.csg import Max, Min, Sin, X, Y, Z
from parity import compare_trees_fast, oracle_tree

pytestmark = pytest.mark.gpu

LOW, WORLD, DIMS = (-1.5, -1.5, -1.5), 3.0, [16, 8, 4]


def test_trees_that_change_between_algebraic_and_transcendental_tapes():
    ctx = frep.Context(0, hbm_budget_bytes=16 << 30)
    csg = scenes.random_csg(60, seed=9, grid_dims=DIMS)
    waves = Sin(X() * 9.0) + Sin(Y() * 9.0) + Sin(Z() * 9.0) - 0.2
    half = Min(csg.shape, Max(waves, X() - 0.1))  # the sine decides x < 0.1 alone
    tapes = [frep.Tape(s) for s in (csg.shape, waves, half)]
    storages = [frep.VoxelStorage(DIMS, LOW, WORLD, node_words=1 << 25, tape_words=1 << 25).init(ctx, t) for t in tapes]
    oracles = [oracle_tree(scenes.Scene("flag", t, DIMS, LOW, WORLD, None, 64, 64), t) for t in tapes]
    batch = frep.Batch(ctx, storages)
    for turn in range(4):
        for i, vs in enumerate(storages):
            vs.tape = tapes[(i + turn) % 3]
        batch.set_tapes()
        batch.voxelize()
        for i, vs in enumerate(storages):
            assert compare_trees_fast(vs.export(), oracles[(i + turn) % 3]) == [], (turn, i)
    batch.close()
    for turn in range(3):  # alone
        vs = storages[0]
        vs.tape = tapes[turn]
        frep.Voxelizer(ctx, vs).voxelize(0.0)
        assert compare_trees_fast(vs.export(), oracles[turn]) == [], turn
