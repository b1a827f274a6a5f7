"""The scratch of a single tree's passes holds room for item tapes where the
budget allows, and keeps it. That room gives way: a budget that holds the pools,
the passes' own scratch and the next allocation still holds them after a
voxelization that took the room (a further tree, the side arrays of reuse, a
batch's scratch, point evaluation), and the trees stay those of the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import frep
from frep import scenes
from parity import compare_trees_fast, oracle_tree

pytestmark = pytest.mark.gpu

MB = 1 << 20
LARGE = dict(node_words=1 << 26, tape_words=1 << 25)  # item room: 32 KB for each warp of the passes
SMALL = dict(node_words=1 << 22, tape_words=1 << 21)  # no item room
POINTS = 1 << 20


@pytest.fixture(scope="module")
def scene():
    sc = scenes.random_csg(30, seed=17, grid_dims=[16, 8, 4])
    tape = frep.Tape(sc.shape)
    return sc, tape, oracle_tree(sc, tape)


def _tree(ctx, sc, tape, pools):
    return frep.VoxelStorage(sc.grid_dims, sc.low_vertex, sc.world_size, **pools).init(ctx, tape)


def _used(ctx):
    return ctx.memory()[0]


def _points():
    return np.random.default_rng(5).uniform(-1.2, 1.2, (POINTS, 4)).astype(np.float32)


def _grown(ctx, call):
    before = _used(ctx)
    call()
    return _used(ctx) - before


@pytest.mark.parametrize("what", ["tree", "reuse", "batch", "points"])
def test_item_room_gives_way(scene, what):
    sc, tape, want = scene
    big = frep.Context(0, hbm_budget_bytes=16 << 30)
    other = _tree(big, sc, tape, SMALL)
    scratch = _grown(big, lambda: frep.Voxelizer(big, other).voxelize(0.0))
    first = []
    pools = _grown(big, lambda: first.append(_tree(big, sc, tape, LARGE)))
    roomy = _grown(big, lambda: frep.Voxelizer(big, first[0]).voxelize(0.0))
    assert roomy > scratch + 60 * MB
    arrays = 8 * (LARGE["node_words"] // 8 + 1)
    if what == "tree":  # a second tree, and its scratch in place of the room
        budget = 2 * pools + 2 * scratch
    elif what == "reuse":  # a second tree reuses the first
        budget = 2 * pools + roomy + scratch + arrays
    elif what == "batch":
        batches = []
        need = _grown(big, lambda: (batches.append(frep.Batch(big, first)), batches[0].voxelize()))
        batches[0].close()
        budget = pools + scratch + need
    else:
        budget = pools + scratch + POINTS * 20
    for vs in (other, first[0]):
        vs.cleanup()
    big.close()

    ctx = frep.Context(0, hbm_budget_bytes=max(budget, pools + roomy) + MB)
    a = _tree(ctx, sc, tape, LARGE)
    frep.Voxelizer(ctx, a).voxelize(0.0)
    assert compare_trees_fast(a.export(), want) == []
    trees = [a]
    if what in ("tree", "reuse"):
        b = _tree(ctx, sc, tape, LARGE)
        frep.Voxelizer(ctx, b).voxelize(0.0, reuse=a if what == "reuse" else None)
        assert compare_trees_fast(b.export(), want) == []
        trees.append(b)
    elif what == "batch":
        batch = frep.Batch(ctx, trees)
        batch.voxelize()
        assert compare_trees_fast(a.export(), want) == []
        batch.close()
    else:
        pts = _points()
        np.testing.assert_array_equal(ctx.eval_points(tape, pts), tape.eval_points(pts))
    for vs in trees:  # again, with whatever scratch is left
        frep.Voxelizer(ctx, vs).voxelize(0.0)
        assert compare_trees_fast(vs.export(), want) == []
    used, limit = ctx.memory()
    assert used <= limit
    for vs in trees:
        vs.cleanup()
    assert _used(ctx) == 0
    ctx.close()


def test_scratch_of_a_captured_voxelization_stays(scene):
    """A graph holds the scratch's address: no other allocation takes its room."""
    import torch
    sc, tape, want = scene
    big = frep.Context(0, hbm_budget_bytes=16 << 30)
    first = []
    pools = _grown(big, lambda: first.append(_tree(big, sc, tape, LARGE)))
    roomy = _grown(big, lambda: frep.Voxelizer(big, first[0]).voxelize(0.0))
    first[0].cleanup()
    big.close()
    ctx = frep.Context(0, hbm_budget_bytes=2 * pools + roomy - 8 * MB)
    a = _tree(ctx, sc, tape, LARGE)
    v = frep.Voxelizer(ctx, a)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        v.voxelize(0.0, stream=stream)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            v.voxelize(0.0, stream=stream)
        before = _used(ctx)
        with pytest.raises(frep.FrepError):
            _tree(ctx, sc, tape, LARGE)
        assert _used(ctx) == before
        graph.replay()
        stream.synchronize()
    assert compare_trees_fast(a.export(), want) == []
    del graph
    a.cleanup()
    ctx.close()
