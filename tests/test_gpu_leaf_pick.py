"""The last-level pass that the level scan picks (leaf_rule.h) is the one that
runs, in launches of one tree and of a batch, with and without reuse, on both
sides of its lines and for every last dim; each tree equals the oracle's."""
from __future__ import annotations

import pytest
import torch

import frep
from frep import scenes
from parity import compare_trees_fast, oracle_tree

pytestmark = pytest.mark.gpu

UNIT, DEMO = ((-1.5,) * 3, 3.0), ((-20.0,) * 3, 40.0)


@pytest.fixture(scope="module")
def ctx():
    return frep.Context(0, hbm_budget_bytes=48 << 30)


def _scene(shape, dims, box=UNIT):
    return scenes.Scene("leaf", frep.Tape(shape), list(dims), box[0], box[1], None, 64, 64)


def _storage(ctx, sc):
    return frep.VoxelStorage(sc.grid_dims, sc.low_vertex, sc.world_size, node_words=1 << 27, tape_words=1 << 25).init(
        ctx, sc.shape)


def _passes(call):
    """us spent in the passes over micro-ops and over words."""
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    us = {"leaf_level_kernel": 0.0, "point_level_kernel": 0.0}
    for e in p.events():
        for k in us:
            if e.device_type == torch.autograd.DeviceType.CUDA and k in e.name:
                us[k] += e.time_range.end - e.time_range.start
    if not any(us.values()):
        pytest.skip("no kernel times: the profiler is not available")
    return us["leaf_level_kernel"], us["point_level_kernel"]


CSG = scenes.random_csg(100, seed=16).shape
CASES = [  # shape, grid, box, micro-ops
    (CSG, [16, 16, 4], UNIT, True), (CSG, [12, 8, 8], UNIT, True), (CSG, [16, 16], UNIT, True), (CSG, [8, 32], UNIT, True),
    (scenes.random_csg(300, seed=340).shape, [16, 4], UNIT, True), (scenes.random_csg(100, seed=16).shape, [32, 4], UNIT, False),
    (scenes.random_csg(300, seed=340).shape, [16, 8], UNIT, False), (CSG, [12, 8, 4], UNIT, False),
    (scenes.DEMO_SHAPES["TangleCube"](0), [12, 20, 4], DEMO, True), (scenes.DEMO_SHAPES["TangleCube"](0), [16, 8, 8], DEMO, False),
    (scenes.DEMO_SHAPES["ElasticCube"](0), [16, 8, 8], DEMO, True), (scenes.DEMO_SHAPES["ElasticCube"](0), [16, 16, 4], DEMO, False),
    (scenes.random_csg(30, seed=15).shape, [12, 8, 8], UNIT, False),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_one_tree(ctx, case):
    shape, dims, box, micro = CASES[case]
    sc = _scene(shape, dims, box)
    vs = _storage(ctx, sc)
    v = frep.Voxelizer(ctx, vs)
    v.voxelize(0.25)
    assert compare_trees_fast(vs.export(), oracle_tree(sc, vs.tape, tape_time=0.25)) == []
    ops, words = _passes(lambda: v.voxelize(0.25))
    assert (ops > words) == micro, (ops, words)
    vs.cleanup()


def test_reuse_lists_nodes_for_either_pass(ctx):
    sc = _scene(CSG, [16, 16, 4])
    want = oracle_tree(sc, sc.shape)
    other = _storage(ctx, _scene(scenes.random_csg(100, seed=17).shape, [16, 16, 4]))
    frep.Voxelizer(ctx, other).voxelize(0.0)
    vs, again = _storage(ctx, sc), _storage(ctx, sc)
    # of another scene's tree next to nothing is copied, of the same scene's all
    ops, words = _passes(lambda: frep.Voxelizer(ctx, vs).voxelize(0.0, reuse=other))
    assert ops > words
    assert compare_trees_fast(vs.export(), want) == []
    ops, words = _passes(lambda: frep.Voxelizer(ctx, again).voxelize(0.0, reuse=vs))
    assert ops < 20.0
    assert compare_trees_fast(again.export(), want) == []
    for t in (other, vs, again):
        t.cleanup()


@pytest.mark.parametrize("rounding", [1, 2])
def test_scratch_of_fitted_pools(ctx, rounding):
    """Trees whose pools leave no item room: the pass over micro-ops gets what the
    interval passes' masks take (one cell per lane from 24 slots on and in the
    hybrid mode), all, half or too little of its warps."""
    from frep.autotune import fit_pools
    for shape in (CSG, scenes.spheres_union(22).shape, scenes.spheres_union(30).shape,
                  scenes.random_csg(33, seed=33).shape, scenes.MengerSponge(2)):
        sc = _scene(shape, [16, 16, 4])
        p = fit_pools(ctx, [sc.shape], [sc.grid_dims], sc.low_vertex, sc.world_size, margin=0.25)[0]
        vs = frep.VoxelStorage(sc.grid_dims, sc.low_vertex, sc.world_size, rounding=rounding, node_words=p.node_words,
                               tape_words=p.tape_words).init(ctx, sc.shape)
        frep.Voxelizer(ctx, vs).voxelize(0.0)
        assert compare_trees_fast(vs.export(), oracle_tree(sc, vs.tape, rounding=rounding)) == [], vs.tape.n_slots
        vs.cleanup()


def test_fitted_pools_leave_room_for_one_cell_plans(ctx):
    """25 slots: the interval passes run one cell per lane and their masks hold
    less than half of a record for each warp of the pass over micro-ops."""
    from frep.autotune import fit_pools
    sc = _scene(scenes.spheres_union(22).shape, [32, 16, 4])
    p = fit_pools(ctx, [sc.shape], [sc.grid_dims], sc.low_vertex, sc.world_size, margin=0.25)[0]
    vs = frep.VoxelStorage(sc.grid_dims, sc.low_vertex, sc.world_size, node_words=p.node_words,
                           tape_words=p.tape_words).init(ctx, sc.shape)
    v = frep.Voxelizer(ctx, vs)
    v.voxelize(0.0)
    assert compare_trees_fast(vs.export(), oracle_tree(sc, vs.tape)) == []
    ops, words = _passes(lambda: v.voxelize(0.0))
    assert ops > words, (ops, words)
    vs.cleanup()


def test_batches(ctx):
    """Twelve trees are together what one of them is not; the trees of a batch
    keep one pass per last dim class, whatever else ends at that level."""
    scs = [_scene(scenes.random_csg(20 + 12 * i, seed=60 + i).shape, [16, 8, 4]) for i in range(12)]
    scs += [_scene(scenes.random_csg(25, seed=80).shape, [12, 12]), _scene(CSG, [16, 8]), _scene(CSG, [16, 4])]
    storages = [frep.VoxelStorage(sc.grid_dims, sc.low_vertex, sc.world_size, node_words=1 << 23, tape_words=1 << 23).init(
        ctx, sc.shape) for sc in scs]
    wants = [oracle_tree(sc, sc.shape) for sc in scs]
    for chosen, micro in ((list(range(12)), True), ([0, 13, 14], False), (list(range(15)), None)):
        batch = frep.Batch(ctx, [storages[i] for i in chosen])
        batch.voxelize()
        for i in chosen:
            assert compare_trees_fast(storages[i].export(), wants[i]) == [], i
        if micro is not None:
            ops, words = _passes(batch.voxelize)
            assert (ops > words) == micro, (ops, words)
        batch.close()
