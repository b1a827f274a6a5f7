"""The last-level pass over micro-ops (leaf_level_kernel) at the edges of its
work split: every power-of-two last dim, tapes that fit one staging and that do
not, few tapes (decoded by the whole warp) and many (one per lane), nodes that
share a tape and that do not, opcodes outside the jump table; and the sizes that
stay with the point pass (slot files above 32, last dims that are no power of
two). Each tree equals the oracle's bit for bit, alone and in a batch of all."""
from __future__ import annotations

import pytest

import frep
from frep import scenes
from parity import compare_trees_fast, device_tree, oracle_tree

pytestmark = pytest.mark.gpu

CASES = [
    ("csg", 5, [8, 4]), ("csg", 33, [16, 4]), ("csg", 300, [16, 4]), ("csg", 200, [16, 8, 4]), ("csg", 60, [16, 8]),
    ("csg", 90, [8, 16]), ("csg", 25, [4, 32]), ("csg", 260, [8, 8]), ("csg", 40, [12, 12]), ("csg", 40, [20, 4]),
    ("spheres", 3, [4]), ("spheres", 1, [16]), ("spheres", 45, [16, 4]), ("gyroid", 8, [16, 8, 4]), ("gyroid", 3, [16, 8]),
]


@pytest.fixture(scope="module")
def ctx():
    return frep.Context(0, hbm_budget_bytes=24 << 30)


def _scene(kind, n, dims):
    if kind == "csg":
        return scenes.random_csg(n, seed=40 + n, grid_dims=dims)
    if kind == "gyroid":
        return scenes.stress_gyroid(n, seed=3, grid_dims=dims)
    sc = scenes.spheres_union(n, seed=n)
    sc.grid_dims = list(dims)
    return sc


def test_trees_equal_the_oracle_alone_and_in_a_batch(ctx):
    scs, storages, oracles = [], [], []
    for kind, n, dims in CASES:
        sc = _scene(kind, n, dims)
        vs = frep.VoxelStorage(sc.grid_dims, sc.low_vertex, sc.world_size, node_words=1 << 25, tape_words=1 << 24)
        vs.init(ctx, sc.shape)
        frep.Voxelizer(ctx, vs).voxelize(0.25)
        oracles.append(oracle_tree(sc, vs.tape, tape_time=0.25))
        assert compare_trees_fast(vs.export(), oracles[-1]) == [], (kind, n, dims)
        scs.append(sc)
        storages.append(vs)
    batch = frep.Batch(ctx, storages)
    batch.voxelize([0.25] * len(storages))
    for case, vs, orc in zip(CASES, storages, oracles):
        assert compare_trees_fast(vs.export(), orc) == [], case
    batch.close()


def test_wide_slot_files_keep_the_point_pass(ctx):
    sc = scenes.spheres_union(40, seed=2)
    sc.grid_dims = [16, 4]
    tape = frep.Tape(sc.shape, const_reload=0xFFFFFFFF)
    assert tape.n_slots > 32
    vs = device_tree(ctx, scenes.Scene("wide", tape, sc.grid_dims, sc.low_vertex, sc.world_size, sc.camera, 64, 64))
    assert compare_trees_fast(vs.export(), oracle_tree(sc, tape)) == []
