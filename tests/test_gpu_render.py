"""The renderer where its branches change, against the oracle: images that do
not fill the 8 x 8 tiles (lanes past the edge join the warp's work), cell sizes
on both sides of the reciprocal division's range, tapes with more slots than
the smallest slot array, hits on full cells of the root (the whole shape's tape
beside short ones in a warp), layers in one launch."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import frep
import oracle
from frep import csg, scenes
from parity import compare_hits, device_tree, oracle_tree, render_both

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = frep.Context(0, hbm_budget_bytes=8 << 30)
    yield c
    c.close()


def _check(ctx, sc, width, height):
    vs = device_tree(ctx, sc, rounding=1)
    orc = oracle_tree(sc, vs.tape, rounding=1)
    d_rgba, d_hits, o_rgba, o_hits = render_both(ctx, vs, orc, sc, frep.Lights(shadow_mask=1), width=width, height=height)
    assert compare_hits(d_hits, o_hits, vs.export(), orc) == []
    np.testing.assert_array_equal(d_rgba, o_rgba)
    return o_hits, vs


@pytest.mark.parametrize("width,height", [(1, 1), (7, 3), (9, 17), (33, 8), (64, 65)])
def test_image_edges(ctx, width, height):
    _check(ctx, scenes.random_csg(20, seed=3, grid_dims=[8, 8]), width, height)


@pytest.mark.parametrize("world,dims", [(4.0, (8, 8)), (2.5, (12, 4)), (2.5, (4, 4, 4, 4, 4)), (1e8, (4, 4)),
                                        (2.0 ** 27, (4, 8)), (2.0 ** -18, (4, 4))])
def test_world_sizes(ctx, world, dims):
    sc = scenes.random_csg(12, seed=5, grid_dims=list(dims))
    sc = dataclasses.replace(sc, low_vertex=(-world / 2,) * 3, world_size=world)
    _check(ctx, sc, 96, 64)


def test_full_root_cells_beside_short_tapes(ctx):
    """An orthographic camera in the middle of the scene: rays that start inside
    the box end at once on full root cells, the others on the last level."""
    sc = scenes.random_csg(60, seed=9, grid_dims=[16, 4])
    body = csg.Box((-0.5, -0.5, -0.5), (1.0, 1.0, 1.0))
    cam = dataclasses.replace(sc.camera, position=(0.0, 0.1, 0.0), orthographic=True, ortho_width=2.4)
    sc = dataclasses.replace(sc, shape=csg.Union(sc.shape, body), camera=cam)
    hits, _ = _check(ctx, sc, 256, 192)
    assert (hits[..., 4] == 0).any() and (hits[..., 4] == 1).any()


@pytest.mark.parametrize("n", [40, 70])  # more than 32, more than 64 slots
def test_many_slots(ctx, n):
    a = 2.399963  # a polygon's sides, each used twice, first to last and last to first
    sides = [csg.X() * float(np.cos(a * i)) + csg.Y() * float(np.sin(a * i)) - 0.8 for i in range(n)]
    up, down = sides[0], sides[-1]
    for i in range(1, n):
        up = csg.Max(up, sides[i])
        down = csg.Max(down, sides[-1 - i] * (1.0 + 0.001 * i))
    sc = scenes.random_csg(4, seed=1, grid_dims=[8, 4])
    sc = dataclasses.replace(sc, shape=csg.Max(csg.Max(up, down), csg.Abs(csg.Z()) - 0.5))
    assert frep.Tape(sc.shape).n_slots > (32 if n == 40 else 64)
    hits, _ = _check(ctx, sc, 60, 44)
    assert (hits[..., 4] != 0xFFFFFFFF).any()


def test_temporal_layers_odd_size(ctx):
    import torch
    sc = scenes.random_csg(16, seed=21, grid_dims=[12, 4], width=37, height=21)
    vs = device_tree(ctx, sc, rounding=1)
    orc = oracle_tree(sc, vs.tape, rounding=1)
    rt = frep.Raytracer(ctx, vs)
    rt.lights = frep.Lights(shadow_mask=1)
    cam = dataclasses.replace(sc.camera, jitter_seed=0.5)
    _, layers = rt.trace_temporal(cam, 0.0, sc.width, sc.height, 3)
    torch.cuda.synchronize()
    for i in range(3):
        ci = dataclasses.replace(cam, jitter=True, jitter_seed=0.5 + i)
        want, _ = orc.render(oracle.camera_vector(ci, sc.width, sc.height), rt.lights, 0.0)
        np.testing.assert_array_equal(layers[i].cpu().numpy(), want)


@pytest.mark.parametrize("world,dims", [(2500.0, (4, 4, 4, 4)), (25000.0, (4, 4, 4)), (1e8, (4, 4))])
def test_rays_that_stop_advancing(ctx, world, dims):
    """Steps smaller than the spacing of t: rays repeat their cells until the
    step bound, and their records say so."""
    sc = scenes.random_csg(12, seed=5, grid_dims=list(dims))
    sc = dataclasses.replace(sc, low_vertex=(-world / 2,) * 3, world_size=world)
    vs = device_tree(ctx, sc, rounding=1)
    orc = oracle_tree(sc, vs.tape, rounding=1)
    d_rgba, d_hits, o_rgba, o_hits = render_both(ctx, vs, orc, sc, frep.Lights(shadow_mask=1), width=96, height=64)
    np.testing.assert_array_equal(d_hits[..., 7], o_hits[..., 7])
    assert o_hits[..., 7].max() == 65537
    np.testing.assert_array_equal(d_rgba, o_rgba)
