"""Point evaluation on the device where its kernels change (one or four points
per thread, slots in shared or global memory, tails of blocks), against the
host's evaluation of the same tape (the same operations, the same bits)."""
from __future__ import annotations

import numpy as np
import pytest

import frep
from frep import csg, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = frep.Context(0, hbm_budget_bytes=4 << 30)
    yield c
    c.close()


def _many_slots(n):
    a = 2.399963
    sides = [csg.X() * float(np.cos(a * i)) + csg.Y() * float(np.sin(a * i)) - 0.8 for i in range(n)]
    up, down = sides[0], sides[-1]
    for i in range(1, n):
        up = csg.Max(up, sides[i])
        down = csg.Max(down, sides[-1 - i] * (1.0 + 0.001 * i))
    return csg.Max(up, down)


FEW = 148 * 2 * 64 * 4  # from here four points per thread


@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000, FEW - 1, FEW, FEW + 257])
@pytest.mark.parametrize("shape", ["csg", "ElasticCube", "-x", "spheres", "constant", 36, 60])
def test_points_equal_the_host(ctx, n, shape):
    expr = {"csg": lambda: scenes.random_csg(12, seed=4).shape, "ElasticCube": lambda: scenes.DEMO_SHAPES["ElasticCube"](0),
            "-x": lambda: -csg.X(), "spheres": lambda: scenes.spheres_union(70).shape,
            "constant": lambda: csg.Constant(1.5) + csg.Constant(0.25)}.get(shape, lambda: _many_slots(shape))()
    tape = frep.Tape(expr)
    if shape == "spheres":  # its constants are not rows
        assert tape.n_slots > 48
    rng = np.random.default_rng(n)
    pts = rng.uniform(-2, 2, (n, 4)).astype(np.float32)
    if n > 60:
        pts[7] = [np.nan, 0.5, -0.0, 1.0]
        pts[21] = [np.inf, -np.inf, 0.25, 0.0]
    np.testing.assert_array_equal(ctx.eval_points(tape, pts).view(np.uint32) & _nan_mask(ctx.eval_points(tape, pts)),
                                  tape.eval_points(pts).view(np.uint32) & _nan_mask(tape.eval_points(pts)))


def _nan_mask(v):
    """All bits, or for a NaN the exponent's (its payload is the processor's)."""
    return np.where(np.isnan(v), np.uint32(0x7F800000), np.uint32(0xFFFFFFFF))
