"""RTS and RESHARP in a mixed context hand their single-precision maps on as doubles, and a
program that compares two runs of them compares doubles: a change of the kernels must not
move them.  tests/golden/mixed_maps.json holds values of such maps at fixed places (inputs
from the seeds below) over the forms that an axis can take: compile-time lists, run-time
Stockham and Bluestein lengths, in-plane sizes of the plane kernels, short and long axes.
Bound: 1e-9 relative, that of doubles (a rounding of the maps' own arithmetic is 6e-8)."""
import json
import os

import numpy as np
import pytest

from qsmgpu import Grid, bgremove, inversion

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "mixed_maps.json")
DIMS = [(64, 64, 20), (96, 128, 96), (36, 40, 44), (37, 34, 29), (189, 33, 18), (80, 72, 100), (160, 24, 144), (20, 218, 22),
        (30, 14, 131), (400, 18, 16), (16, 22, 448), (101, 103, 107), (182, 218, 182)]
PLACES = 200


def inputs(dims):
    """A field with structure inside an ellipsoid, from integer arithmetic and one generator."""
    nx, ny, nz = dims
    rng = np.random.default_rng(1000003 * nx + 1009 * ny + nz)
    z, y, x = np.meshgrid(*[np.arange(n) for n in (nz, ny, nx)], indexing="ij", sparse=True)
    mask = sum(((2.0 * a - (n - 1)) / (0.9 * n)) ** 2 for a, n in ((x, nx), (y, ny), (z, nz))) < 1.0
    f = rng.standard_normal((nz, ny, nx)) * 0.01 + ((x // 5 + y // 7 + z // 3) % 4) * 0.02
    return Grid.new(nx, ny, nz), f * mask, mask.astype(np.uint8)


def maps(dims, ctx):
    grid, f, m = inputs(dims)
    chi = inversion.rts(f, m, grid, (0.2, 0.3, np.sqrt(1 - 0.13)), ctx=ctx)
    local, eroded = bgremove.resharp(f, m, grid, bgremove.ResharpParams(radius=3.0, max_iter=12), ctx=ctx)
    return {"rts": chi, "resharp": local}, eroded


def sampled(dims, out):
    at = np.random.default_rng(sum(dims)).integers(0, out.size, PLACES)
    inside = np.flatnonzero(out.reshape(-1))
    at[::2] = inside[np.linspace(0, inside.size - 1, at[::2].size).astype(np.int64)]
    return at, out.reshape(-1)[at]


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_mixed_maps_stay(ctx32, dims):
    with open(GOLDEN) as f:
        want = json.load(f)["x".join(map(str, dims))]
    got, eroded = maps(dims, ctx32)
    assert int(eroded.sum()) == want["eroded"]
    for name, out in got.items():
        w = want[name]
        assert np.linalg.norm(out) == pytest.approx(w["norm"], rel=1e-9), name
        _, v = sampled(dims, out)
        scale = np.maximum(np.abs(w["values"]), w["norm"] / np.sqrt(out.size))
        worst = float(np.max(np.abs(v - np.array(w["values"])) / scale))
        assert worst <= 1e-9, (name, worst)
