"""Sphere kernels without transforms (spectrum by cosine sums, erosion by distance and by
counts), order statistics by sampled brackets, staged host copies and the wrapped Laplacian,
each at the sizes where its cases meet.  Masks, ranks and copies are compared exactly; fields
with the oracle at the bound the background-removal tests hold (1e-10 relative L2 in double:
the sphere spectrum sums at most a few thousand cosines, each to 1e-15)."""
import numpy as np
import pytest
import torch

import qsmgpu
from qsmgpu import Grid, bgremove, inversion, unwrap
from oracle import qsm_oracle as O
from test_gpu_rts import rel

pytestmark = pytest.mark.gpu


def og(grid):
    return O.Grid(grid.dims, grid.voxel_size)


def volume(dims, seed, vs=(1.0, 1.0, 1.0), holes=0.02):
    grid = Grid.new(*dims, *vs)
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*[np.arange(n) for n in grid.shape], indexing="ij")
    m = sum(((a - (n - 1) / 2) / (0.55 * n)) ** 2 for a, n in ((x, grid.nx), (y, grid.ny), (z, grid.nz))) < 1
    m &= rng.random(grid.shape) > holes
    return grid, rng.standard_normal(grid.shape) * 0.01, m.astype(np.uint8)


# odd and even lengths, a radius below one voxel, one that reaches half the volume (2 r + 1 = nx,
# 2 r = nx) and beyond it, rows longer than a warp and than two words, anisotropic voxels
@pytest.mark.parametrize("dims,vs,radius", [
    ((9, 8, 7), (1.0, 1.0, 1.0), 0.6), ((9, 8, 7), (1.0, 1.0, 1.0), 1.0), ((9, 10, 11), (1.0, 1.0, 1.0), 4.0),
    ((8, 8, 8), (1.0, 1.0, 1.0), 4.0), ((7, 6, 5), (1.0, 1.0, 1.0), 5.0), ((33, 18, 17), (0.6, 0.9, 1.3), 3.0),
    ((66, 9, 10), (1.0, 1.5, 0.7), 2.5), ((31, 32, 33), (1.0, 1.0, 1.0), 6.0), ((40, 36, 3), (1.0, 1.0, 2.0), 3.0)])
def test_smv_spheres(ctx64, ctx32, dims, vs, radius):
    grid, f, m = volume(dims, sum(dims), vs)
    lr, mr = O.smv(f, m, og(grid), radius)
    for ctx, tol in ((ctx64, 1e-10), (ctx32, 1e-5)):
        lo, mo = bgremove.smv(f, m, grid, radius, ctx=ctx)
        assert np.array_equal(mo, mr)
        # absolute to the field: a mask eroded to a few voxels leaves no scale of its own
        assert np.linalg.norm(lo - lr) <= tol * np.linalg.norm(f)


@pytest.mark.parametrize("dims,vs", [((24, 22, 20), (1.0, 1.0, 1.0)), ((33, 31, 17), (0.8, 1.0, 1.25)),
                                     ((70, 12, 13), (1.0, 1.0, 1.0))])
def test_vsharp_radii_reach_across_the_faces(ctx64, ctx32, dims, vs):
    """Full masks wrap around the faces; a weighted one (values above 1) takes the counts."""
    for kind in ("holes", "full", "weighted"):
        grid, f, m = volume(dims, 7, vs)
        if kind == "full":
            m = np.ones_like(m)
        if kind == "weighted":
            m = m * np.random.default_rng(3).integers(1, 4, m.shape).astype(np.uint8)
        radii = [5.0, 4.0, 3.0, 2.0, 1.0]
        lr, mr = O.vsharp_with_radii(f, m, og(grid), radii, 0.05)
        for ctx, tol in ((ctx64, 1e-9), (ctx32, 1e-4)):
            lo, mo = bgremove.vsharp_with_radii(f, m, grid, radii, 0.05, ctx=ctx)
            assert np.array_equal(mo, mr), kind
            assert np.linalg.norm(lo - lr) <= tol * np.linalg.norm(f), kind


RANKS = [0.0, 0.1, 30.0, 50.0, 60.0, 99.9, 100.0]


# one sort's size and its neighbours, one and several bracket passes, masks that leave little
@pytest.mark.parametrize("n,keep", [(2047, 1.0), (2048, 1.0), (2049, 1.0), (4096, 0.5), (30011, 1.0), (300007, 0.02),
                                    (300007, 0.9), (3000017, 0.3)])
@pytest.mark.parametrize("values", ["normal", "few", "equal", "infinite", "sorted"])
def test_rank_brackets_match_sort(ctx64, n, keep, values):
    rng = np.random.default_rng(n)
    v = rng.standard_normal(n)
    if values == "few":
        v = np.round(v)
    elif values == "equal":
        v = np.full(n, -0.25)
    elif values == "infinite":
        v[rng.random(n) < 0.4] = np.inf
        v[rng.random(n) < 0.1] = -np.inf
    elif values == "sorted":
        v = np.sort(v)
    m = None
    if keep < 1.0:
        # one contiguous stretch and scattered voxels: strided samples that miss the mask
        m = (rng.random(n) < keep / 2).astype(np.uint8)
        m[n // 3:n // 3 + int(n * keep / 2)] = 1
    dv = torch.from_numpy(v).cuda()
    dm = torch.from_numpy(m).cuda() if m is not None else None
    sel = np.sort(v if m is None else v[m > 0])
    with np.errstate(invalid="ignore"):
        want = [O.prctile(sel, p) for p in RANKS]
    for _ in range(2):
        got = inversion.prctile_device(ctx64, dv.data_ptr(), dm.data_ptr() if m is not None else 0, n, RANKS)
        np.testing.assert_array_equal(got, want)


# around the 4 MiB from which pageable copies are staged, around whole 1 MiB slots, more than
# eight threads' two slots each
@pytest.mark.parametrize("dims", [(128, 64, 63), (127, 65, 64), (128, 64, 64), (129, 64, 64), (131, 127, 1),
                                  (128, 128, 129), (160, 150, 101)], ids=lambda d: "x".join(map(str, d)))
def test_staged_copies_are_exact(ctx64, dims):
    grid = Grid.new(*dims)
    rng = np.random.default_rng(sum(dims))
    f = rng.standard_normal(grid.shape)
    m = (rng.random(grid.shape) < 0.5).astype(np.uint8)
    p = inversion.TkdParams(0.2)
    df, dm = torch.from_numpy(f).cuda(), torch.from_numpy(m).cuda()
    out = torch.empty(grid.shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    inversion.tkd_device(ctx64, df.data_ptr(), dm.data_ptr(), grid, (0, 0, 1), p, out.data_ptr())
    torch.cuda.synchronize()
    want = out.cpu().numpy()
    np.testing.assert_array_equal(inversion.tkd(f, m, grid, (0, 0, 1), p, ctx=ctx64), want)
    pinned = torch.from_numpy(f).pin_memory().numpy()
    np.testing.assert_array_equal(inversion.tkd(pinned, m, grid, (0, 0, 1), p, ctx=ctx64), want)


@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 5, 7), (33, 8, 9), (64, 3, 2), (31, 17, 5), (257, 4, 3)],
                         ids=lambda d: "x".join(map(str, d)))
def test_wrapped_laplacian_edges(ctx64, ctx32, dims):
    grid = Grid.new(*dims, 0.9, 1.1, 1.3)
    rng = np.random.default_rng(sum(dims))
    phase = rng.uniform(-np.pi, np.pi, grid.shape)
    m = (rng.random(grid.shape) < 0.8).astype(np.uint8)
    ref = O.laplacian_unwrap(phase, m, og(grid))
    for ctx, tol in ((ctx64, 1e-10), (ctx32, 1e-4)):
        assert rel(unwrap.laplacian_unwrap(phase, m, grid, ctx=ctx), ref) < tol
