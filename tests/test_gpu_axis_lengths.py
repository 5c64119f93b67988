"""Transform passes for every axis length: the compile-time plans without functors (88
lengths), the dense two-factor passes of the lengths with a larger prime factor, and the
functor passes around both, at each length's X, Y and Z role, on grids whose other axes
leave partial tiles.  The transform is compared with numpy's, the passes with functors
(TKD: loader, k-space operator, masked store) with the float64 oracle, and both with the
runtime engine of the same context (plan mode "runtime").

Bounds: a transform of n points as two dense factors a and b rounds each output about
sqrt(a) + sqrt(b) times: relative L2 about eps * (sqrt(a) + sqrt(b)) / sqrt(n) * sqrt(n) in
the worst arrangement, under 6e-8 * (sqrt(257) + 1) = 1e-6 in float and 2e-15 in double for
the largest prime here; three axes at most double it.  2e-6 and 1e-12 are also what the
other transform tests hold."""
import numpy as np
import pytest

import qsmgpu
from qsmgpu import Grid, inversion
from qsmgpu import fft as qfft
from oracle import qsm_oracle as O
from test_gpu_rts import case, rel
from test_more_plans import more_plans

pytestmark = pytest.mark.gpu

MORE = sorted(p[0] for p in more_plans())
# primes and products with one: smallest, around a warp and a tile, 2 p, 3 p, p q, the largest
# radix 509 and one length beyond the two-factor kernels' shared memory in double
DENSE = [17, 19, 31, 34, 37, 51, 97, 127, 131, 218, 249, 251, 257, 323, 361, 382, 509, 1018]


def roles(n):
    return [(n, 5, 7), (7, n, 3), (3, 9, n)]


def check_fft(ctx, n, tol):
    for dims in roles(n):
        grid = Grid.new(*dims)
        x = np.random.default_rng(n).standard_normal(grid.shape)
        want = np.fft.fftn(x)
        err = float(np.linalg.norm(qfft.fft3d_real(x, grid, ctx=ctx) - want) / np.linalg.norm(want))
        assert err < tol, (dims, err)


@pytest.mark.parametrize("n", DENSE)
def test_transform_dense(ctx64, ctx32, n):
    check_fft(ctx64, n, 1e-12)
    check_fft(ctx32, n, 2e-6)


@pytest.mark.parametrize("group", range(8))
def test_transform_more_plans(ctx64, ctx32, group):
    for n in MORE[group::8]:
        check_fft(ctx64, n, 1e-12)
        check_fft(ctx32, n, 2e-6)


@pytest.fixture(scope="module")
def runtime_ctxs():
    out = []
    for precision in ("f64", "mixed"):
        c = qsmgpu.Context(0, precision)
        c.plan_mode = "runtime"
        out.append(c)
    yield out
    for c in out:
        c.close()


@pytest.mark.parametrize("dims", [(37, 21, 66), (66, 37, 21), (21, 66, 37), (109, 17, 13), (15, 218, 12), (14, 19, 131),
                                  (182, 11, 9), (189, 33, 9), (2, 127, 3)],
                         ids=lambda d: "x".join(map(str, d)))
def test_functor_passes(ctx64, ctx32, runtime_ctxs, dims):
    grid = Grid.new(*dims, 1.0, 0.9, 1.2)
    bdir = (0.2, 0.3, np.sqrt(1 - 0.13))
    rng = np.random.default_rng(sum(dims))
    f = rng.standard_normal(grid.shape)
    m = (rng.random(grid.shape) < 0.7).astype(np.uint8)
    ref = O.tkd(f, m, O.Grid(grid.dims, grid.voxel_size), bdir, O.TkdParams(0.15))
    p = inversion.TkdParams(0.15)
    for ctx, rt, tol in ((ctx64, runtime_ctxs[0], 1e-11), (ctx32, runtime_ctxs[1], 1e-5)):
        got = inversion.tkd(f, m, grid, bdir, p, ctx=ctx)
        assert rel(got, ref) < tol
        assert rel(got, inversion.tkd(f, m, grid, bdir, p, ctx=rt)) < tol
        assert np.all(got[m == 0] == 0.0)


@pytest.mark.parametrize("dims", [(109, 20, 22), (20, 131, 18), (66, 78, 34), (189, 8, 6), (256, 3, 5)],
                         ids=lambda d: "x".join(map(str, d)))
def test_tv_admm_on_dense_and_long_rows(ctx64, ctx32, runtime_ctxs, dims):
    grid = Grid.new(*dims)
    f, m = case(grid, (0, 0, 1), sum(dims))
    p = inversion.TvParams(2e-4, 2e-2, 0.0, 6)
    want = inversion.tv_admm(f, m, grid, (0, 0, 1), p, ctx=runtime_ctxs[0])
    assert rel(inversion.tv_admm(f, m, grid, (0, 0, 1), p, ctx=ctx64), want) < 1e-10
    assert rel(inversion.tv_admm(f, m, grid, (0, 0, 1), p, ctx=ctx32), want) < 1e-4
