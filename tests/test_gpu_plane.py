"""The X and Y passes of small in-plane matrices as one kernel (csrc/plane.cuh): every pair of
its lengths, plane counts at the ends of its rule and just outside it, against the runtime
engine of the same precision (TV-ADMM) and the float64 oracle (TKD).  Bounds: 1e-11 and 1e-5
for one chain of transforms, 1e-10 and 1e-4 for a few iterations, as in
test_gpu_axis_lengths."""
import numpy as np
import pytest

import qsmgpu
from qsmgpu import Grid, inversion
from oracle import qsm_oracle as O
from test_gpu_rts import case, rel

pytestmark = pytest.mark.gpu

SIZES = [(64, 64, 5), (64, 64, 31), (64, 64, 32), (64, 96, 33), (64, 128, 47), (64, 64, 150), (96, 64, 95), (128, 64, 89),
         (96, 96, 88), (96, 96, 89), (96, 128, 100), (128, 96, 120), (128, 128, 148), (128, 128, 149)]


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


@pytest.mark.parametrize("dims", SIZES, ids=lambda d: "x".join(map(str, d)))
def test_plane_kernels(ctx64, ctx32, runtime_ctxs, dims):
    grid = Grid.new(*dims, 1.0, 0.9, 1.2)
    bdir = (0.2, 0.3, np.sqrt(1 - 0.13))
    rng = np.random.default_rng(sum(dims))
    f = rng.standard_normal(grid.shape)
    m = (rng.random(grid.shape) < 0.7).astype(np.uint8)
    ref = O.tkd(f, m, O.Grid(grid.dims, grid.voxel_size), bdir, O.TkdParams(0.15))
    for ctx, tol in ((ctx64, 1e-11), (ctx32, 1e-5)):
        got = inversion.tkd(f, m, grid, bdir, inversion.TkdParams(0.15), ctx=ctx)
        assert rel(got, ref) < tol and np.all(got[m == 0] == 0.0)
    fp, mp = case(grid, bdir, sum(dims))
    p = inversion.TvParams(2e-4, 2e-2, 0.0, 4)
    want = inversion.tv_admm(fp, mp, grid, bdir, p, ctx=runtime_ctxs[0])
    assert rel(inversion.tv_admm(fp, mp, grid, bdir, p, ctx=ctx64), want) < 1e-10
    assert rel(inversion.tv_admm(fp, mp, grid, bdir, p, ctx=ctx32), want) < 1e-4
