"""RTS at long z axes: which lengths it refuses (those whose multiplier pass the run-time
engine cannot hold in one kernel: by their plan, in each precision), and its values at the
longest ones it takes, against the float64 oracle at test_gpu_rts's bounds."""
import numpy as np
import pytest

import qsmgpu
from qsmgpu import Grid, inversion
from oracle import qsm_oracle as O
from test_gpu_rts import case, rel

pytestmark = pytest.mark.gpu

# Stockham and Bluestein lengths on both sides of each line
TAKEN = {"f64": [853, 960, 1175, 1201, 1728, 1792, 2000, 2048, 2058], "mixed": [599, 1023, 1120, 1152, 1792, 1875, 1920, 2048]}
REFUSED = {"f64": [961, 1010, 1755, 1782, 1944, 2047, 2079, 2112, 4032, 4096],
           "mixed": [601, 641, 1188, 1215, 1458, 2047, 2430, 3375, 3600, 4096]}


def ask(ctx, n):
    g = Grid.new(2, 2, n)
    return inversion.rts(np.ones(g.shape), np.ones(g.shape, np.uint8), g, (0, 0, 1), inversion.RtsParams(max_iter=1), ctx=ctx)


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_refusals(precision):
    with qsmgpu.Context(0, precision) as ctx:
        for n in TAKEN[precision]:
            assert np.isfinite(ask(ctx, n)).all(), n
        for n in REFUSED[precision]:
            with pytest.raises(qsmgpu.QsmError):
                ask(ctx, n)


@pytest.mark.parametrize("precision,nz", [("f64", 1201), ("f64", 2048), ("f64", 2058), ("mixed", 1023), ("mixed", 2048)])
def test_values(ctx64, ctx32, precision, nz):
    bdir = (0.2, 0.3, np.sqrt(1 - 0.13))
    grid = Grid.new(6, 5, nz)
    f, m = case(grid, bdir, nz)
    p = dict(tol=0.0, max_iter=6)
    ref = O.rts(f, m, O.Grid(grid.dims, grid.voxel_size), bdir, O.RtsParams(**p), exact_dc=True)
    ctx, tol = (ctx64, 1e-9) if precision == "f64" else (ctx32, 1e-4)
    assert rel(inversion.rts(f, m, grid, bdir, inversion.RtsParams(**p), ctx=ctx), ref) < tol
