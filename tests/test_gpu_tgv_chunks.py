"""TGV's columns by the planes a thread owns: one (the kernels' one-plane form, up to a wave of
single planes), two to four, and boxes at both sides of the first line; against the float32
oracle after 8 iterations at the 1e-4 of test_gpu_half_spectrum's columns."""
import numpy as np
import pytest

from qsmgpu import Grid, inversion
from oracle import qsm_oracle as O
from test_gpu_ilsqr import OBLIQUE, og
from test_gpu_rts import rel
from test_gpu_tgv import phantom_phase

pytestmark = pytest.mark.gpu

# full masks, one erosion and the inner one: the box is the whole volume, in 32x4 tiles; 1184
# blocks are a wave of eight on each of 148 SMs
DIMS = [(40, 36, 20), (32, 60, 78), (32, 64, 74), (32, 64, 75), (64, 64, 37), (64, 64, 38), (64, 64, 64), (96, 80, 60),
        (100, 96, 70)]


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_chunks(ctx64, dims):
    grid = Grid.new(*dims, 1.0, 1.1, 0.9)
    phase, _ = phantom_phase(grid, OBLIQUE, sum(dims))
    m = np.ones(grid.shape, np.uint8)
    m[tuple(n // 2 for n in grid.shape)] = 0  # and a hole
    p = dict(iterations=8, erosions=1)
    got = inversion.tgv_qsm(phase, m, grid, inversion.TgvParams(**p), OBLIQUE, ctx=ctx64)
    ref = O.tgv_qsm(phase, m, og(grid), O.TgvParams(**p), OBLIQUE)
    assert rel(got, ref) < 1e-4
