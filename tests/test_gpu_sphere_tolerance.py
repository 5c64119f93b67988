"""Mask erosion by spheres that tolerate missing voxels (SHARP's and V-SHARP's threshold), by
the number they tolerate: 0, 1, 2 (bit planes), 3 and more (sums through transforms), and
masks with values above 1.  Masks are compared exactly with the oracle's; the masks are full
but for zero voxels placed close together, so that the spheres around them miss from one to
all of them.  A call's device time must not depend on the mask's values: a mask of threes costs
the transform of one mask and one filter per radius more than a 0/1 mask, about twice a radius'
own work; four times is allowed."""
import numpy as np
import pytest
import torch

from qsmgpu import Grid, bgremove
from oracle import qsm_oracle as O

pytestmark = pytest.mark.gpu


def og(grid):
    return O.Grid(grid.dims, grid.voxel_size)


def holed(grid, count, seed):
    """Ones with `count` zeros inside a cube of 4 voxels, and as many strewn about."""
    rng = np.random.default_rng(seed)
    m = np.ones(grid.shape, np.uint8)
    at = np.array([n // 3 for n in grid.shape])
    for k in range(count):
        m[tuple(at + rng.integers(0, 4, 3))] = 0
        m[tuple(int(rng.integers(0, n)) for n in grid.shape)] = 0
    return m


# radius in voxels, voxels inside, tolerated: 8 (2109, 0), 10 (4169, 1), 12 (7153, 2), 14
# (11513, 3), 20 (33401, 10), and 12 mm at 0.8, 0.5 and 0.4 mm
@pytest.mark.parametrize("vs,radius,dims", [(1.0, 8.0, (40, 36, 33)), (1.0, 10.0, (48, 41, 36)), (1.0, 12.0, (45, 48, 50)),
                                            (1.0, 14.0, (64, 60, 49)), (1.0, 20.0, (72, 66, 64)), (0.8, 12.0, (50, 48, 44)),
                                            (0.5, 12.0, (80, 64, 70)), (0.4, 12.0, (70, 96, 66))])
def test_tolerances(ctx64, ctx32, vs, radius, dims):
    grid = Grid.new(*dims, vs, vs, vs)
    total = int(np.count_nonzero(O.smv_kernel(og(grid), radius)))
    tol = total - (int(np.floor((1.0 - np.sqrt(1e-7)) * total)) + 1)
    f = np.random.default_rng(1).standard_normal(grid.shape) * 0.01
    for count in sorted({1, tol, tol + 1, 2 * tol + 2} - {0}):
        m = holed(grid, count, count)
        _, want = O.sharp(f, m, og(grid), O.SharpParams(0.05, radius))
        for ctx in (ctx64, ctx32):
            _, got = bgremove.sharp(f, m, grid, bgremove.SharpParams(0.05, radius), ctx=ctx)
            assert np.array_equal(got, want), (count, tol)


@pytest.mark.parametrize("radii", [[20.0, 14.0, 12.0, 11.0, 10.0, 3.0], list(np.linspace(14.0, 1.0, 260))],
                         ids=["mixed", "many"])
def test_vsharp_over_tolerances(ctx64, radii):
    grid = Grid.new(44, 40, 37) if len(radii) < 10 else Grid.new(30, 32, 29)
    f = np.random.default_rng(2).standard_normal(grid.shape) * 0.01
    m = holed(grid, 8, 5)
    weighted = m * np.random.default_rng(3).integers(1, 4, m.shape).astype(np.uint8)
    for mask in (m, weighted):
        _, want = O.vsharp_with_radii(f, mask, og(grid), radii, 0.05)
        _, got = bgremove.vsharp_with_radii(f, mask, grid, radii, 0.05, ctx=ctx64)
        assert np.array_equal(got, want)


def test_time_does_not_depend_on_the_masks_values(ctx32):
    grid = Grid.new(192, 192, 128)
    z, y, x = np.meshgrid(*[np.arange(n) for n in grid.shape], indexing="ij", sparse=True)
    m = (sum(((2.0 * a - (n - 1)) / (0.85 * n)) ** 2 for a, n in zip((x, y, z), grid.dims)) < 1).astype(np.uint8)
    f = torch.randn(grid.shape, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    out, om = torch.empty_like(f), torch.empty(grid.shape, dtype=torch.uint8, device="cuda")

    def device_ms(mask):
        dm = torch.from_numpy(mask).cuda()
        torch.cuda.synchronize()
        call = lambda: bgremove.vsharp_with_radii_device(ctx32, f.data_ptr(), dm.data_ptr(), grid,
                                                         [float(r) for r in range(12, 0, -1)], 0.05, out.data_ptr(),
                                                         om.data_ptr())
        call()
        ctx32.set_profiling(True)
        try:
            ctx32.profile_reset()
            call()
            return sum(ms for _, ms in ctx32.profile().values())
        finally:
            ctx32.set_profiling(False)

    assert device_ms(3 * m) < 4.0 * device_ms(m)
