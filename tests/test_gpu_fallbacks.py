"""Calls whose larger buffers cannot be had: the staged host copies without their page-locked
slots.  The failure is simulated on the host (qsm_ctx_inject_alloc_failure); the call then
does without, with the same result."""
import numpy as np
import pytest
import torch

import qsmgpu
from qsmgpu import Grid, inversion

pytestmark = pytest.mark.gpu


def test_host_calls_without_pinned_slots():
    """A host call of 8 MB makes the device volumes (field, mask, result), then the slots."""
    grid = Grid.new(128, 128, 64)
    rng = np.random.default_rng(1)
    f = rng.standard_normal(grid.shape)
    m = (rng.random(grid.shape) < 0.5).astype(np.uint8)
    p = inversion.TkdParams(0.2)
    with qsmgpu.Context(0, "f64") as ctx:
        want = inversion.tkd(f, m, grid, (0, 0, 1), p, ctx=ctx)
    with qsmgpu.Context(0, "f64") as ctx:
        ctx.inject_alloc_failure(3)
        np.testing.assert_array_equal(inversion.tkd(f, m, grid, (0, 0, 1), p, ctx=ctx), want)
        # the failure was taken by the slots, and the next copies have them
        np.testing.assert_array_equal(inversion.tkd(f, m, grid, (0, 0, 1), p, ctx=ctx), want)
