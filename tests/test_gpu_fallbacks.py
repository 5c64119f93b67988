"""Calls whose larger buffers cannot be had: the staged host copies without their page-locked
slots, and order statistics without their key buffers.  The failure is simulated on the host
(qsm_ctx_inject_alloc_failure); the call then does without, with the same result.  And which
of its two ways a selection takes, seen by the kernels that ran: brackets where they can hold
the ranks, the radix passes where the sample misses them."""
import numpy as np
import pytest
import torch

import qsmgpu
from qsmgpu import Grid, inversion, nifti
from oracle import qsm_oracle as O

pytestmark = pytest.mark.gpu


def test_host_calls_without_pinned_slots():
    """A host call of 26 MB makes the device volumes (field, mask, result), then the slots."""
    grid = Grid.new(192, 128, 136)
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



# around the 24 MiB from which pageable copies are staged, and whole and broken shares of the
# staging threads
@pytest.mark.parametrize("dims", [(191, 128, 128), (192, 128, 128), (193, 128, 128), (256, 128, 128), (257, 128, 128),
                                  (256, 256, 176)], ids=lambda d: "x".join(map(str, d)))
def test_staged_copies_of_large_volumes_are_exact(ctx64, dims):
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
    np.testing.assert_array_equal(inversion.tkd(f, m, grid, (0, 0, 1), p, ctx=ctx64), out.cpu().numpy())


@pytest.mark.parametrize("dims", [(32, 32, 32), (64, 64, 65), (128, 128, 129), (200, 180, 150)],
                         ids=lambda d: "x".join(map(str, d)))
def test_nifti_images_of_every_share(ctx64, dims):
    """Float32 images of a part of a chunk to three shares, in and out of the device."""
    n = dims[0] * dims[1] * dims[2]
    v = np.random.default_rng(n).standard_normal(n).astype(np.float32).astype(np.float64)
    raw = nifti.save_nifti(v, dims, (1.0, 1.0, 1.0), np.eye(4).ravel())
    d = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    nifti.load_nifti_device(raw, d.data_ptr(), n, ctx=ctx64)
    np.testing.assert_array_equal(d.cpu().numpy(), v)
    assert nifti.save_nifti_device(d.data_ptr(), dims, (1.0, 1.0, 1.0), np.eye(4).ravel(), ctx=ctx64) == raw


PERCENTS = [0.1, 30.0, 60.0, 99.9]


def selection(n, kind):
    rng = np.random.default_rng(n)
    v = rng.standard_normal(n)
    if kind == "few":
        v = np.round(v)
    elif kind == "equal":
        v = np.full(n, -0.25)
    elif kind == "sorted":
        v = np.sort(v)
    return v


def percentiles(ctx, v, m):
    """The library's values, the oracle's, and whether the radix passes ran."""
    dv = torch.from_numpy(v).cuda()
    dm = torch.from_numpy(m).cuda() if m is not None else None
    torch.cuda.synchronize()
    ctx.set_profiling(True)
    try:
        ctx.profile_reset()
        got = inversion.prctile_device(ctx, dv.data_ptr(), dm.data_ptr() if m is not None else 0, v.size, PERCENTS)
        kernels = ctx.profile()
    finally:
        ctx.set_profiling(False)
    sel = np.sort(v if m is None else v[m > 0])
    return got, [O.prctile(sel, p) for p in PERCENTS], "select_hist" in kernels


@pytest.mark.parametrize("kind", ["normal", "few", "equal", "sorted"])
@pytest.mark.parametrize("n,keep", [(2048, 1.0), (2049, 1.0), (30011, 1.0), (300007, 0.5), (3000017, 0.3), (6000000, 1.0)])
def test_brackets_hold_the_ranks(ctx64, kind, n, keep):
    v = selection(n, kind)
    m = (np.random.default_rng(n + 1).random(n) < keep).astype(np.uint8) if keep < 1.0 else None
    got, want, radix = percentiles(ctx64, v, m)
    np.testing.assert_array_equal(got, want)
    assert not radix


def test_radix_passes_where_the_sample_misses(ctx64):
    """3000 selected values in one stretch of 3 million: two or three of the 2048 sampled
    places lie in it, too few to set a bracket."""
    v = selection(3000017, "normal")
    m = np.zeros(v.size, np.uint8)
    m[1000000:1003000] = 1
    got, want, radix = percentiles(ctx64, v, m)
    np.testing.assert_array_equal(got, want)
    assert radix


@pytest.mark.parametrize("after", [2, 3])
def test_order_statistics_without_key_buffers(after):
    """A masked selection makes the count, the bracket state and two key buffers."""
    v = selection(300007, "normal")
    m = (np.random.default_rng(4).random(v.size) < 0.5).astype(np.uint8)
    with qsmgpu.Context(0, "f64") as ctx:
        ctx.inject_alloc_failure(after)
        got, want, radix = percentiles(ctx, v, m)
        np.testing.assert_array_equal(got, want)
        assert radix
