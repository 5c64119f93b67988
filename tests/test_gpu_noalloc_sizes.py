"""qsm_tkd_device_noalloc over the forms its passes take without buffers of their own: listed
lengths in small and larger volumes (functors inside the pass or staged in the output buffer,
the Z multiplier in it), dense and Bluestein lengths, long rows, and rows so short that the
multiplier does not fit the output buffer; out of place, in place, and into a buffer on an odd
multiple of 8 bytes (the multiplier's copies are of 16).  1e-10 relative to the
regular entry point, as in test_zz_no_alloc."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from qsmgpu import Grid, _lib, inversion

pytestmark = pytest.mark.gpu

DIMS = [(48, 40, 36), (128, 96, 90), (66, 189, 100), (128, 128, 128), (101, 34, 37), (37, 101, 227), (400, 40, 30),
        (30, 26, 448), (3, 50, 60), (5, 64, 70), (2, 9, 128)]


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_noalloc(ctx64, dims):
    grid = Grid.new(*dims, 1.0, 0.9, 1.1)
    rng = np.random.default_rng(sum(dims))
    f = torch.from_numpy(rng.standard_normal(grid.shape) * 0.05).cuda()
    m = torch.from_numpy((rng.random(grid.shape) > 0.15).astype(np.uint8)).cuda()
    want, got = torch.empty_like(f), torch.full_like(f, float("nan"))
    torch.cuda.synchronize()
    bdir = (math.sin(0.3), 0.1, math.cos(0.3))
    inversion.tkd_device(ctx64, f.data_ptr(), m.data_ptr(), grid, bdir, inversion.TkdParams(0.19), want.data_ptr())
    lib = _lib.load()
    b = C.cast((C.c_double * 3)(*bdir), _lib.c_double_p)
    g, p = grid._c(), _lib.QsmTkdParams(0.19)
    stream = torch.cuda.current_stream().cuda_stream
    same = f.clone()
    odd = torch.empty(f.numel() + 1, dtype=torch.float64, device="cuda")[1:].view(f.shape)
    for src, dst in ((f, got), (same, same), (f, odd)):
        assert lib.qsm_tkd_device_noalloc(C.c_void_p(src.data_ptr()), C.c_void_p(m.data_ptr()), C.byref(g), b, C.byref(p),
                                          C.c_void_p(dst.data_ptr()), C.c_void_p(stream)) == 0
        torch.cuda.synchronize()
        err = float((dst - want).norm() / want.norm())
        assert err < 1e-10, err
