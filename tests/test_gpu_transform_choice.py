"""Which form of transform a length takes (two_factor.cu).  The dense two-factor passes are
taken only where their error is no larger than the run-time engine's, and lengths above 384
with prime factors up to 13 stay on the run-time Stockham engine, which is faster there: such
a pass gives the run-time engine's own bits.  Errors are against 80-bit transforms of the same
values, over all three axis roles; the two forms' errors are sample statistics of some 10^4
outputs, equal within 1 % where the forms tie, so 1.02 separates them from a form that is
worse."""
import numpy as np
import pytest
import scipy.fft

import qsmgpu
from qsmgpu import Grid
from qsmgpu import fft as qfft

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def runtime_ctxs():
    out = {}
    for precision in ("f64", "mixed"):
        out[precision] = qsmgpu.Context(0, precision)
        out[precision].plan_mode = "runtime"
    yield out
    for c in out.values():
        c.close()


def error(ctx, x, grid, exact):
    y = qfft.fft3d_real(x, grid, ctx=ctx)
    d = np.stack([(y.real - exact.real).astype(np.float64), (y.imag - exact.imag).astype(np.float64)])
    return float(np.linalg.norm(d) / np.linalg.norm(exact.astype(np.complex128)))


# primes and products around the lines in each precision, and the largest radix of each
@pytest.mark.parametrize("n", [97, 131, 139, 173, 179, 197, 227, 254, 271, 307, 346, 349, 367, 373, 383, 394, 446, 509])
def test_error_is_no_larger_than_the_engines(ctx64, ctx32, runtime_ctxs, n):
    for dims in ((n, 24, 21), (24, n, 21), (24, 21, n)):
        grid = Grid.new(*dims)
        x = np.random.default_rng(n).standard_normal(grid.shape)
        exact = scipy.fft.fftn(x.astype(np.longdouble))
        for ctx, precision in ((ctx64, "f64"), (ctx32, "mixed")):
            got, ref = (error(c, x, grid, exact) for c in (ctx, runtime_ctxs[precision]))
            assert got <= 1.02 * ref, (dims, precision, got, ref)


@pytest.mark.parametrize("n", [385, 400, 448, 500, 512, 576, 768])
def test_long_smooth_lengths_stay_on_the_engine(ctx64, ctx32, runtime_ctxs, n):
    for dims in ((n, 1, 1), (1, n, 1), (1, 1, n)):
        grid = Grid.new(*dims)
        x = np.random.default_rng(n).standard_normal(grid.shape)
        for ctx, precision in ((ctx64, "f64"), (ctx32, "mixed")):
            np.testing.assert_array_equal(qfft.fft3d_real(x, grid, ctx=ctx),
                                          qfft.fft3d_real(x, grid, ctx=runtime_ctxs[precision]))
