"""iLSQR where its half-spectrum passes are compile-time kernels: base and wide lengths on
each axis (the weighted X pass, the Z pass with the norm), thin in the others, against the
float64 oracle; the whole solve at 64x96x128 and with 384-point rows against the run-time
engine; and the operator alone through the same passes on inputs of every symmetry.

Bounds: FP64 as in test_gpu_ilsqr, the larger of 1e-9 and 100 times the oracle's own change
under input noise of 1e-15 (single-precision Krylov steps: 2e-3, or 100 times under 6e-8)."""
import numpy as np
import pytest

import qsmgpu
from qsmgpu import Grid, inversion
from oracle import qsm_oracle as O
from test_gpu_ilsqr import OBLIQUE, _lsqr_operator, _oracle_lsqr_operator, check_all, og, phantom_case
from test_gpu_rts import rel

pytestmark = pytest.mark.gpu

THIN = [(64, 18, 20), (72, 17, 16), (160, 10, 12), (384, 6, 8), (12, 64, 14), (14, 12, 64), (10, 96, 128), (12, 14, 176),
        (66, 13, 15), (448, 6, 7), (16, 12, 400)]


def oracle_and_sensitivity(grid, f, mask, noise):
    ref = O.ilsqr(f, mask, og(grid), OBLIQUE, O.IlsqrParams())
    shaken = f * (1.0 + noise * np.random.default_rng(1).standard_normal(f.shape))
    return ref, max(rel(a, b) for a, b in zip(O.ilsqr(shaken, mask, og(grid), OBLIQUE, O.IlsqrParams()), ref))


@pytest.mark.parametrize("dims", THIN, ids=lambda d: "x".join(map(str, d)))
def test_against_the_oracle(ctx64, dims):
    grid = Grid.new(*dims, 1.0, 1.1, 0.9)
    f, mask = phantom_case(grid, OBLIQUE, seed=sum(dims))
    ref, sens = oracle_and_sensitivity(grid, f, mask, 1e-15)
    got = inversion.ilsqr(f, mask, grid, OBLIQUE, inversion.IlsqrParams(), ctx=ctx64)
    check_all(got, ref, max(1e-9, 100.0 * sens))


@pytest.mark.parametrize("dims", [(64, 18, 20), (160, 10, 12), (10, 96, 128)], ids=lambda d: "x".join(map(str, d)))
def test_single_precision_krylov(ctx32, dims):
    grid = Grid.new(*dims, 1.0, 1.1, 0.9)
    f, mask = phantom_case(grid, OBLIQUE, seed=sum(dims))
    ref, sens = oracle_and_sensitivity(grid, f, mask, 6e-8)
    ctx32.krylov_precision = "mixed"
    try:
        got = inversion.ilsqr(f, mask, grid, OBLIQUE, inversion.IlsqrParams(), ctx=ctx32)
    finally:
        ctx32.krylov_precision = "f64"
    check_all(got, ref, max(2e-3, 100.0 * sens))


@pytest.mark.parametrize("dims", [(64, 96, 128), (384, 24, 20), (176, 160, 64)], ids=lambda d: "x".join(map(str, d)))
def test_compiled_and_runtime_plans_agree(ctx64, dims):
    """The run-time engine's operator meets the oracle at small sizes; both are FP64 and differ
    by rounding only, amplified as in the oracle comparison (under 1e-9 there)."""
    grid = Grid.new(*dims, 1.0, 1.1, 0.9)
    f, mask = phantom_case(grid, OBLIQUE, seed=sum(dims))
    got = inversion.ilsqr(f, mask, grid, OBLIQUE, inversion.IlsqrParams(), ctx=ctx64)
    with qsmgpu.Context(0, "f64") as rt:
        rt.plan_mode = "runtime"
        want = inversion.ilsqr(f, mask, grid, OBLIQUE, inversion.IlsqrParams(), ctx=rt)
    check_all(got, want, 1e-9)


@pytest.mark.parametrize("dims", [(2, 2, 2), (9, 7, 5), (64, 6, 8), (6, 64, 7), (6, 8, 64), (384, 3, 4), (37, 12, 10)],
                         ids=lambda d: "x".join(map(str, d)))
def test_operator_runs_the_solvers_passes(ctx64, ctx32, dims):
    """Hermitian spectra, anti-Hermitian ones (whose image is imaginary: y = 0 up to rounding),
    one plane and the self-paired columns alone; 1e-12 and 2e-6 of the input's own image."""
    grid = Grid.new(*dims, 1.0, 1.2, 0.9)
    rng = np.random.default_rng(sum(dims))
    w = rng.uniform(0.0, 1.0, grid.shape)
    spec = np.fft.fftn(rng.standard_normal(grid.shape))
    plane = np.zeros_like(spec)
    plane[:, :, 0] = spec[:, :, 0] * (1.0 + 0.5j)
    nyq = np.zeros_like(spec)
    nyq[grid.nz // 2, grid.ny // 2, :] = spec[grid.nz // 2, grid.ny // 2, :] * (0.3 - 1.0j)
    for x in (spec, 1j * spec, plane, nyq):
        want = _oracle_lsqr_operator(grid, OBLIQUE, w, x)
        scale = np.linalg.norm(O.dipole_kernel(og(grid), OBLIQUE) * x)
        for ctx, tol in ((ctx64, 1e-12), (ctx32, 2e-6)):
            got = _lsqr_operator(ctx, grid, OBLIQUE, w, x)
            assert np.linalg.norm(got - want) <= tol * scale
        ctx64.set_profiling(True)
        try:
            ctx64.profile_reset()
            _lsqr_operator(ctx64, grid, OBLIQUE, w, x)
            kernels = ctx64.profile()
        finally:
            ctx64.set_profiling(False)
        # the solver's weighted X pass (one kernel at listed lengths) and never full rows
        assert "fft_x_c2c" not in kernels and ("fft_x_lsqr" in kernels) == (dims[0] in (64, 384))
