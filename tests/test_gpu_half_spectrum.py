"""Solvers whose inner arrangement depends on sizes: the iterative least squares on half
spectra (odd and even axes, whose self-conjugate planes differ), the TGV columns (masks that
touch the faces, thin structures outside the eroded mask, box sizes around a tile), and the
unrolled adjoint at checkpoint intervals that leave segments of every length."""
import numpy as np
import pytest
import torch

import qsmgpu
from qsmgpu import Grid, inversion
from oracle import qsm_oracle as O
from test_gpu_ilsqr import OBLIQUE, check_all, og, phantom_case
from test_gpu_rts import rel
from test_gpu_tgv import RAD_PER_PPM, phantom_phase
from test_gpu_tv_adjoint import case as adjoint_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(17, 16, 15), (16, 17, 18), (15, 16, 17), (19, 13, 11), (18, 14, 12)],
                         ids=lambda d: "x".join(map(str, d)))
def test_ilsqr_half_spectrum_parities(ctx64, dims):
    """Bound as in test_ilsqr_default_params_f64: max(1e-9, 100 x the oracle's sensitivity)."""
    grid = Grid.new(*dims, 1.0, 1.1, 0.9)
    f, mask = phantom_case(grid, OBLIQUE, seed=sum(dims))
    got = inversion.ilsqr(f, mask, grid, OBLIQUE, inversion.IlsqrParams(), ctx=ctx64)
    ref = O.ilsqr(f, mask, og(grid), OBLIQUE, O.IlsqrParams())
    noise = 1.0 + 1e-15 * np.random.default_rng(1).standard_normal(f.shape)
    ref2 = O.ilsqr(f * noise, mask, og(grid), OBLIQUE, O.IlsqrParams())
    sens = max(rel(a, b) for a, b in zip(ref2, ref))
    check_all(got, ref, max(1e-9, 100.0 * sens))


def tgv_masks(grid, seed):
    nz, ny, nx = grid.shape
    rng = np.random.default_rng(seed)
    full = np.ones(grid.shape, np.uint8)
    thin = np.zeros(grid.shape, np.uint8)
    thin[2:nz - 2, 2:ny - 2, 2:nx - 2] = 1
    thin[:, ny // 2, nx // 2] = 1          # a line through the faces, gone after one erosion
    thin[nz // 2, :, 1] = 1
    ragged = (rng.random(grid.shape) < 0.97).astype(np.uint8)
    return {"full": full, "thin": thin, "ragged": ragged}


@pytest.mark.parametrize("dims", [(31, 9, 8), (32, 8, 9), (33, 13, 12), (36, 12, 23), (12, 33, 19)],
                         ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("erosions", [0, 1])
def test_tgv_columns(ctx64, dims, erosions):
    """10 iterations against the float32 oracle at the 1e-4 of test_gpu_tgv."""
    grid = Grid.new(*dims, 1.0, 1.2, 0.9)
    phase, _ = phantom_phase(grid, OBLIQUE, sum(dims))
    for kind, m in tgv_masks(grid, 5).items():
        p = dict(iterations=10, erosions=erosions)
        if not O.erode_mask(m, erosions + 1).any():  # refused, as the reference does
            with pytest.raises(qsmgpu.QsmError):
                inversion.tgv_qsm(phase, m, grid, inversion.TgvParams(**p), OBLIQUE, ctx=ctx64)
            continue
        got = inversion.tgv_qsm(phase, m, grid, inversion.TgvParams(**p), OBLIQUE, ctx=ctx64)
        ref = O.tgv_qsm(phase, m, og(grid), O.TgvParams(**p), OBLIQUE)
        assert rel(got, ref) < 1e-4, (kind, rel(got, ref))


def test_adjoint_checkpoint_intervals(ctx64):
    """Every interval gives the gradients of the interval 1 (all states stored) to rounding:
    recomputed states are the stored ones bit for bit, so only sums' order could differ."""
    grid, f, mask, _ = adjoint_case((20, 18, 16), 4)
    g = torch.from_numpy(np.random.default_rng(0).standard_normal(grid.shape)).cuda()
    df, dm = torch.from_numpy(f).cuda(), torch.from_numpy(mask).cuda()
    torch.cuda.synchronize()

    def run(K, C, grad=True):
        chi, gf = torch.empty_like(df), torch.zeros_like(df)
        torch.cuda.synchronize()
        gl = inversion.tv_admm_unrolled_vjp_device(ctx64, df.data_ptr(), dm.data_ptr(), grid, (0, 0, 1), 2e-4, 2e-2, K, C,
                                                   g.data_ptr() if grad else 0, chi.data_ptr(),
                                                   gf.data_ptr() if grad else 0)
        return chi.cpu().numpy(), gf.cpu().numpy(), gl

    for K in (1, 2, 7, 12):
        want = run(K, 1)
        for C in (2, 3, 4, 6, 7, 11, 12, 30):
            got = run(K, C)
            np.testing.assert_array_equal(got[0], want[0])
            np.testing.assert_array_equal(run(K, C, grad=False)[0], want[0])
            assert rel(got[1], want[1]) < 1e-13 and abs(got[2] - want[2]) <= 1e-12 * abs(want[2]), (K, C)
