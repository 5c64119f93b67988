"""Measured calls of the qsmgpu API: what each stands for, its inputs, one pass, and its 64-bit value.

A case is a dict: `kind` (which entry point), grid sizes, `precision` of the context, and
the parameters that a call of that kind takes.  Volumes are made on the GPU from a seed:
ellipsoid susceptibility phantoms in an ellipsoid brain mask, their dipole field with
noise, point-dipole background fields and wrapped phase.  A program keeps one context per
precision and calls it for every volume, so contexts are shared by all cases.

Maps of a mixed context are single-precision results in double buffers; `run` hands them
on in single precision, as they are stored (NIfTI maps are float32).
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "qsm.rs_b200"))

import qsmgpu  # noqa: E402
from qsmgpu import Grid, bgremove, inversion, multi_echo, unwrap  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
RAD_PER_PPM = 2.0 * math.pi * 42.58 * 3.0 * 0.020  # 3 T, TE 20 ms
ECHO_TIMES = (0.004, 0.012, 0.020, 0.028)
BACKGROUND_RADII = [float(r) for r in range(12, 0, -1)]  # V-SHARP's default radii, mm


def listed():
    return [
        # closed-form inversion of a small volume: the shortest call, where launches and
        # latency count
        dict(name="tkd_64_f64", kind="tkd", nx=64, ny=64, nz=64, precision="f64"),
        # the whole-head chain at 1 mm: unwrapping, background removal, inversion
        dict(name="unwrap_256x256x176_mixed", kind="unwrap", nx=256, ny=256, nz=176, precision="mixed"),
        dict(name="vsharp_256x256x176_mixed", kind="vsharp", nx=256, ny=256, nz=176, precision="mixed"),
        dict(name="tv_256x256x176_mixed", kind="tv", nx=256, ny=256, nz=176, precision="mixed", iterations=250),
        # plain TV-ADMM in the reference's arithmetic on a small phantom
        dict(name="tv_64_f64", kind="tv", nx=64, ny=64, nz=64, precision="f64", iterations=250),
        # the pipeline's default inversion from host arrays, in the default context, on the
        # MNI-152 grid (218 = 2 * 109)
        dict(name="rts_182x218x182_f64", kind="rts", nx=182, ny=218, nz=182, precision="f64"),
        # conjugate gradients on an odd, ragged grid, from host arrays
        dict(name="resharp_189x231x165_f64", kind="resharp", nx=189, ny=231, nz=165, precision="f64"),
        # a study's volumes of uneven size in one call
        dict(name="tv_batch_8_mixed", kind="tv_batch", volumes=8, low=96, high=224, shapes=7, precision="mixed",
             iterations=50),
        # training through 50 unrolled iterations: the forward pass and its gradients (in
        # double: a gradient depends on which voxels lie above the shrinkage threshold)
        dict(name="tv_vjp_160x192x160_f64", kind="tv_vjp", nx=160, ny=192, nz=160, precision="f64", iterations=50),
        # a high-resolution matrix: field fit over four echoes and the iLSQR inversion
        dict(name="fit_384x384x256_4_echoes", kind="fit", nx=384, ny=384, nz=256, precision="f64"),
        dict(name="ilsqr_384x384x256_mixed", kind="ilsqr", nx=384, ny=384, nz=256, precision="mixed"),
        # single-step TGV from wrapped phase, default 1000 iterations
        dict(name="tgv_256x256x176", kind="tgv", nx=256, ny=256, nz=176, precision="mixed", iterations=1000),
    ]


# the largest volume (voxels) that is drawn for each kind
_LARGEST = dict(tkd=3.0e7, unwrap=3.0e7, vsharp=1.1e7, tv=6.0e6, rts=1.0e7, resharp=7.0e6, tv_batch=2.0e7,
                tv_vjp=4.0e6, fit=3.0e7, ilsqr=6.0e6, tgv=1.0e7)


def draw(rng):
    kind = rng.choice(sorted(_LARGEST))
    c = dict(kind=kind, precision=rng.choice(["f64", "mixed"]))
    if kind == "tv_batch":
        c.update(volumes=rng.randint(2, 8), low=rng.randint(64, 96), high=rng.randint(97, 200),
                 shapes=rng.randrange(1 << 20), iterations=rng.randint(10, 50))
        return c
    voxels = math.exp(rng.uniform(math.log(1.0e5), math.log(_LARGEST[kind])))
    ratios = [rng.uniform(0.75, 1.3) for _ in range(3)]
    edge = (voxels / (ratios[0] * ratios[1] * ratios[2])) ** (1.0 / 3.0)
    step = rng.choice([1, 2, 2, 8, 16])  # odd sizes, even ones, and scanners' matrix sizes
    for axis, r in zip(("nx", "ny", "nz"), ratios):
        c[axis] = min(384, max(36, int(round(edge * r / step)) * step))
    if kind == "tv_vjp":
        c["precision"] = "f64"
    if kind in ("tv", "tv_vjp"):
        c["iterations"] = rng.randint(10, 50)
    if kind == "tgv":
        c["iterations"] = rng.randint(100, 600)
    return c


def _shapes(case):
    """Grid sizes (nx, ny, nz) of a case's volumes."""
    if case["kind"] != "tv_batch":
        return [(case["nx"], case["ny"], case["nz"])]
    rng = random.Random(case["shapes"])
    return [tuple(rng.randint(case["low"], case["high"]) // s * s for s in (1, 2, 4)) for _ in range(case["volumes"])]


# ------------------------------------------------------------------------- inputs --
def _freq(n, d=1.0):
    return torch.fft.fftfreq(n, d, dtype=F64, device=DEV)


def _dipole(dims, bdir):
    nx, ny, nz = dims
    kx, ky, kz = _freq(nx)[None, None, :], _freq(ny)[None, :, None], _freq(nz)[:, None, None]
    b = np.asarray(bdir) / np.linalg.norm(bdir)
    k2 = kx * kx + ky * ky + kz * kz
    d = 1.0 / 3.0 - (kx * b[0] + ky * b[1] + kz * b[2]) ** 2 / torch.where(k2 > 0, k2, torch.ones_like(k2))
    return torch.where(k2 > 0, d, torch.zeros_like(d))


def _filter(x, m):
    return torch.fft.ifftn(torch.fft.fftn(x) * m).real


def _axes(dims):
    return [torch.arange(n, dtype=F64, device=DEV).reshape([-1 if a == 2 - i else 1 for a in range(3)])
            for i, n in enumerate(dims)]


class _Volume:
    """One seeded phantom: mask, susceptibility, field direction, fields and phase."""

    def __init__(self, dims, seed):
        rng = random.Random(seed)
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(rng.randrange(1 << 40))
        self.dims = dims
        self.shape = (dims[2], dims[1], dims[0])
        tilt, turn = math.radians(rng.uniform(0.0, 25.0)), rng.uniform(0.0, 2.0 * math.pi)
        self.bdir = (math.sin(tilt) * math.cos(turn), math.sin(tilt) * math.sin(turn), math.cos(tilt))
        self.xyz = _axes(dims)
        self.centre = [(n - 1) / 2.0 for n in dims]
        self.semi = [0.39 * dims[0], 0.46 * dims[1], 0.42 * dims[2]]
        inside = sum(((a - c) / s) ** 2 for a, c, s in zip(self.xyz, self.centre, self.semi))
        self.mask = (inside <= 1.0).to(torch.uint8).contiguous()
        chi = torch.zeros(self.shape, dtype=F64, device=DEV)
        for _ in range(12):
            c = [m + 0.6 * s * rng.uniform(-1.0, 1.0) for m, s in zip(self.centre, self.semi)]
            r = [max(2.0, rng.uniform(0.02, 0.08) * max(dims)) for _ in range(3)]
            chi = torch.where(sum(((a - q) / s) ** 2 for a, q, s in zip(self.xyz, c, r)) <= 1.0,
                              torch.full_like(chi, rng.uniform(-0.1, 0.2)), chi)
        self.chi = chi * self.mask
        self.rng = rng

    def noise(self, sigma):
        return sigma * torch.randn(self.shape, dtype=F64, device=DEV, generator=self.gen)

    def local_field(self):
        return _filter(self.chi, _dipole(self.dims, self.bdir)) + self.noise(0.01) * self.mask

    def total_field(self):
        """Local field plus four point dipoles outside the mask (ppm)."""
        f = self.local_field()
        for _ in range(4):
            ends = [self.rng.choice([-1.0, 1.0]) * self.rng.uniform(1.05, 1.25) for _ in range(3)]
            at = [c + e * s for c, e, s in zip(self.centre, ends, self.semi)]
            dx, dy, dz = (a - q for a, q in zip(self.xyz, at))
            r2 = dx * dx + dy * dy + dz * dz + 1.0
            strength = self.rng.uniform(2.0e3, 6.0e3) * (max(self.dims) / 256.0) ** 3
            f = f + strength * (3.0 * dz * dz / r2 - 1.0) / r2 ** 1.5
        return f

    def phase(self):
        p = RAD_PER_PPM * self.total_field()
        return torch.atan2(torch.sin(p), torch.cos(p)).contiguous()


def _inputs(case, seed):
    """The tensors of a case, and what describes them."""
    kind = case["kind"]
    vols = [_Volume(d, seed * 64 + i) for i, d in enumerate(_shapes(case))]
    out = []
    for v in vols:
        i = dict(grid=Grid.new(*v.dims), bdir=v.bdir, mask=v.mask)
        if kind in ("unwrap", "tgv"):
            i["field"] = v.phase()
        elif kind in ("vsharp", "resharp"):
            i["field"] = v.total_field().contiguous()
        elif kind == "fit":
            f = RAD_PER_PPM / 0.020 * v.local_field()
            i["phases"] = torch.stack([t * f + 0.3 + v.noise(0.02) for t in ECHO_TIMES])
            i["mags"] = torch.stack([(math.exp(-t / 0.030) * (0.2 + 0.8 * v.mask) + v.noise(0.01)).abs()
                                     for t in ECHO_TIMES])
        else:
            i["field"] = v.local_field().contiguous()
        if kind == "tv_vjp":  # of a squared error: part of the contrast is missing, and noise
            i["grad"] = (2.0 * (v.noise(0.01) - 0.2 * v.chi) * v.mask).contiguous()
        out.append(i)
    return out


# --------------------------------------------------------------------------- calls --
_contexts = {}


def _context(precision):
    if precision not in _contexts:
        _contexts[precision] = qsmgpu.Context(0, precision)
    return _contexts[precision]


def _tv_params(case):
    return inversion.TvParams(tol=0.0, max_iter=case["iterations"])


def prepare(case, seed):
    ctx = _context(case["precision"])
    kind = case["kind"]
    ins = _inputs(case, seed)
    s = dict(case=case, ctx=ctx, ins=ins, stream=torch.cuda.ExternalStream(ctx.stream_handle()))
    if kind in ("rts", "resharp"):
        for i in ins:
            i["field"], i["mask"] = i["field"].cpu().numpy(), i["mask"].cpu().numpy()
        return s
    n_out = dict(fit=3, ilsqr=4, tv_vjp=2).get(kind, 1)
    shape = ins[0]["mask"].shape
    s["out"] = [torch.empty(shape, dtype=F64, device=DEV) for _ in range(n_out)]
    if kind in ("vsharp", "fit"):
        s["mask_out"] = torch.empty(shape, dtype=torch.uint8, device=DEV)
    if kind == "tv_batch":
        s["out"] = [torch.empty(i["mask"].shape, dtype=F64, device=DEV) for i in ins]
    return s


def _maps(s, more=()):
    """The call's maps, in the precision that they were computed in."""
    outs = s["out"]
    if s["case"]["precision"] == "mixed":
        with torch.cuda.stream(s["stream"]):
            outs = [o.float() for o in outs]
    return list(outs) + list(more)


def run(state):
    case, ctx, i = state["case"], state["ctx"], state["ins"][0]
    kind, g, bdir = case["kind"], i["grid"], i["bdir"]
    if kind == "rts":
        return inversion.rts(i["field"], i["mask"], g, bdir, ctx=ctx)
    if kind == "resharp":
        return list(bgremove.resharp(i["field"], i["mask"], g, ctx=ctx))
    o = [t.data_ptr() for t in state["out"]]
    m = i["mask"].data_ptr()
    if kind == "fit":
        multi_echo.multi_echo_linear_fit_device(ctx, i["phases"].data_ptr(), i["mags"].data_ptr(), ECHO_TIMES,
                                                len(ECHO_TIMES), m, g.n_total(), multi_echo.LinearFitParams(), o[0],
                                                o[1], o[2], state["mask_out"].data_ptr())
        return list(state["out"]) + [state["mask_out"]]
    if kind == "tv_batch":
        inversion.tv_admm_batch_device(ctx, [(v["field"].data_ptr(), v["mask"].data_ptr(), p, v["grid"], v["bdir"])
                                             for v, p in zip(state["ins"], o)], _tv_params(case))
        return _maps(state)
    f = i["field"].data_ptr()
    if kind == "tkd":
        inversion.tkd_device(ctx, f, m, g, bdir, inversion.TkdParams(), o[0])
    elif kind == "unwrap":
        unwrap.laplacian_unwrap_device(ctx, f, m, g, o[0])
    elif kind == "vsharp":
        bgremove.vsharp_with_radii_device(ctx, f, m, g, BACKGROUND_RADII, 0.05, o[0], state["mask_out"].data_ptr())
        return _maps(state, [state["mask_out"]])
    elif kind == "tv":
        inversion.tv_admm_device(ctx, f, m, g, bdir, _tv_params(case), o[0])
    elif kind == "tv_vjp":
        p = inversion.TvParams()
        slope = inversion.tv_admm_unrolled_vjp_device(ctx, f, m, g, bdir, p.lambda_, p.rho, case["iterations"], 10,
                                                      i["grad"].data_ptr(), o[0], o[1])
        return _maps(state, [np.array([slope])])
    elif kind == "ilsqr":
        inversion.ilsqr_device(ctx, f, m, g, bdir, inversion.IlsqrParams(), *o)
    elif kind == "tgv":
        inversion.tgv_qsm_device(ctx, f, m, g, inversion.TgvParams(iterations=case["iterations"], tol=0.0), bdir, o[0])
        with torch.cuda.stream(state["stream"]):
            return state["out"][0].float()  # TGV always iterates in single precision
    return _maps(state)


def work(case):
    """Bytes of the inputs and outputs, and the arithmetic of the transforms and stencils."""
    kind = case["kind"]
    n = float(sum(a * b * c for a, b, c in _shapes(case)))
    fft = sum(2.5 * a * b * c * math.log2(a * b * c) for a, b, c in _shapes(case))  # one real 3D transform
    it = case.get("iterations", 0)
    flops = {
        "tkd": 2 * fft, "unwrap": 2 * fft + 40 * n, "vsharp": 17 * fft, "tv": (2 * it + 2) * fft + 50 * it * n,
        "tv_batch": (2 * it + 2) * fft + 50 * it * n, "tv_vjp": (4 * it + 4) * fft + 110 * it * n,
        "rts": 44 * fft + 1000 * n, "resharp": 128 * fft + 300 * n, "fit": 100 * n, "ilsqr": 410 * fft + 3000 * n,
        "tgv": 270.0 * it * n,
    }[kind]
    each = {"vsharp": 18, "resharp": 18, "fit": 16 * len(ECHO_TIMES) + 26, "tv_vjp": 33, "ilsqr": 41}.get(kind, 17)
    return {"bytes": each * n, "flops": flops}


# ----------------------------------------------------------------- values in 64 bits --
def _wrap(x):
    y = torch.fmod(x, 2.0 * math.pi)
    return torch.where(y > math.pi, y - 2.0 * math.pi, torch.where(y < -math.pi, y + 2.0 * math.pi, y))


def _grad(x):
    return [torch.roll(x, -1, d) - x for d in (2, 1, 0)]


def _bdiv(g):
    return sum(c - torch.roll(c, 1, d) for c, d in zip(g, (2, 1, 0)))


def _axis_sum(dims, f):
    return f(dims[0])[None, None, :] + f(dims[1])[None, :, None] + f(dims[2])[:, None, None]


def _laplacian(dims):
    """Eigenvalues of the negative 7-point Laplacian at 1 mm."""
    return _axis_sum(dims, lambda n: 2.0 - 2.0 * torch.cos(2.0 * math.pi * torch.arange(n, dtype=F64, device=DEV) / n))


def _sphere(dims, radius):
    """Spectrum of the normalised sphere kernel."""
    def sq(n):
        c = torch.arange(n, dtype=F64, device=DEV)
        return torch.where(c <= n // 2, c, c - n) ** 2
    inside = (_axis_sum(dims, sq) <= radius * radius).to(F64)
    return torch.fft.fftn(inside / inside.sum()).real


def _shrink(v, t):
    return torch.where(v > t, v - t, torch.where(v < -t, v + t, torch.zeros_like(v)))


def _admm(x0, mult, thr, iterations, tol, x_prev):
    """x_i = x0 - mult * bdiv(g), then the shrinkage step; stops once the change is below tol."""
    g = u = [torch.zeros_like(x0)] * 3
    for it in range(iterations):
        x = x0 - _filter(_bdiv(g), mult)
        if tol > 0.0 and float((x - x_prev).norm() / (x.norm() + 1e-20)) < tol:
            return x
        x_prev = x
        if it + 1 < iterations:
            v = [a + b for a, b in zip(_grad(x), u)]
            z = [_shrink(a, thr) for a in v]
            u, g = [a - b for a, b in zip(v, z)], [2.0 * b - a for a, b in zip(v, z)]
    return x


def _tv(field, dims, bdir, lam, rho, iterations):
    d = _dipole(dims, bdir)
    a = d * d + rho * _laplacian(dims)
    inv = torch.where(a.abs() > 1e-20, 1.0 / a, torch.zeros_like(a))
    return _admm(_filter(field, d * inv), rho * inv, lam / rho, iterations, 0.0, torch.zeros_like(field))


def _rts(field, mask, dims, bdir):
    delta, mu, rho = 0.15, 1e5, 10.0
    d = _dipole(dims, bdir)
    well = d.abs() > delta
    r = d / (d * d + 1e-6)
    c = r
    for _ in range(4):
        c = c + (1.0 - c * d) * r
    x1 = _filter(field, torch.where(well, c, torch.zeros_like(c))) * mask
    m = mu * well.to(F64)
    a = m + rho * _laplacian(dims)
    inv = torch.where(a.abs() > 1e-20, rho / a, torch.zeros_like(a))
    return _admm(_filter(x1, m / rho * inv), inv, 1.0 / rho, 20, 1e-2, x1) * mask


def _erode(mask, sphere):
    return (_filter(mask.to(F64), sphere) > 1.0 - math.sqrt(1e-7)).to(torch.uint8)


def _vsharp(field, mask, dims):
    local, final, first = torch.zeros_like(field), torch.zeros_like(mask), None
    for r in BACKGROUND_RADII:
        s = _sphere(dims, r)
        first = s if first is None else first
        new = (_erode(mask, s) == 1) & (final == 0)
        local = torch.where(new, _filter(field, 1.0 - s), local)
        final = torch.where(new, torch.ones_like(final), final)
    q = 1.0 - first
    inv = torch.where(q.abs() < 0.05, torch.zeros_like(q), 1.0 / q)
    return _filter(local, inv) * final, final


def _resharp(field, mask, dims):
    s = _sphere(dims, 6.0)
    eroded = _erode(mask, s)
    w, q = eroded.to(F64), 1.0 - s

    def hth(x):
        return _filter(w * _filter(x, q), q)
    b = hth(field)
    x, r, p = torch.zeros_like(b), b.clone(), b.clone()
    rs = float((r * r).sum())
    for _ in range(30):
        ap = hth(p) + 1e-4 * p
        pap = float((p * ap).sum())
        if abs(pap) < 1e-20:
            break
        x, r = x + rs / pap * p, r - rs / pap * ap
        new = float((r * r).sum())
        if math.sqrt(new) < 1e-6 * float(b.norm()):
            break
        p, rs = r + new / rs * p, new
    return torch.where(eroded == 1, x, torch.zeros_like(x)), eroded


def _fit(ph, mg, mask):
    sw = sum(mg)
    te = [float(t) for t in ECHO_TIMES]
    t_mean = sum(w * t for w, t in zip(mg, te)) / sw
    p_mean = sum(w * p for w, p in zip(mg, ph)) / sw
    sxx = sum(w * (t - t_mean) * (t - t_mean) for w, t in zip(mg, te))
    sxy = sum(w * (t - t_mean) * (p - p_mean) for w, t, p in zip(mg, te, ph))
    slope = sxy / sxx
    icpt = p_mean - slope * t_mean
    res = sum(w * (p - (icpt + slope * t)) ** 2 for w, t, p in zip(mg, te, ph)) / sw * len(te)
    ok = (mask != 0) & (sw >= 1e-10) & (sxx > 1e-10)
    slope, icpt, res = (torch.where(ok, v, torch.zeros_like(v)) for v in (slope, icpt, res))
    picked = res[(mask > 0) & (res > 0) & torch.isfinite(res)].sort().values
    limit = picked[min(int(90.0 / 100.0 * picked.numel()), picked.numel() - 1)]
    return [slope, icpt, res, ((mask > 0) & (res < limit)).to(torch.uint8)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ilsqr", "tgv"):
        return None  # truncated iterations with a fitted stencil or percentile weights
    ins = _inputs(case, seed)
    if kind == "tv_batch":
        return [_tv(i["field"], i["grid"].dims, i["bdir"], 2e-4, 2e-2, case["iterations"]) * i["mask"] for i in ins]
    i = ins[0]
    dims, mask, bdir = i["grid"].dims, i["mask"], i["bdir"]
    if kind == "fit":
        return _fit(list(i["phases"]), list(i["mags"]), mask)
    f = i["field"]
    if kind == "tkd":
        d = _dipole(dims, bdir)
        cut = torch.where(d >= 0, torch.full_like(d, 1.0 / 0.15), torch.full_like(d, -1.0 / 0.15))
        return [_filter(f, torch.where(d.abs() <= 0.15, cut, 1.0 / d)) * mask]
    if kind == "unwrap":
        lap = sum(_wrap(torch.roll(f, -1, a) - f) - _wrap(f - torch.roll(f, 1, a)) for a in (2, 1, 0)) * mask
        e = -_laplacian(dims)
        return [_filter(lap, torch.where(e.abs() > 1e-20, 1.0 / e, torch.zeros_like(e))) * mask]
    if kind == "vsharp":
        return list(_vsharp(f, mask, dims))
    if kind == "resharp":
        return list(_resharp(f, mask, dims))
    if kind == "rts":
        return _rts(f, mask, dims, bdir)
    if kind == "tv":
        return [_tv(f, dims, bdir, 2e-4, 2e-2, case["iterations"]) * mask]
    lam = torch.tensor(2e-4, dtype=F64, device=DEV, requires_grad=True)
    field = f.clone().requires_grad_(True)
    chi = _tv(field, dims, bdir, lam, 2e-2, case["iterations"]) * mask
    grads = torch.autograd.grad(chi, [field, lam], i["grad"])
    return [chi.detach(), grads[0], grads[1].reshape(1)]
