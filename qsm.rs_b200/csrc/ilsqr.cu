// iLSQR dipole inversion (src/inversion/ilsqr.rs:1307-1351) -> (chi, xsa, xfs, xlsqr).
//
// Step 1, lsqr_step (ilsqr.rs:953-1030).  Laplacian weights w (mask-adaptive stencil,
//   thresholds at the 60th / 99.9th percentile by exact selection), b = D*FFT(w*f), then
//   complex LSQR (ilsqr.rs:177-321, relative-residual stop) on k-space vectors with
//   A = A^H = D*FFT(w*Re IFFT(D*x)).  D is not symmetric under k -> -k on even-length
//   Nyquist planes, so the reference iterates on the whole complex vector; but b and every
//   output of A are D times the spectrum of a real image, and so is every vector of the
//   iteration.  The solver therefore holds h = m G on the half spectrum, where D G is the
//   reference's vector and m(k) = sqrt((D(k)^2 + D(-k)^2)/2).  D G -> m G keeps norms
//   (summing |h|^2 with c = 2, or 1 on the self-paired columns), and with it
//     A: h -> m FFT(w IFFT(m h)),
//   so this is the same iteration on half the values.  One application is five passes,
//     Z inv (pre: *s*m) -> Y inv -> X [c2r, w/N, r2c] -> Y fwd -> Z fwd (post: *m - c*old)
//   where s is the deferred 1/beta or 1/alpha of the input vector and the Z fwd pass
//   also accumulates the FP64 norm of its output.  The block that finishes that pass
//   last completes the norm and runs the scalar recurrence on the device, so one LSQR
//   iteration (two applications and the x/w update) is 11 launches without a host
//   synchronisation, replayed as a CUDA graph.  (On full spectra an application took 1.85 ms
//   in FP64 at 384x384x256, and on half spectra 1.04 ms.)
// Step 2, fastqsm_step (ilsqr.rs:1037-1167).  F = FFT(f); k-space weights |D|^0.001
//   normalised by the 1st/30th percentiles of all values; the SMV (r = 3) kernel
//   spectrum; the Eq. 9/11 filters and the TKD (t0 = 1/8, sign(+0) = +1) are real k-space
//   factors followed by the real part, hence half-spectrum chains with the symmetrised
//   factor; and the 2x2 least-squares fit over all voxels (FP64 sums).
// Step 3, susceptibility_artifacts_step (ilsqr.rs:1174-1289).  Gradient weights from
//   the mask-adaptive gradient of xfs (percentiles 50 / 70 per component); LSMR
//   (ilsqr.rs:344-517) on real vectors.  Its k-space mask mic = |D| < 0.1 acts through
//   Re IFFT(FFT(x)*mic), which equals a half-spectrum transform with the multiplier
//   (mic(k) + mic(-k))/2; periodic gradient / divergence stencils carry the weights,
//   the axpy terms and the FP64 norms.
// Step 4: chi = mask * (xlsqr - xsa).
#include "functors.cuh"
#include "select.h"
#include "smv.h"
#include "solvers.h"

#include <algorithm>
#include <cmath>

namespace qsm {

namespace {

// ===================================================================== setup ==
// Mask-adaptive second difference along one axis at linear index l (coordinate c of
// n, stride s), src/inversion/ilsqr.rs:583-669.  The stencil selector is
// 2*m[l+s] + m[l-s] in u8 arithmetic inside, forward (2) at c = 0 and backward (1) at
// c = n-1.
__device__ double lap1(const double* __restrict__ f, const uint8_t* __restrict__ m, long long l, int c, int n,
                       long long s) {
  int sel;
  if (c >= 1 && c <= n - 2) sel = (uint8_t)(2u * m[l + s] + m[l - s]);
  else sel = (c == 0) ? 2 : (c == n - 1 ? 1 : 0);
  if (sel == 3) return f[l - s] - 2.0 * f[l] + f[l + s];
  if (sel == 2) {
    if (c + 3 < n && m[l + 2 * s] != 0 && m[l + 3 * s] != 0)
      return 2.0 * f[l] - 5.0 * f[l + s] + 4.0 * f[l + 2 * s] - f[l + 3 * s];
    if (c + 2 < n && m[l + 2 * s] != 0) return f[l] - 2.0 * f[l + s] + f[l + 2 * s];
    return f[l + s] - f[l];
  }
  if (sel == 1) {
    if (c >= 3 && m[l - 3 * s] != 0 && m[l - 2 * s] != 0)
      return -f[l - 3 * s] + 4.0 * f[l - 2 * s] - 5.0 * f[l - s] + 2.0 * f[l];
    if (c >= 2 && m[l - 2 * s] != 0) return f[l - 2 * s] - 2.0 * f[l - s] + f[l];
    return f[l - s] - f[l];
  }
  return 0.0;
}

// compute_laplacian, src/inversion/ilsqr.rs:528-566 (0 outside the mask)
__global__ void k_ilsqr_lap(const double* __restrict__ f, const uint8_t* __restrict__ m, int nx, int ny, int nz,
                            double hx, double hy, double hz, double* __restrict__ lap) {
  const long long N = (long long)nx * ny * nz, sxy = (long long)nx * ny;
  for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < N; l += (long long)gridDim.x * blockDim.x) {
    double v = 0.0;
    if (m[l] != 0) {
      const int i = (int)(l % nx);
      const int j = (int)((l / nx) % ny);
      const int k = (int)(l / sxy);
      v += hx * lap1(f, m, l, i, nx, 1);
      v += hy * lap1(f, m, l, j, ny, nx);
      v += hz * lap1(f, m, l, k, nz, sxy);
    }
    lap[l] = v;
  }
}

// Percentile weight of one value (src/inversion/ilsqr.rs:703-716, 882-897): 1 below
// tmin, 0 above tmax, linear in between when the range exceeds 1e-10.
__device__ __forceinline__ double pct_weight(double v, double tmin, double tmax) {
  const double range = tmax - tmin;
  if (v < tmin) return 1.0;
  if (v > tmax) return 0.0;
  if (range > 1e-10) return (tmax - v) / range;
  return 0.0;
}

template <typename T>
__global__ void k_lap_weights(long long N, const double* __restrict__ lap, const uint8_t* __restrict__ m,
                              double tmin, double tmax, T* __restrict__ w) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x)
    w[i] = m[i] != 0 ? (T)pct_weight(lap[i], tmin, tmax) : T(0);
}

// fgrad_masked, src/inversion/ilsqr.rs:767-823: forward difference when the forward
// neighbour is inside the axis and the mask, else backward, else 0; 0 outside the mask.
template <typename T>
__global__ void k_fgrad_masked(const T* __restrict__ f, const uint8_t* __restrict__ m, int nx, int ny, int nz,
                               double hx, double hy, double hz, double* __restrict__ g) {
  const long long N = (long long)nx * ny * nz, sxy = (long long)nx * ny;
  for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < N; l += (long long)gridDim.x * blockDim.x) {
    double gx = 0.0, gy = 0.0, gz = 0.0;
    if (m[l] != 0) {
      const int i = (int)(l % nx);
      const int j = (int)((l / nx) % ny);
      const int k = (int)(l / sxy);
      const double fl = (double)f[l];
      if (i < nx - 1 && m[l + 1] != 0) gx = hx * ((double)f[l + 1] - fl);
      else if (i > 0 && m[l - 1] != 0) gx = hx * (fl - (double)f[l - 1]);
      if (j < ny - 1 && m[l + nx] != 0) gy = hy * ((double)f[l + nx] - fl);
      else if (j > 0 && m[l - nx] != 0) gy = hy * (fl - (double)f[l - nx]);
      if (k < nz - 1 && m[l + sxy] != 0) gz = hz * ((double)f[l + sxy] - fl);
      else if (k > 0 && m[l - sxy] != 0) gz = hz * (fl - (double)f[l - sxy]);
    }
    g[l] = gx;
    g[N + l] = gy;
    g[2 * N + l] = gz;
  }
}

// gradient_weights_component, src/inversion/ilsqr.rs:854-900 (times mask[i] as f64)
template <typename T>
__global__ void k_grad_weights(long long N, const double* __restrict__ g, const uint8_t* __restrict__ m, double tx0,
                               double tx1, double ty0, double ty1, double tz0, double tz1, T* __restrict__ w) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const uint8_t mi = m[i];
    if (mi == 0) {
      w[i] = T(0);
      w[N + i] = T(0);
      w[2 * N + i] = T(0);
      continue;
    }
    const double mv = (double)mi;
    w[i] = (T)(pct_weight(g[i], tx0, tx1) * mv);
    w[N + i] = (T)(pct_weight(g[N + i], ty0, ty1) * mv);
    w[2 * N + i] = (T)(pct_weight(g[2 * N + i], tz0, tz1) * mv);
  }
}

// |D(k)|^n_exp over the full spectrum in natural order (src/inversion/ilsqr.rs:735-737)
__global__ void k_dipole_pow(KSpace K, int nx, int ny, int nz, double n_exp, double* __restrict__ out) {
  const long long N = (long long)nx * ny * nz;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(i % nx);
    const int iy = (int)((i / nx) % ny);
    const int iz = (int)(i / ((long long)nx * ny));
    const double d = K.dipole(__ldg(K.fx + ix), __ldg(K.fy + iy), __ldg(K.fz + iz));
    out[i] = pow(fabs(d), n_exp);
  }
}

// ====================================================================== LSQR ==
struct LsqrState {
  int done;   // every later kernel returns at once
  int stop;   // convergence seen by the rotation; committed after the x/w update
  int iters;  // completed iterations
  unsigned counter;
  double alpha, beta;
  double su, sv;  // deferred scales of u and v: 1/beta and 1/alpha (1 when zero)
  double rho_bar, phi_bar, bnorm, t1, t2, tol;
};

// The scalar recurrence after the norm of an application's output (modes as OpLsqrHalf).
__device__ inline void lsqr_last(LsqrState* st, int mode, double total) {
  const double nrm = sqrt(total);
  if (mode == 0 || mode == 2) {
    st->beta = nrm;
    st->su = nrm > 0.0 ? 1.0 / nrm : 1.0;
    if (mode == 2) {
      st->bnorm = nrm;
      st->phi_bar = nrm;
    }
    return;
  }
  st->alpha = nrm;
  st->sv = nrm > 0.0 ? 1.0 / nrm : 1.0;
  if (mode == 3) {
    st->rho_bar = nrm;
    if (nrm * st->beta == 0.0) st->done = 1;
    return;
  }
  // Givens rotation and step lengths, src/inversion/ilsqr.rs:261-290
  const double alpha = nrm, beta = st->beta;
  const double rho = sqrt(st->rho_bar * st->rho_bar + beta * beta);
  const double c = st->rho_bar / rho;
  const double s = beta / rho;
  const double theta = s * alpha;
  st->rho_bar = -c * alpha;
  const double phi = c * st->phi_bar;
  st->phi_bar *= s;
  st->t1 = phi / rho;
  st->t2 = -theta / rho;
  st->iters += 1;
  if (st->phi_bar / (st->bnorm + 1e-20) <= st->tol) st->stop = 1;
}

__device__ __forceinline__ double dip(const KSpace& K, int ix, int iy, int iz) {
  return K.dipole(__ldg(K.fx + ix), __ldg(K.fy + iy), __ldg(K.fz + iz));
}

// v * s * m: the input of A, s its deferred scale
template <typename T> struct OpScaleM {
  using C = cplx_t<T>;
  const T* m;
  const double* s;
  static constexpr bool kNoPost = true;
  __device__ __forceinline__ C pre(C v, int, int, int, long long idx) const {
    return cscale(cscale(v, (T)__ldg(s)), __ldg(m + idx));
  }
  __device__ __forceinline__ C post(C v, int, int, int, long long) const { return v; }
};

// Z forward epilogue of an application of A.  mode 0: u = A v - alpha*u (then beta);
// 1: v = A u - beta*v (then alpha and the rotation); 2: b (then beta = ||b||);
// 3: v = A^H u (then alpha; alpha*beta = 0 ends the solve with x = 0).
template <typename T> struct OpLsqrHalf {
  using C = cplx_t<T>;
  const T* m;
  int nx;
  const C* old;
  LsqrState* st;
  int mode;
  // the compile-time pass stages `old` through shared memory (k_pass_yz_dx_old)
  static constexpr bool kReadsOld = true;
  static constexpr bool kNoPre = true;
  struct Scalars {
    double coef, sc;
  };
  __device__ __forceinline__ C pre(C v, int, int, int, long long) const { return v; }
  __device__ __forceinline__ const C* old_src() const { return mode <= 1 ? old : nullptr; }
  __device__ __forceinline__ Scalars scalars() const {
    if (mode > 1) return Scalars{0.0, 0.0};
    return Scalars{mode == 0 ? -st->alpha : -st->beta, mode == 0 ? st->su : st->sv};
  }
  __device__ __forceinline__ C post_old(C v, int ix, int, int, long long idx, C oldv, const Scalars& s,
                                        double& acc) const {
    C r = cscale(v, __ldg(m + idx));
    if (mode <= 1) r = cadd(r, cscale(cscale(oldv, (T)s.sc), (T)s.coef));
    const double c = (ix == 0 || 2 * ix == nx) ? 1.0 : 2.0;
    acc += c * ((double)r.x * (double)r.x + (double)r.y * (double)r.y);
    return r;
  }
  __device__ __forceinline__ C post(C v, int ix, int iy, int iz, long long idx, double& acc) const {
    return post_old(v, ix, iy, iz, idx, mode <= 1 ? old[idx] : v, scalars(), acc);
  }
  __device__ void last(double total) const { lsqr_last(st, mode, total); }
};

// m = sqrt(sym(D^2)), and sym(D) / m (0 where m is), which takes h to the reference's
// spectrum under the real part
template <typename T> struct OpHalfD {
  using C = cplx_t<T>;
  KSpace K;
  int ratio;
  __device__ __forceinline__ C mid(C v, int ix, int iy, int iz, long long) const {
    const KSpace& k = K;
    const double m = sqrt(K.sym(ix, iy, iz, [&](double kx, double ky, double kz, int, int, int) {
      const double d = k.dipole(kx, ky, kz);
      return d * d;
    }));
    if (!ratio) return cscale(v, (T)m);
    const double d = K.sym(ix, iy, iz, [&](double kx, double ky, double kz, int, int, int) { return k.dipole(kx, ky, kz); });
    return cscale(v, (T)(m > 0.0 ? d / m : 0.0));
  }
};

// X pass of an application of A: half spectrum -> real rows -> * w / N -> half spectrum, in
// place (FP a FixedPlan).  Two rows are one complex pencil; the inverse transform's last
// stage weights its values in registers and hands them to the forward transform (the
// reversed plan), whose results are split into the two half spectra.
template <typename T, class FP>
__global__ void k_x_weight_fx(Geom g, const cplx_t<T>* __restrict__ twg, cplx_t<T>* __restrict__ spec,
                              const T* __restrict__ w, T invn, const int* __restrict__ done) {
  using C = cplx_t<T>;
  constexpr int N = FP::n, TT = FP::T, NXH = N / 2 + 1;
  if (done != nullptr && *done) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr bool TWP = x_tw_padded<T>();
  C* tw = reinterpret_cast<C*>(smraw);
  C* sm = tw + x_tw_len<T>(N);
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  for (int i = tid; i < N; i += blockDim.x * blockDim.y) tw[TWP ? tw_pad(i) : i] = twg[i];
  const int t = threadIdx.x;
  const int nrows = g.nrows();
  const int a = 2 * (blockIdx.x * blockDim.y + threadIdx.y), b = a + 1;
  const bool active = a < nrows && t < TT;
  const bool hasb = b < nrows;
  C* sp = sm + threadIdx.y * x_rowlen<T>(N);
  SAPadded<x_pad<T, FP>()> sa;
  C* ra = spec + (long long)a * g.pitch;
  C* rb = spec + (long long)b * g.pitch;
  auto fetch = [&](int e) -> C {
    const bool lo = e <= N / 2;
    const int k = lo ? e : N - e;
    C xa = ra[k];
    C xb = hasb ? rb[k] : mk<C>(T(0), T(0));
    if (k == 0 || 2 * k == N) {
      xa.y = T(0);
      xb.y = T(0);
    }
    return lo ? mk<C>(xa.x - xb.y, xa.y + xb.x) : mk<C>(xa.x + xb.y, xb.x - xa.y);
  };
  const T* wa = w + (long long)a * N;
  auto hook = [&](int e, C x) -> C {
    return mk<C>(__ldg(wa + e) * (x.x * invn), hasb ? __ldg(wa + N + e) * (x.y * invn) : T(0));
  };
  auto emit = [&](int e, C v) { sp[sa(e)] = v; };
  C v[kFftEmax];
  EmitInRegs<decltype(hook)> keep{hook};
  FetchInRegs in_regs;
  FP::template run_v<+1, TWP>(v, t, active, sp, sa, tw, fetch, keep);
  ReversePlan<FP>::type::template run_v<-1, TWP>(v, t, active, sp, sa, tw, in_regs, emit);
  if (active) {
    const T half = T(0.5);
#pragma unroll
    for (int c = 0; c < (NXH + TT - 1) / TT; ++c) {
      const int k = t + c * TT;
      if (k < NXH) {
        const C zk = sp[sa(k)];
        const C zn = sp[sa(k == 0 ? 0 : N - k)];
        ra[k] = mk<C>((zk.x + zn.x) * half, (zk.y - zn.y) * half);
        if (hasb) rb[k] = mk<C>((zk.y + zn.y) * half, (zn.x - zk.x) * half);
      }
    }
  }
}

// The same over any length; `img` is a real volume for lengths without the compile-time
// kernel.
template <typename T>
void run_x_weight(qsm_ctx* ctx, const Fft3<T>& f, cplx_t<T>* spec, const T* w, T invn, T* img, const int* done) {
  if (compiled_plans(ctx)) {
#define QSM_TRY_XW(N_, T_, R0_, R1_, R2_)                                                                        \
    if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(f.px)) {                                                       \
      using FP = FixedPlan<N_, T_, R0_, R1_, R2_>;                                                               \
      const int P = x_fx_pencils<FP>(ctx, ((long long)f.g.nrows() + 1) / 2);                                     \
      const size_t smem = (size_t)(x_tw_len<T>(N_) + P * x_rowlen<T>(N_)) * sizeof(cplx_t<T>);                   \
      auto kern = k_x_weight_fx<T, FP>;                                                                          \
      ensure_smem(kern, smem);                                                                                   \
      LaunchScope ls(ctx, "fft_x_lsqr");                                                                         \
      kern<<<x_fx_blocks(((long long)f.g.nrows() + 1) / 2, P), dim3(T_, P), smem, ctx->stream>>>(                  \
          f.g, f.twx, spec, w, invn, done);                                                                      \
      ls.done();                                                                                                 \
      return;                                                                                                    \
    }
    QSM_FIXED_PLANS(QSM_TRY_XW)
    QSM_FIXED_PLANS_WIDE(QSM_TRY_XW)
#undef QSM_TRY_XW
  }
  run_x_c2r<T>(ctx, f, spec, StoreReal<T>{img, f.g.nx, invn}, done);
  run_x_r2c<T>(ctx, f, spec, LoadProduct<T, T>{img, w, f.g.nx}, done);
}

// What an application of A works with.
template <typename T> struct LsqrOperator {
  const Fft3<T>* f;
  const T* m;  // OpHalfD
  const T* w;
  T invn;
  cplx_t<T>* t;  // a half spectrum
  T* img;        // a real volume
  LsqrState* st;
  double* partials;
  unsigned* counter;
};
// dst = A(s x) with the epilogue of `mode` (OpLsqrHalf): h -> m FFT(w IFFT(m h)) on half spectra.
template <typename T>
void lsqr_apply(qsm_ctx* ctx, const LsqrOperator<T>& a, const cplx_t<T>* x, const double* s, cplx_t<T>* dst,
                const cplx_t<T>* old, int mode) {
  const Fft3<T>& f = *a.f;
  const int* done = &a.st->done;
  run_yz<T, +1, 2, true>(ctx, f, x, a.t, OpScaleM<T>{a.m, s}, done);
  run_yz<T, +1, 1>(ctx, f, a.t, a.t, OpId<T>{}, done);
  run_x_weight<T>(ctx, f, a.t, a.w, a.invn, a.img, done);
  run_yz<T, -1, 1>(ctx, f, a.t, a.t, OpId<T>{}, done);
  run_yz_acc<T, -1, 2, true>(ctx, f, a.t, dst, OpLsqrHalf<T>{a.m, f.g.nx, old, a.st, mode}, a.partials, a.counter, done,
                             "fft_z_lsqr");
}

template <typename T>
__global__ void k_lsqr_init_w(long long n, const cplx_t<T>* __restrict__ v, cplx_t<T>* __restrict__ w,
                              const LsqrState* st) {
  if (st->done) return;
  const T sv = (T)st->sv;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    w[i] = cscale(v[i], sv);
}

// x += t1*w; w = v + t2*w (src/inversion/ilsqr.rs:285-290); the last block commits a
// convergence stop.
template <typename T>
__global__ void k_lsqr_update(long long n, cplx_t<T>* __restrict__ x, cplx_t<T>* __restrict__ w,
                              const cplx_t<T>* __restrict__ v, LsqrState* st, double* partials) {
  if (st->done) return;
  const T t1 = (T)st->t1, t2 = (T)st->t2, sv = (T)st->sv;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const cplx_t<T> wi = w[i];
    x[i] = cadd(x[i], cscale(wi, t1));
    w[i] = cadd(cscale(v[i], sv), cscale(wi, t2));
  }
  double z[1] = {0.0};
  if (grid_sum_last<1>(z, partials, &st->counter) && threadIdx.x == 0 && st->stop) st->done = 1;
}

// ============================================================ FastQSM ops ==
// Eq. 9/11 filter wfs + h*(1 - wfs) with wfs = clamp((|D|^n - lo)/(hi - lo)),
// src/inversion/ilsqr.rs:739-757, 1080-1088; with sign: times sign(D) (ilsqr.rs:1057-1060)
template <typename T> struct OpFsFilter {
  using C = cplx_t<T>;
  KSpace K;
  const T* h;  // SMV kernel spectrum (even, real)
  double n_exp, lo, range;
  int with_sign;
  __device__ __forceinline__ C mid(C v, int ix, int iy, int iz, long long idx) const {
    const double hh = (double)__ldg(h + idx), ne = n_exp, l = lo, rg = range;
    const int sgn = with_sign;
    const KSpace& k = K;
    const double m = K.sym(ix, iy, iz, [&](double kx, double ky, double kz, int, int, int) {
      const double d = k.dipole(kx, ky, kz);
      double w = pow(fabs(d), ne);
      if (rg > 1e-20) w = (w - l) / rg;
      w = fmin(fmax(w, 0.0), 1.0);
      const double r = w + hh * (1.0 - w);
      return sgn ? (d > 0.0 ? r : (d < 0.0 ? -r : 0.0)) : r;
    });
    return cscale(v, (T)m);
  }
};
// inv_d = signum(D)/t0 where |D| < t0, else 1/D (ilsqr.rs:1118-1126)
template <typename T> struct OpTkdInv {
  using C = cplx_t<T>;
  KSpace K;
  double t0;
  __device__ __forceinline__ C mid(C v, int ix, int iy, int iz, long long) const {
    const double t = t0;
    const KSpace& k = K;
    const double m = K.sym(ix, iy, iz, [&](double kx, double ky, double kz, int, int, int) {
      const double d = k.dipole(kx, ky, kz);
      return fabs(d) < t ? copysign(1.0, d) / t : 1.0 / d;
    });
    return cscale(v, (T)m);
  }
};

// sums of xfs, xtkd, xfs^2, xfs*xtkd over all voxels (ilsqr.rs:1141-1146)
template <typename T>
__global__ void k_fs_sums(long long N, const T* __restrict__ a, const T* __restrict__ b, double* partials,
                          unsigned* counter, double* out) {
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const double x = (double)a[i], y = (double)b[i];
    s[0] += x;
    s[1] += y;
    s[2] += x * x;
    s[3] += x * y;
  }
  if (grid_sum_last<4>(s, partials, counter) && threadIdx.x == 0)
    for (int k = 0; k < 4; ++k) out[k] = s[k];
}

template <typename T>
__global__ void k_fs_final(long long N, const T* __restrict__ xfs, const uint8_t* __restrict__ m, double a, double b,
                           T* __restrict__ out, double* __restrict__ out64) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const double v = m[i] != 0 ? a * (double)xfs[i] + b : 0.0;
    out[i] = (T)v;
    if (out64) out64[i] = v;
  }
}

// ====================================================================== LSMR ==
struct LsmrState {
  int done;
  int iters;
  unsigned counter;
  int pad;
  double alpha, beta, su, sv;
  double alpha_bar, zeta_bar, rho, rho_bar, c_bar, s_bar, zeta;
  double normb, betadd, betad, rhodold, tautildeold, thetatilde;
  double norm_a2, maxrbar, minrbar;
  double atol, btol;
  double c_hbar, c_x, c_h;  // update coefficients of this iteration
  double normr, norm_a, cond_a, norm_ar;
};

// mic(k) = |D(k)| < 0.1 symmetrised over k -> -k (ilsqr.rs:1192-1194)
template <typename T> struct OpMic {
  using C = cplx_t<T>;
  KSpace K;
  __device__ __forceinline__ C mid(C v, int ix, int iy, int iz, long long) const {
    const double m = K.sym(ix, iy, iz, [&](double kx, double ky, double kz, int, int, int) {
      return fabs(K.dipole(kx, ky, kz)) < 0.1 ? 1.0 : 0.0;
    });
    return cscale(v, (T)m);
  }
};

template <typename T> struct LoadScaled {  // x * s (s = deferred scale in the state)
  const T* p;
  const double* s;
  int nx;
  __device__ __forceinline__ T operator()(int row, int e) const { return p[(long long)row * nx + e] * (T)*s; }
};
// v = Re IFFT(...)/N - beta*v (ilsqr.rs:1260-1276 then :425-427), with ||v||^2; the
// last block runs the LSMR recurrences (ilsqr.rs:433-492).  init: v = A^T u only.
template <typename T> struct StoreLsmrV {
  T* v;
  int nx;
  T invn;
  LsmrState* st;
  double* partials;
  int init;
  double acc;
  __device__ __forceinline__ void operator()(int row, int e, T val) {
    const long long i = (long long)row * nx + e;
    T r = val * invn;
    if (!init) r = r + (T)(-st->beta) * (v[i] * (T)st->sv);
    v[i] = r;
    acc += (double)r * (double)r;
  }
  __device__ void finish() {
    double a[1] = {acc};
    if (!grid_sum_last<1>(a, partials, &st->counter)) return;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    if (tid != 0) return;
    const double alpha = sqrt(a[0]);
    st->alpha = alpha;
    st->sv = alpha > 0.0 ? 1.0 / alpha : 1.0;
    if (init) {
      st->alpha_bar = alpha;
      st->zeta_bar = alpha * st->beta;
      st->norm_a2 = alpha * alpha;
      if (alpha * st->beta == 0.0) st->done = 1;
      return;
    }
    const double beta = st->beta;
    const double rho_old = st->rho;
    const double rho = sqrt(st->alpha_bar * st->alpha_bar + beta * beta);
    const double c = st->alpha_bar / rho;
    const double s = beta / rho;
    const double theta_new = s * alpha;
    st->alpha_bar = c * alpha;
    const double rho_bar_old = st->rho_bar;
    const double zeta_old = st->zeta;
    const double theta_bar = st->s_bar * rho;
    const double rho_temp = st->c_bar * rho;
    const double rho_bar = sqrt(rho_temp * rho_temp + theta_new * theta_new);
    st->c_bar = rho_temp / rho_bar;
    st->s_bar = theta_new / rho_bar;
    const double zeta = st->c_bar * st->zeta_bar;
    st->zeta_bar *= -st->s_bar;
    st->c_hbar = theta_bar * rho / (rho_old * rho_bar_old);
    st->c_x = zeta / (rho * rho_bar);
    st->c_h = theta_new / rho;
    st->rho = rho;
    st->rho_bar = rho_bar;
    st->zeta = zeta;
    // ||r|| estimate (undamped), ilsqr.rs:452-471
    const double betaacute = st->betadd;
    const double betahat = c * betaacute;
    st->betadd = -s * betaacute;
    const double thetatildeold = st->thetatilde;
    const double rhotildeold = sqrt(st->rhodold * st->rhodold + theta_bar * theta_bar);
    const double ctildeold = st->rhodold / rhotildeold;
    const double stildeold = theta_bar / rhotildeold;
    st->thetatilde = stildeold * rho_bar;
    st->rhodold = ctildeold * rho_bar;
    st->betad = -stildeold * st->betad + ctildeold * betahat;
    st->tautildeold = (zeta_old - thetatildeold * st->tautildeold) / rhotildeold;
    const double taud = (zeta - st->thetatilde * st->tautildeold) / st->rhodold;
    const double bd = st->betad - taud;
    st->normr = sqrt(0.0 + bd * bd + st->betadd * st->betadd);
    // ||A|| and cond(A), ilsqr.rs:474-484
    st->norm_a2 += beta * beta;
    st->norm_a = sqrt(st->norm_a2);
    st->norm_a2 += alpha * alpha;
    st->maxrbar = fmax(st->maxrbar, rho_bar_old);
    if (st->iters > 0) st->minrbar = fmin(st->minrbar, rho_bar_old);
    st->cond_a = fmax(st->maxrbar, rho_temp) / fmin(st->minrbar, rho_temp);
    st->norm_ar = fabs(st->zeta_bar);
  }
};

// u = w * fgrad(x) - alpha*u (ilsqr.rs:1226-1238, then :420-421), periodic forward
// differences; accumulates ||u||^2.  init: u = w * fgrad(x0) = b (no subtraction).
template <typename Tin, typename T>
__global__ void k_lsmr_grad(int nx, int ny, int nz, T hx, T hy, T hz, const Tin* __restrict__ x,
                            const T* __restrict__ w, T* __restrict__ u, LsmrState* st, double* partials, int init) {
  if (st->done) return;
  const long long N = (long long)nx * ny * nz, sxy = (long long)nx * ny;
  const T coef = init ? T(0) : (T)(-st->alpha);
  const T su = (T)st->su;
  double acc[1] = {0.0};
  for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < N; l += (long long)gridDim.x * blockDim.x) {
    const unsigned r = (unsigned)l / (unsigned)nx;  // N < 2^32 (checked by the host)
    const int i = (int)((unsigned)l - r * (unsigned)nx);
    const int j = (int)(r % (unsigned)ny);
    const int k = (int)(r / (unsigned)ny);
    const long long lx = i + 1 < nx ? l + 1 : l + 1 - nx;
    const long long ly = j + 1 < ny ? l + nx : l + nx - sxy;
    const long long lz = k + 1 < nz ? l + sxy : l + sxy - N;
    const T xl = (T)x[l];
    const T g[3] = {((T)x[lx] - xl) * hx, ((T)x[ly] - xl) * hy, ((T)x[lz] - xl) * hz};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      T r = w[c * N + l] * g[c];
      if (!init) r = r + coef * (u[c * N + l] * su);
      u[c * N + l] = r;
      acc[0] += (double)r * (double)r;
    }
  }
  if (grid_sum_last<1>(acc, partials, &st->counter) && threadIdx.x == 0) {
    const double beta = sqrt(acc[0]);
    st->beta = beta;
    st->su = beta > 0.0 ? 1.0 / beta : 1.0;
    if (init) {
      st->normb = beta;
      st->betadd = beta;
    }
  }
}

// q = -bdiv(w * u) (ilsqr.rs:1248-1258), periodic backward differences
template <typename T>
__global__ void k_lsmr_div(int nx, int ny, int nz, T hx, T hy, T hz, const T* __restrict__ w,
                           const T* __restrict__ u, T* __restrict__ q, const LsmrState* st) {
  if (st->done) return;
  const long long N = (long long)nx * ny * nz, sxy = (long long)nx * ny;
  const T su = (T)st->su;
  auto wy = [&](int c, long long l) { return w[c * N + l] * (u[c * N + l] * su); };
  for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < N; l += (long long)gridDim.x * blockDim.x) {
    const unsigned r = (unsigned)l / (unsigned)nx;
    const int i = (int)((unsigned)l - r * (unsigned)nx);
    const int j = (int)(r % (unsigned)ny);
    const int k = (int)(r / (unsigned)ny);
    const long long lx = i > 0 ? l - 1 : l - 1 + nx;
    const long long ly = j > 0 ? l - nx : l - nx + sxy;
    const long long lz = k > 0 ? l - sxy : l - sxy + N;
    const T div = (wy(0, l) - wy(0, lx)) * hx + (wy(1, l) - wy(1, ly)) * hy + (wy(2, l) - wy(2, lz)) * hz;
    q[l] = -div;
  }
}

template <typename T>
__global__ void k_lsmr_init(long long N, const T* __restrict__ v, T* __restrict__ h, T* __restrict__ hbar,
                            T* __restrict__ x, const LsmrState* st) {
  const T sv = (T)st->sv;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    h[i] = v[i] * sv;
    hbar[i] = T(0);
    x[i] = T(0);
  }
}

// h_bar = h - c1*h_bar; x += c2*h_bar; h = v - c3*h (ilsqr.rs:445-449), then ||x|| and
// the stopping tests (ilsqr.rs:487-510) in the last block.
template <typename T>
__global__ void k_lsmr_update(long long N, T* __restrict__ h, T* __restrict__ hbar, T* __restrict__ x,
                              const T* __restrict__ v, LsmrState* st, double* partials) {
  if (st->done) return;
  const T c1 = (T)st->c_hbar, c2 = (T)st->c_x, c3 = (T)st->c_h, sv = (T)st->sv;
  double acc[1] = {0.0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const T hb = h[i] - c1 * hbar[i];
    hbar[i] = hb;
    const T xi = x[i] + c2 * hb;
    x[i] = xi;
    h[i] = v[i] * sv - c3 * h[i];
    acc[0] += (double)xi * (double)xi;
  }
  if (grid_sum_last<1>(acc, partials, &st->counter) && threadIdx.x == 0) {
    const double normx = sqrt(acc[0]);
    const double test1 = st->normr / (st->normb + 1e-20);
    const double test2 = st->norm_ar / ((st->norm_a * st->normr) + 1e-20);
    const double test3 = 1.0 / (st->cond_a + 1e-20);
    const double rtol = st->btol + st->atol * st->norm_a * normx / (st->normb + 1e-20);
    st->iters += 1;
    if (test3 <= 1.0 / 1e8 || test2 <= st->atol || test1 <= rtol) st->done = 1;
  }
}

template <typename T>
__global__ void k_ilsqr_out(long long N, const double* __restrict__ xlsqr, const T* __restrict__ xsa,
                            const uint8_t* __restrict__ m, double* __restrict__ chi, double* __restrict__ xsa_out) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const bool in = m[i] != 0;
    const double s = in ? (double)xsa[i] : 0.0;
    chi[i] = in ? xlsqr[i] - s : 0.0;
    if (xsa_out) xsa_out[i] = s;
  }
}

// Replay `one` (a fixed sequence of launches that all return once *done is set) up to
// `iters` times: as a CUDA graph of one iteration polled every 8 launches, or eagerly
// while profiling.  Returns the number of iterations the device counted.
template <class One>
void run_iterations(qsm_ctx* ctx, size_t iters, const int* d_done, One one) {
  if (iters == 0) return;
  int h_done = 0;
  auto poll = [&]() {
    d2h(ctx, &h_done, d_done, sizeof(int));
    sync(ctx);
    return h_done != 0;
  };
  if (ctx->profiling) {
    for (size_t it = 0; it < iters; ++it) {
      one();
      if ((it + 1) % 8 == 0 && poll()) return;
    }
    return;
  }
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  const uint64_t l0 = ctx->launches;
  QSM_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
  try {
    one();
  } catch (...) {
    cudaStreamEndCapture(ctx->stream, &graph);
    if (graph) cudaGraphDestroy(graph);
    throw;
  }
  QSM_CUDA(cudaStreamEndCapture(ctx->stream, &graph));
  const uint64_t per = ctx->launches - l0;
  ctx->launches = l0;
  cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ie != cudaSuccess) throw QsmError(QSM_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(ie));
  try {
    for (size_t it = 0; it < iters; ++it) {
      QSM_CUDA(cudaGraphLaunch(exec, ctx->stream));
      ctx->launches += per;
      if ((it + 1) % 8 == 0 && it + 1 < iters && poll()) break;
    }
  } catch (...) {
    cudaGraphExecDestroy(exec);
    throw;
  }
  cudaGraphExecDestroy(exec);
}

}  // namespace

// T: arithmetic of the Krylov steps (LSQR, step 1; LSMR, step 3) and of their vectors;
// TD: arithmetic of the direct step 2 (fastQSM filtering, TKD, the fit).  An FP64 context
// runs both in double; a mixed context runs step 2 in float and the Krylov steps in
// double unless its Krylov precision is set to mixed: the reference stops LSQR after 50
// iterations short of its tolerance, so its result is the truncated Krylov iterate, and
// float rounding in the operator is amplified about a thousandfold there.
template <typename T, typename TD>
void ilsqr_impl(qsm_ctx* ctx, const GridDims& d, const double* f, const uint8_t* mask, const double bdir[3],
                const qsm_ilsqr_params& p, qsm_progress_fn progress, void* user, double* chi, double* xsa_out,
                double* xfs_out, double* xlsqr_out) {
  using C = cplx_t<T>;
  using CD = cplx_t<TD>;
  const long long N = d.n;
  const char* pre = sizeof(T) == 4 ? "il32." : "il64.";
  auto nm = [&](const char* s) { return std::string(pre) + s; };
  const char* pre_d = sizeof(TD) == 4 ? "il32." : "il64.";
  auto nmd = [&](const char* s) { return std::string(pre_d) + s; };
  auto report = [&](size_t k) {
    if (progress) progress(user, k, 4);
  };
  double* xlsqr = xlsqr_out ? xlsqr_out : ws<double>(ctx, nm("xlsqr"), (size_t)N);
  const long long count = count_selected(ctx, mask, N);
  if (count == 0) {
    // every weight and every masked output is zero (the reference returns zeros)
    for (double* o : {chi, xsa_out, xfs_out, xlsqr_out})
      if (o) QSM_CUDA(cudaMemsetAsync(o, 0, sizeof(double) * N, ctx->stream));
    for (size_t k = 1; k <= 4; ++k) report(k);
    sync(ctx);
    return;
  }
  Fft3<T> fh = make_fft3<T>(ctx, d);
  KSpace K = make_kspace(ctx, d, bdir);
  const long long NH = fh.g.hsize();
  const T invn = (T)(1.0 / (double)N);
  double* partials = ws<double>(ctx, nm("partials"), std::max(x_partials(fh, 1), (size_t)kMaxPersistentBlocks * 4));
  unsigned* counter = ws<unsigned>(ctx, nm("counter"), 1);
  QSM_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned), ctx->stream));
  C* t = ws<C>(ctx, nm("t"), (size_t)NH);
  C* ub = ws<C>(ctx, nm("u"), (size_t)NH);
  C* vb = ws<C>(ctx, nm("v"), (size_t)NH);
  C* wb = ws<C>(ctx, nm("w"), (size_t)NH);
  C* xb = ws<C>(ctx, nm("x"), (size_t)NH);
  for (C* b : {t, ub, vb, wb, xb}) QSM_CUDA(cudaMemsetAsync(b, 0, sizeof(C) * NH, ctx->stream));
  double* dwork = ws<double>(ctx, nm("dwork"), (size_t)(3 * N));
  const double hx2 = 1.0 / (d.vsx * d.vsx), hy2 = 1.0 / (d.vsy * d.vsy), hz2 = 1.0 / (d.vsz * d.vsz);

  // ------------------------------------------------------------- step 1 --
  report(1);
  T* wl = ws<T>(ctx, nm("wlap"), (size_t)N);
  {
    LaunchScope ls(ctx, "ilsqr_lap");
    k_ilsqr_lap<<<grid1d(N), 256, 0, ctx->stream>>>(f, mask, d.nx, d.ny, d.nz, hx2, hy2, hz2, dwork);
    ls.done();
  }
  {
    const std::vector<double> th = percentiles(ctx, dwork, mask, N, count, {60.0, 99.9});
    LaunchScope ls(ctx, "ilsqr_lap_weights");
    k_lap_weights<T><<<grid1d(N), 256, 0, ctx->stream>>>(N, dwork, mask, th[0], th[1], wl);
    ls.done();
  }
  LsqrState* lst = ws<LsqrState>(ctx, nm("lsqr"), 1);
  {
    LsqrState init{};
    init.tol = 0.01;  // tol_lsqr, ilsqr.rs:966
    h2d(ctx, lst, &init, sizeof(init));
  }
  const int* ldone = &lst->done;
  T* mult = ws<T>(ctx, nm("m"), (size_t)NH);  // m, then sym(D)/m, then LSMR's k-space mask
  T* img = ws<T>(ctx, nm("img"), (size_t)N);
  spec_multiplier<T>(ctx, fh, OpHalfD<T>{K, 0}, mult, nullptr);
  // b = D * FFT(w*f) -> u, beta = ||b||
  run_x_r2c<T>(ctx, fh, t, LoadProduct<double, T>{f, wl, d.nx}, nullptr);
  run_yz<T, -1, 1>(ctx, fh, t, t, OpId<T>{}, nullptr);
  run_yz_acc<T, -1, 2, true>(ctx, fh, t, ub, OpLsqrHalf<T>{mult, d.nx, nullptr, lst, 2}, partials, counter, nullptr,
                             "fft_z_lsqr");
  const LsqrOperator<T> A{&fh, mult, wl, invn, t, img, lst, partials, counter};
  // v = A^H u, alpha; w = v
  lsqr_apply<T>(ctx, A, ub, &lst->su, vb, nullptr, 3);
  {
    LaunchScope ls(ctx, "lsqr_init");
    k_lsqr_init_w<T><<<grid1d(NH), 256, 0, ctx->stream>>>(NH, vb, wb, lst);
    ls.done();
  }
  const unsigned ugrid = grid1d(NH);
  run_iterations(ctx, 50, ldone, [&]() {  // maxit_lsqr, ilsqr.rs:967
    lsqr_apply<T>(ctx, A, vb, &lst->sv, ub, ub, 0);
    lsqr_apply<T>(ctx, A, ub, &lst->su, vb, vb, 1);
    LaunchScope ls(ctx, "lsqr_update");
    k_lsqr_update<T><<<ugrid, 256, 0, ctx->stream>>>(NH, xb, wb, vb, lst, partials);
    ls.done();
  });
  // xlsqr = mask * Re IFFT(D G_x), D G_x = sym(D)/m h_x under the real part
  spec_multiplier<T>(ctx, fh, OpHalfD<T>{K, 1}, mult, nullptr);
  {
    LsqrState one{};
    one.su = 1.0;
    h2d(ctx, lst, &one, sizeof(one));
  }
  run_yz<T, +1, 2, true>(ctx, fh, xb, t, OpScaleM<T>{mult, &lst->su}, nullptr);
  run_yz<T, +1, 1>(ctx, fh, t, t, OpId<T>{}, nullptr);
  run_x_c2r<T>(ctx, fh, t, StoreMaskedF64<T>{xlsqr, mask, d.nx, invn}, nullptr);

  // ------------------------------------------------------------- step 2 --
  report(2);
  // step 2 runs in TD; with TD == T its buffers are step 1's (same names, same sizes)
  Fft3<TD> fd = make_fft3<TD>(ctx, d);
  const TD invnd = (TD)(1.0 / (double)N);
  CD* Fb = ws<CD>(ctx, nmd("v"), (size_t)NH);  // FFT(f) along x and y
  CD* td = ws<CD>(ctx, nmd("t"), (size_t)NH);
  TD* hs = ws<TD>(ctx, nmd("h"), (size_t)NH);  // SMV kernel spectrum (r = 3)
  smv_multiplier<TD>(ctx, fd, smv_sphere(d, 3.0), kSmvS, 0.0, hs);
  run_x_r2c<TD>(ctx, fd, Fb, LoadCast<double, TD>{f, d.nx}, nullptr);
  run_yz<TD, -1, 1>(ctx, fd, Fb, Fb, OpId<TD>{}, nullptr);
  OpFsFilter<TD> filt{K, hs, 0.001, 0.0, 0.0, 1};
  {
    LaunchScope ls(ctx, "ilsqr_dipole_pow");
    k_dipole_pow<<<grid1d(N), 256, 0, ctx->stream>>>(K, d.nx, d.ny, d.nz, 0.001, dwork);
    ls.done();
    const std::vector<double> th = percentiles(ctx, dwork, nullptr, N, N, {1.0, 30.0});
    filt.lo = th[0];
    filt.range = th[1] - th[0];
  }
  TD* xfs_raw = ws<TD>(ctx, nmd("xfs_raw"), (size_t)N);
  TD* xtkd = ws<TD>(ctx, nmd("xtkd"), (size_t)N);
  TD* xfs = ws<TD>(ctx, nmd("xfs"), (size_t)N);
  run_z_fused<TD>(ctx, fd, Fb, td, filt, nullptr);
  run_yz<TD, +1, 1>(ctx, fd, td, td, OpId<TD>{}, nullptr);
  run_x_c2r<TD>(ctx, fd, td, StoreMaskedT<TD>{xfs, mask, d.nx, invnd}, nullptr);
  run_x_r2c<TD>(ctx, fd, td, LoadCast<TD, TD>{xfs, d.nx}, nullptr);
  run_yz<TD, -1, 1>(ctx, fd, td, td, OpId<TD>{}, nullptr);
  filt.with_sign = 0;
  run_z_fused<TD>(ctx, fd, td, td, filt, nullptr);
  run_yz<TD, +1, 1>(ctx, fd, td, td, OpId<TD>{}, nullptr);
  run_x_c2r<TD>(ctx, fd, td, StoreMaskedT<TD>{xfs_raw, mask, d.nx, invnd}, nullptr);
  run_z_fused<TD>(ctx, fd, Fb, td, OpTkdInv<TD>{K, 1.0 / 8.0}, nullptr);
  run_yz<TD, +1, 1>(ctx, fd, td, td, OpId<TD>{}, nullptr);
  run_x_c2r<TD>(ctx, fd, td, StoreMaskedT<TD>{xtkd, mask, d.nx, invnd}, nullptr);
  {
    double* sums = ws<double>(ctx, nmd("sums"), 4);
    LaunchScope ls(ctx, "fastqsm_sums");
    k_fs_sums<TD><<<grid1d(N), 256, 0, ctx->stream>>>(N, xfs_raw, xtkd, partials, counter, sums);
    ls.done();
    double s[4];
    d2h(ctx, s, sums, sizeof(s));
    sync(ctx);
    const double n_all = (double)N;
    const double det = s[2] * n_all - s[0] * s[0];
    double a = 1.0, b = 0.0;
    if (std::fabs(det) > 1e-20) {
      a = (n_all * s[3] - s[0] * s[1]) / det;
      b = (s[2] * s[1] - s[0] * s[3]) / det;
    }
    LaunchScope ls2(ctx, "fastqsm_final");
    k_fs_final<TD><<<grid1d(N), 256, 0, ctx->stream>>>(N, xfs_raw, mask, a, b, xfs, xfs_out);
    ls2.done();
  }

  // ------------------------------------------------------------- step 3 --
  report(3);
  T* wg = ws<T>(ctx, nm("wgrad"), (size_t)(3 * N));
  {
    LaunchScope ls(ctx, "ilsqr_fgrad_masked");
    k_fgrad_masked<TD><<<wave_grid(ctx, k_fgrad_masked<TD>, N), 256, 0, ctx->stream>>>(xfs, mask, d.nx, d.ny, d.nz, 1.0 / d.vsx, 1.0 / d.vsy,
                                                          1.0 / d.vsz, dwork);
    ls.done();
    const std::vector<double> tx = percentiles(ctx, dwork, mask, N, count, {50.0, 70.0});
    const std::vector<double> ty = percentiles(ctx, dwork + N, mask, N, count, {50.0, 70.0});
    const std::vector<double> tz = percentiles(ctx, dwork + 2 * N, mask, N, count, {50.0, 70.0});
    LaunchScope ls2(ctx, "ilsqr_grad_weights");
    k_grad_weights<T><<<wave_grid(ctx, k_grad_weights<T>, N), 256, 0, ctx->stream>>>(N, dwork, mask, tx[0], tx[1], ty[0], ty[1], tz[0], tz[1], wg);
    ls2.done();
  }
  LsmrState* mst = ws<LsmrState>(ctx, nm("lsmr"), 1);
  {
    LsmrState init{};
    init.rho = 1.0;
    init.rho_bar = 1.0;
    init.c_bar = 1.0;
    init.rhodold = 1.0;
    init.minrbar = 1e100;
    init.atol = p.tol;
    init.btol = p.tol;
    h2d(ctx, mst, &init, sizeof(init));
  }
  const int* mdone = &mst->done;
  // N-length LSMR vectors reuse the idle LSQR buffers (each holds 2*NH >= N reals)
  T* vv = reinterpret_cast<T*>(vb);
  T* hh = reinterpret_cast<T*>(wb);
  T* hbar = reinterpret_cast<T*>(xb);
  T* rq = reinterpret_cast<T*>(t);  // r / q image
  T* u3 = ws<T>(ctx, nm("lsmr_u"), (size_t)(3 * N));
  T* xx = ws<T>(ctx, nm("lsmr_x"), (size_t)N);
  C* spec = ws<C>(ctx, nm("lsmr_spec"), (size_t)fh.g.hsize());
  QSM_CUDA(cudaMemsetAsync(spec, 0, sizeof(C) * fh.g.hsize(), ctx->stream));
  const T hx = (T)(1.0 / d.vsx), hy = (T)(1.0 / d.vsy), hz = (T)(1.0 / d.vsz);
  spec_multiplier<T>(ctx, fh, OpMic<T>{K}, mult, nullptr);
  auto mic_chain = [&](const auto& load, const auto& store) {
    run_x_r2c<T>(ctx, fh, spec, load, mdone);
    run_yz<T, -1, 1>(ctx, fh, spec, spec, OpId<T>{}, mdone);
    run_z_fused_m<T>(ctx, fh, spec, spec, mult, mdone);
    run_yz<T, +1, 1>(ctx, fh, spec, spec, OpId<T>{}, mdone);
    run_x_c2r<T>(ctx, fh, spec, store, mdone);
  };
  auto at_u = [&](int init) {  // v = A^T u (- beta v)
    {
      LaunchScope ls(ctx, "lsmr_div");
      k_lsmr_div<T><<<grid1d(N), 256, 0, ctx->stream>>>(d.nx, d.ny, d.nz, hx, hy, hz, wg, u3, rq, mst);
      ls.done();
    }
    mic_chain(LoadCast<T, T>{rq, d.nx}, StoreLsmrV<T>{vv, d.nx, invn, mst, partials, init, 0.0});
  };
  {
    LaunchScope ls(ctx, "lsmr_grad");
    k_lsmr_grad<double, T><<<wave_grid(ctx, k_lsmr_grad<double, T>, N), 256, 0, ctx->stream>>>(d.nx, d.ny, d.nz, hx, hy, hz, xlsqr, wg, u3, mst,
                                                                partials, 1);
    ls.done();
  }
  at_u(1);
  {
    LaunchScope ls(ctx, "lsmr_init");
    k_lsmr_init<T><<<grid1d(N), 256, 0, ctx->stream>>>(N, vv, hh, hbar, xx, mst);
    ls.done();
  }
  run_iterations(ctx, p.max_iter, mdone, [&]() {
    mic_chain(LoadScaled<T>{vv, &mst->sv, d.nx}, StoreReal<T>{rq, d.nx, invn});
    {
      LaunchScope ls(ctx, "lsmr_grad");
      k_lsmr_grad<T, T><<<wave_grid(ctx, k_lsmr_grad<T, T>, N), 256, 0, ctx->stream>>>(d.nx, d.ny, d.nz, hx, hy, hz, rq, wg, u3, mst, partials, 0);
      ls.done();
    }
    at_u(0);
    LaunchScope ls(ctx, "lsmr_update");
    k_lsmr_update<T><<<wave_grid(ctx, k_lsmr_update<T>, N), 256, 0, ctx->stream>>>(N, hh, hbar, xx, vv, mst, partials);
    ls.done();
  });

  // ------------------------------------------------------------- step 4 --
  {
    LaunchScope ls(ctx, "ilsqr_out");
    k_ilsqr_out<T><<<grid1d(N), 256, 0, ctx->stream>>>(N, xlsqr, xx, mask, chi, xsa_out);
    ls.done();
  }
  sync(ctx);
  report(4);
}

// ---------------------------------------------------- the LSQR operator alone ----
// The operator takes any full spectrum x, but A sees only the real image of D x: with
// Y(k) = (D(k) x(k) + conj(D(-k) x(-k))) / 2 that is h = Y / m (0 where m is, for there
// D(k) = D(-k) = 0), and A's h = m G is y = D G.
template <typename T>
__global__ void __launch_bounds__(128)
    k_lsqr_fold(Geom g, KSpace K, const T* __restrict__ m, const double2* __restrict__ x, cplx_t<T>* __restrict__ h) {
  const int iy = blockIdx.x, iz = blockIdx.y;
  const int my = iy ? g.ny - iy : 0, mz = iz ? g.nz - iz : 0;
  const long long row = ((long long)iz * g.ny + iy) * g.pitch;
  const double2* xa = x + ((long long)iz * g.ny + iy) * g.nx;
  const double2* xb = x + ((long long)mz * g.ny + my) * g.nx;
  for (int ix = threadIdx.x; ix < g.pitch; ix += blockDim.x) {
    cplx_t<T> v = mk<cplx_t<T>>(T(0), T(0));
    if (ix < g.nxh && m[row + ix] != T(0)) {
      const int mx = ix ? g.nx - ix : 0;
      const double da = dip(K, ix, iy, iz), db = dip(K, mx, my, mz), r = 0.5 / (double)m[row + ix];
      const double2 a = xa[ix], b = xb[mx];
      v = mk<cplx_t<T>>((T)((da * a.x + db * b.x) * r), (T)((da * a.y - db * b.y) * r));
    }
    h[row + ix] = v;
  }
}
template <typename T>
__global__ void __launch_bounds__(128)
    k_lsqr_unfold(Geom g, KSpace K, const T* __restrict__ m, const cplx_t<T>* __restrict__ h, double2* __restrict__ y) {
  const int iy = blockIdx.x, iz = blockIdx.y;
  const int my = iy ? g.ny - iy : 0, mz = iz ? g.nz - iz : 0;
  const long long rowa = ((long long)iz * g.ny + iy) * g.pitch, rowb = ((long long)mz * g.ny + my) * g.pitch;
  for (int ix = threadIdx.x; ix < g.nx; ix += blockDim.x) {
    const bool own = ix < g.nxh;
    const long long i = own ? rowa + ix : rowb + (g.nx - ix);
    const double mm = (double)m[i];
    const double r = mm != 0.0 ? dip(K, ix, iy, iz) / mm : 0.0;
    const cplx_t<T> v = h[i];
    y[((long long)iz * g.ny + iy) * g.nx + ix] = make_double2(r * (double)v.x, own ? r * (double)v.y : -r * (double)v.y);
  }
}
template <typename T>
__global__ void k_cast_real(long long n, const double* __restrict__ in, T* __restrict__ out) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = (T)in[i];
}

// y = D * FFT(w * Re(IFFT(D * x))): one application of lsqr_step's operator
// (src/inversion/ilsqr.rs:988-1010) by the solver's own (lsqr_apply).
template <typename T>
void lsqr_operator_impl(qsm_ctx* ctx, const GridDims& d, const double bdir[3], const double* w, const double2* x,
                        double2* y) {
  using C = cplx_t<T>;
  const std::string pre = sizeof(T) == 4 ? "ilop32." : "ilop64.";
  const Fft3<T> f = make_fft3<T>(ctx, d);
  const KSpace K = make_kspace(ctx, d, bdir);
  const size_t N = (size_t)d.n, NH = (size_t)f.g.hsize();
  C* h = ws<C>(ctx, pre + "h", NH);
  C* out = ws<C>(ctx, pre + "y", NH);
  T* m = ws<T>(ctx, pre + "m", NH);
  T* wl = ws<T>(ctx, pre + "w", N);
  LsqrState* st = ws<LsqrState>(ctx, pre + "state", 1);
  const LsqrOperator<T> A{&f, m, wl, (T)(1.0 / (double)d.n), ws<C>(ctx, pre + "t", NH), ws<T>(ctx, pre + "img", N), st,
                          ws<double>(ctx, pre + "partials", std::max(x_partials(f, 1), (size_t)kMaxPersistentBlocks * 4)),
                          ws<unsigned>(ctx, pre + "counter", 1)};
  LsqrState init{};
  init.su = 1.0;
  h2d(ctx, st, &init, sizeof(init));
  QSM_CUDA(cudaMemsetAsync(A.counter, 0, sizeof(unsigned), ctx->stream));
  spec_multiplier<T>(ctx, f, OpHalfD<T>{K, 0}, m, nullptr);
  const dim3 rows((unsigned)d.ny, (unsigned)d.nz);
  {
    LaunchScope ls(ctx, "ilsqr_op_pack");
    k_cast_real<T><<<grid1d(d.n), 256, 0, ctx->stream>>>(d.n, w, wl);
    k_lsqr_fold<T><<<rows, 128, 0, ctx->stream>>>(f.g, K, m, x, h);
    ls.done();
  }
  lsqr_apply<T>(ctx, A, h, &st->su, out, nullptr, 3);
  {
    LaunchScope ls(ctx, "ilsqr_op_unpack");
    k_lsqr_unfold<T><<<rows, 128, 0, ctx->stream>>>(f.g, K, m, out, y);
    ls.done();
  }
  sync(ctx);
}

void ilsqr_device(qsm_ctx* ctx, const double* f, const uint8_t* m, const qsm_grid* grid, const double bdir[3],
                  const qsm_ilsqr_params* p, qsm_progress_fn progress, void* user, double* chi, double* xsa,
                  double* xfs, double* xlsqr) {
  GridDims d = check_grid(grid);
  check_ptr(f, "local_field");
  check_ptr(m, "mask");
  check_ptr(chi, "out_chi");
  check_ptr(p, "params");
  check_bdir(bdir);
  if (std::isnan(p->tol)) throw QsmError(QSM_ERR_INVALID_ARGUMENT, "tol is NaN");
  check_volume_finite(ctx, f, d.n, "local_field");
  if (d.nx < 2 || d.ny < 2 || d.nz < 2)
    throw QsmError(QSM_ERR_UNSUPPORTED_SIZE, "iLSQR needs every axis length >= 2 (one-sided stencils)");
  if (d.n >= (1LL << 32)) throw QsmError(QSM_ERR_UNSUPPORTED_SIZE, "iLSQR volumes hold fewer than 2^32 voxels");
  if (ctx->precision != QSM_PRECISION_MIXED)
    ilsqr_impl<double, double>(ctx, d, f, m, bdir, *p, progress, user, chi, xsa, xfs, xlsqr);
  else if (ctx->krylov_precision == QSM_PRECISION_MIXED)
    ilsqr_impl<float, float>(ctx, d, f, m, bdir, *p, progress, user, chi, xsa, xfs, xlsqr);
  else
    ilsqr_impl<double, float>(ctx, d, f, m, bdir, *p, progress, user, chi, xsa, xfs, xlsqr);
}

}  // namespace qsm

using namespace qsm;

extern "C" {

void qsm_ilsqr_params_default(qsm_ilsqr_params* p) {
  if (!p) return;
  p->tol = 0.01;  // IlsqrParams::default, src/inversion/ilsqr.rs:27-34
  p->max_iter = 50;
}

qsm_status qsm_ilsqr_device(qsm_ctx* ctx, const double* d_local_field, const uint8_t* d_mask, const qsm_grid* grid,
                            const double bdir[3], const qsm_ilsqr_params* params, qsm_progress_fn progress, void* user,
                            double* d_out_chi, double* d_out_xsa, double* d_out_xfs, double* d_out_xlsqr) {
  return guarded(ctx, [&] {
    ilsqr_device(ctx, d_local_field, d_mask, grid, bdir, params, progress, user, d_out_chi, d_out_xsa, d_out_xfs,
                 d_out_xlsqr);
  });
}

qsm_status qsm_ilsqr_lsqr_operator_device(qsm_ctx* ctx, const qsm_grid* grid, const double bdir[3],
                                          const double* d_weights, const double* d_x, double* d_y) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_bdir(bdir);
    check_ptr(d_weights, "weights");
    check_ptr(d_x, "x");
    check_ptr(d_y, "y");
    if ((reinterpret_cast<uintptr_t>(d_x) | reinterpret_cast<uintptr_t>(d_y)) % 16 != 0)
      throw QsmError(QSM_ERR_INVALID_ARGUMENT, "complex vectors must be 16-byte aligned");
    const double2* x = reinterpret_cast<const double2*>(d_x);
    double2* y = reinterpret_cast<double2*>(d_y);
    if (ctx->precision == QSM_PRECISION_MIXED) lsqr_operator_impl<float>(ctx, d, bdir, d_weights, x, y);
    else lsqr_operator_impl<double>(ctx, d, bdir, d_weights, x, y);
  });
}

qsm_status qsm_ilsqr(qsm_ctx* ctx, const double* local_field, const uint8_t* mask, const qsm_grid* grid,
                     const double bdir[3], const qsm_ilsqr_params* params, qsm_progress_fn progress, void* user,
                     double* out_chi, double* out_xsa, double* out_xfs, double* out_xlsqr) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_ptr(local_field, "local_field");
    check_ptr(mask, "mask");
    check_ptr(out_chi, "out_chi");
    const size_t N = (size_t)d.n;
    double* extra[3] = {nullptr, nullptr, nullptr};
    double* hout[3] = {out_xsa, out_xfs, out_xlsqr};
    const char* names[3] = {"io.xsa", "io.xfs", "io.xlsqr"};
    for (int i = 0; i < 3; ++i)
      if (hout[i]) extra[i] = reinterpret_cast<double*>(ws_get(ctx, names[i], N * sizeof(double)));
    with_host_io(ctx, d.n, local_field, mask, out_chi, [&](const double* f, const uint8_t* m, double* o) {
      ilsqr_device(ctx, f, m, grid, bdir, params, progress, user, o, extra[0], extra[1], extra[2]);
      for (int i = 0; i < 3; ++i)
        if (hout[i]) d2h(ctx, hout[i], extra[i], N * sizeof(double));
    });
  });
}

}  // extern "C"
