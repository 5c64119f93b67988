// Laplacian phase unwrapping and SMV-family background removal (SMV, SHARP,
// V-SHARP) on the GPU, plus the pipeline dispatcher run_bg_removal.
//
// Mask erosion decides "SMV(mask) > delta" with delta within ~1e-8 of a rational
// count/total for realistic kernels: it is decided by exact counts (smv.cu), and the sphere
// kernel's multipliers are evaluated in double, whatever the context precision; field
// filtering runs in the working precision.
#include "functors.cuh"
#include "smv.h"
#include "solvers.h"

#include <algorithm>
#include <cstring>

namespace qsm {

// Rust % on f64 is the truncated fmod; out of line, so that its loop costs the callers no
// registers
__device__ __noinline__ double turn_remainder(double x) { return fmod(x, 2.0 * kPi); }

__device__ __forceinline__ double wrap_pi(double x) {
  // src/unwrap/laplacian.rs:21-30
  const double two_pi = 2.0 * kPi;
  // differences of wrapped phases lie within a turn, where the remainder is x itself
  double y = x;
  if (!(fabs(x) < two_pi)) y = turn_remainder(x);
  if (y > kPi) y -= two_pi;
  else if (y < -kPi) y += two_pi;
  return y;
}

// Wrapped 7-point Laplacian (periodic), masked, in double (src/unwrap/laplacian.rs:34-78,
// 146-149), into working precision.  32x8 (x, y) tiles, each thread marching zchunk planes
// with the z neighbours in registers, x neighbours by shuffle.  A pass of its own: inside
// the X transform's loader every row element was a copy of this code with its six fmod
// loops, and the X pass ran 265 us at 256x256x176, 250 with the loops skipped; this kernel
// and the plain X pass take 94 us together.
template <typename T>
__global__ void __launch_bounds__(256)
    k_wrapped_lap(int nx, int ny, int nz, int zchunk, double dx2, double dy2, double dz2, const double* __restrict__ ph,
                  const uint8_t* __restrict__ mask, T* __restrict__ lap) {
  const int lane = threadIdx.x & 31;
  const int e = blockIdx.x * 32 + lane, j = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (j >= ny) return;  // whole warps
  const bool in = e < nx;
  const int i = in ? e : nx - 1;
  const int k0 = blockIdx.z * zchunk, k1 = min(nz, k0 + zchunk);
  const long long sz = (long long)nx * ny;
  const int ip = i + 1 < nx ? i + 1 : 0, im = i > 0 ? i - 1 : nx - 1;
  const double* row = ph + (long long)j * nx;
  const double* rowp = ph + (long long)(j + 1 < ny ? j + 1 : 0) * nx + i;
  const double* rowm = ph + (long long)(j > 0 ? j - 1 : ny - 1) * nx + i;
  double um = row[(k0 > 0 ? k0 - 1 : nz - 1) * sz + i];
  double u = row[k0 * sz + i];
  for (int k = k0; k < k1; ++k) {
    const long long b = k * sz;
    const double up = row[(k + 1 < nz ? k + 1 : 0) * sz + i];
    const double yp = rowp[b], ym = rowm[b];
    double xp = __shfl_down_sync(0xffffffffu, u, 1), xm = __shfl_up_sync(0xffffffffu, u, 1);
    if (lane == 31 || i + 1 >= nx) xp = row[b + ip];
    if (lane == 0) xm = row[b + im];
    const bool on = in && mask[b + (long long)j * nx + i] != 0;
    if (in) {
      T v = T(0);
      if (on) {
        const double lx = (wrap_pi(xp - u) - wrap_pi(u - xm)) * dx2;
        const double ly = (wrap_pi(yp - u) - wrap_pi(u - ym)) * dy2;
        const double lz = (wrap_pi(up - u) - wrap_pi(u - um)) * dz2;
        v = (T)(lx + ly + lz);
      }
      lap[b + (long long)j * nx + i] = v;
    }
    um = u;
    u = up;
  }
}

// Poisson solve multiplier 1/lambda, 0 where |lambda| <= 1e-20 (src/unwrap/laplacian.rs:91-117)
template <typename T> struct OpPoisson {
  using C = cplx_t<T>;
  KSpace K;
  __device__ __forceinline__ C mid(C v, int ix, int iy, int iz, long long) const {
    const double lam = K.poisson(ix, iy, iz);
    if (fabs(lam) > 1e-20) return cscale(v, (T)(1.0 / lam));
    return mk<C>(T(0), T(0));
  }
};

// V-SHARP first-hit selection (src/bgremove/vsharp.rs:168-176): the voxels that this
// radius is the first to keep
template <typename T> struct StoreSelect {
  const uint8_t* first;
  const uint8_t* taken;
  const unsigned* row_hits;  // bit idx mod 32: some voxel of the row is kept first by idx
  T* local;
  int nx, idx;
  T scale;
  static constexpr bool kRowFilter = true;
  __device__ __forceinline__ bool wants_row(int row) const { return (__ldg(row_hits + row) >> (idx & 31)) & 1u; }
  __device__ __forceinline__ void operator()(int row, int e, T v) {
    const long long i = (long long)row * nx + e;
    if (__ldg(first + i) == idx && __ldg(taken + i) == 0) local[i] = v * scale;
  }
  __device__ __forceinline__ void finish() {}
};

// eroded = 1 where the only sphere keeps the voxel
__global__ void k_first_to_mask(long long n, const uint8_t* first, uint8_t* mask) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    mask[i] = first[i] == 0 ? 1 : 0;
}
// row_hits[row] = the set of first[] values (mod 32) in the row; one warp per row
__global__ void __launch_bounds__(256)
    k_row_hits(int nx, int nrows, const uint8_t* __restrict__ first, unsigned* __restrict__ hits) {
  for (int row = blockIdx.x * 8 + (threadIdx.x >> 5); row < nrows; row += gridDim.x * 8) {
    unsigned h = 0u;
    for (int e = threadIdx.x & 31; e < nx; e += 32) {
      const unsigned f = first[(long long)row * nx + e];
      if (f != 255u) h |= 1u << (f & 31u);
    }
    h = __reduce_or_sync(0xffffffffu, h);
    if ((threadIdx.x & 31) == 0) hits[row] = h;
  }
}
// taken |= some sphere keeps the voxel
__global__ void k_first_taken(long long n, const uint8_t* __restrict__ first, uint8_t* __restrict__ taken) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    if (first[i] != 255) taken[i] = 1;
}

// SMV: local = eroded == 1 ? field - SMV(field) : 0 (src/bgremove/smv.rs:50-56)
template <typename T> struct StoreSmvLocal {
  const double* field;
  const uint8_t* eroded;
  double* out;
  int nx;
  T scale;
  __device__ __forceinline__ void operator()(int row, int e, T v) {
    const long long i = (long long)row * nx + e;
    out[i] = __ldg(eroded + i) == 1 ? __ldg(field + i) - (double)(v * scale) : 0.0;
  }
  __device__ __forceinline__ void finish() {}
};

// ------------------------------------------------------------ shared steps --
// Full forward transform (spectrum only) of a loaded real volume.
template <typename T, class Load>
void forward3(qsm_ctx* ctx, const Fft3<T>& f, const Load& ld, cplx_t<T>* dst) {
  run_x_r2c<T>(ctx, f, dst, ld, nullptr);
  run_yz<T, -1, 1>(ctx, f, dst, dst, OpId<T>{}, nullptr);
  run_yz<T, -1, 2>(ctx, f, dst, dst, OpId<T>{}, nullptr);
}

// eroded = mean of the mask over the sphere > delta (src/kernels/smv.rs:73-105)
void smv_erode(qsm_ctx* ctx, const GridDims& d, const uint8_t* mask, const SmvSphere& s, double delta,
               uint8_t* eroded) {
  smv_erode_first(ctx, d, mask, {s}, delta, eroded);
  LaunchScope ls(ctx, "smv_mask");
  k_first_to_mask<<<grid1d(d.n), 256, 0, ctx->stream>>>(d.n, eroded, eroded);
  ls.done();
}

// 1 - sqrt(1e-7), src/bgremove/sharp.rs:79 and vsharp.rs:129
double sharp_delta() { return 1.0 - std::sqrt(1e-7); }

// SHARP core (src/bgremove/sharp.rs:64-131)
template <typename T>
void sharp_impl(qsm_ctx* ctx, const GridDims& d, const double* field, const uint8_t* mask, double threshold,
                double radius, double* out_local, uint8_t* out_mask) {
  using C = cplx_t<T>;
  Fft3<T> f = make_fft3<T>(ctx, d);
  const size_t H = (size_t)f.g.hsize();
  T* m = ws<T>(ctx, "bg.mult", H);
  C* spec = ws<C>(ctx, "spec", H);
  T* g = ws<T>(ctx, "bg.img", (size_t)d.n);
  const SmvSphere s = smv_sphere(d, radius);
  smv_erode(ctx, d, mask, s, sharp_delta(), out_mask);
  const T scale = (T)(1.0 / (double)d.n);
  // high-pass, mask
  smv_multiplier<T>(ctx, f, s, kSmvOneMinusS, 0.0, m);
  run_x_r2c<T>(ctx, f, spec, LoadCast<double, T>{field, d.nx}, nullptr);
  run_yz<T, -1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_z_fused_m<T>(ctx, f, spec, spec, m, nullptr);
  run_yz<T, +1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_x_c2r<T>(ctx, f, spec, StoreMaskEqOne<T>{g, out_mask, d.nx, scale}, nullptr);
  // SHARP deconvolution: |1 - S| < thr -> 0, else X / (1 - S) (sharp.rs:111-119), mask
  smv_multiplier<T>(ctx, f, s, kSmvDeconv, threshold, m);
  run_x_r2c<T>(ctx, f, spec, LoadCast<T, T>{g, d.nx}, nullptr);
  run_yz<T, -1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_z_fused_m<T>(ctx, f, spec, spec, m, nullptr);
  run_yz<T, +1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_x_c2r<T>(ctx, f, spec, StoreMaskedF64<T>{out_local, out_mask, d.nx, scale}, nullptr);
}

// V-SHARP (src/bgremove/vsharp.rs:88-199), radii already sorted descending, >= 2.  The
// erosions of all radii are one distance transform (smv.cu), so the radius that keeps each
// voxel first is known before any field is filtered; a radius then costs its multiplier
// and one inverse transform.
template <typename T>
void vsharp_impl(qsm_ctx* ctx, const GridDims& d, const double* field, const uint8_t* mask,
                 const std::vector<double>& radii, double threshold, qsm_progress_fn progress, void* user,
                 double* out_local, uint8_t* out_mask) {
  using C = cplx_t<T>;
  Fft3<T> f = make_fft3<T>(ctx, d);
  const size_t H = (size_t)f.g.hsize();
  const size_t N = (size_t)d.n;
  T* m = ws<T>(ctx, "bg.mult", H);
  C* Ff = ws<C>(ctx, "bg.Ff", H);
  C* tmp = ws<C>(ctx, "bg.tmpT", H);
  uint8_t* first = ws<uint8_t>(ctx, "bg.first", N);
  unsigned* hits = ws<unsigned>(ctx, "bg.row_hits", (size_t)d.ny * d.nz);
  T* local = ws<T>(ctx, "bg.img", N);
  QSM_CUDA(cudaMemsetAsync(out_mask, 0, N, ctx->stream));
  QSM_CUDA(cudaMemsetAsync(local, 0, N * sizeof(T), ctx->stream));
  forward3<T>(ctx, f, LoadCast<double, T>{field, d.nx}, Ff);
  const T scale = (T)(1.0 / (double)d.n);
  const double delta = sharp_delta();
  std::vector<SmvSphere> spheres;
  for (double r : radii) spheres.push_back(smv_sphere(d, r));
  constexpr size_t kGroup = 254;  // radii per erosion call
  for (size_t g0 = 0; g0 < radii.size(); g0 += kGroup) {
    const size_t g1 = std::min(radii.size(), g0 + kGroup);
    smv_erode_first(ctx, d, mask, std::vector<SmvSphere>(spheres.begin() + g0, spheres.begin() + g1), delta, first);
    {
      LaunchScope ls(ctx, "vsharp_rows");
      k_row_hits<<<x_rows_grid(ctx, k_row_hits, f.g), 256, 0, ctx->stream>>>(d.nx, d.ny * d.nz, first, hits);
      ls.done();
    }
    for (size_t idx = g0; idx < g1; ++idx) {
      if (progress) progress(user, idx + 1, radii.size());
      smv_multiplier<T>(ctx, f, spheres[idx], kSmvOneMinusS, 0.0, m);
      run_yz<T, +1, 2, true>(ctx, f, Ff, tmp, OpPreMult<T>{m}, nullptr);
      run_yz<T, +1, 1>(ctx, f, tmp, tmp, OpId<T>{}, nullptr);
      run_x_c2r<T>(ctx, f, tmp, StoreSelect<T>{first, out_mask, hits, local, d.nx, (int)(idx - g0), scale}, nullptr);
    }
    LaunchScope ls(ctx, "vsharp_mask");
    k_first_taken<<<grid1d(d.n), 256, 0, ctx->stream>>>(d.n, first, out_mask);
    ls.done();
  }
  // deconvolution with the largest kernel's inverse (vsharp.rs:147-156)
  C* spec = ws<C>(ctx, "spec", H);
  smv_multiplier<T>(ctx, f, spheres[0], kSmvDeconv, threshold, m);
  run_x_r2c<T>(ctx, f, spec, LoadCast<T, T>{local, d.nx}, nullptr);
  run_yz<T, -1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_z_fused_m<T>(ctx, f, spec, spec, m, nullptr);
  run_yz<T, +1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_x_c2r<T>(ctx, f, spec, StoreMaskedF64<T>{out_local, out_mask, d.nx, scale}, nullptr);
}

// SMV (src/bgremove/smv.rs:31-59)
template <typename T>
void smv_impl(qsm_ctx* ctx, const GridDims& d, const double* field, const uint8_t* mask, double radius,
              double* out_local, uint8_t* out_mask) {
  using C = cplx_t<T>;
  Fft3<T> f = make_fft3<T>(ctx, d);
  const size_t H = (size_t)f.g.hsize();
  T* m = ws<T>(ctx, "bg.mult", H);
  C* spec = ws<C>(ctx, "spec", H);
  const SmvSphere s = smv_sphere(d, radius);
  smv_erode(ctx, d, mask, s, 1.0 - 1e-10, out_mask);
  smv_multiplier<T>(ctx, f, s, kSmvS, 0.0, m);
  run_x_r2c<T>(ctx, f, spec, LoadCast<double, T>{field, d.nx}, nullptr);
  run_yz<T, -1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_z_fused_m<T>(ctx, f, spec, spec, m, nullptr);
  run_yz<T, +1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_x_c2r<T>(ctx, f, spec, StoreSmvLocal<T>{field, out_mask, out_local, d.nx, (T)(1.0 / (double)d.n)}, nullptr);
}

// ------------------------------------------------------------------ iSMV --
// src/bgremove/ismv.rs:48-157.  Device state: iterations done, the change norm and its
// tolerance; the iteration whose top-of-loop test stops the loop (0: none).
struct IsmvState {
  int done;
  int k;  // iterations completed
  unsigned counter;
  int stop_at;
  double nr, eps;
};

// f_0 = field; nr_0 = ||eroded * field||, eps = tol * nr_0 (ismv.rs:106-120); a zero
// norm stops the loop at its first test
template <typename T>
__global__ void k_ismv_init(long long N, const double* __restrict__ field, const uint8_t* __restrict__ eroded,
                            double tol, size_t max_iter, T* __restrict__ f, IsmvState* st, double* partials) {
  double acc[1] = {0.0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const double v = field[i];
    f[i] = (T)v;
    const double e = v * (double)eroded[i];
    acc[0] += e * e;
  }
  if (grid_sum_last<1>(acc, partials, &st->counter) && threadIdx.x == 0) {
    const double nr = sqrt(acc[0]);
    st->nr = nr;
    st->eps = tol * nr;
    st->k = 0;
    st->stop_at = 0;
    st->done = 0;
    if (max_iter > 0 && nr <= tol * nr) {
      st->done = 1;
      st->stop_at = 1;
    }
  }
}

// f_k = eroded * Re IFFT(F(f_{k-1}) S) + (m0 - eroded) field, FP64 sum of (f0 - f_k)^2
// with f0 = eroded * field at k = 1 and f_{k-1} after (ismv.rs:127-155); the last block
// stores the norm and runs the next iteration's top-of-loop test.
template <typename T> struct StoreIsmv {
  T* out;
  const T* prev;  // f_{k-1}, or null at k = 1
  const double* field;
  const uint8_t* mask;
  const uint8_t* eroded;
  int nx;
  T scale;
  IsmvState* st;
  double* partials;
  int max_iter;
  double acc[1];
  __device__ __forceinline__ void operator()(int row, int e, T v) {
    const long long i = (long long)row * nx + e;
    const double er = (double)__ldg(eroded + i);
    const double fld = __ldg(field + i);
    const double m0 = __ldg(mask + i) != 0 ? 1.0 : 0.0;
    const T fn = (T)(er * (double)(v * scale) + fld * (m0 - er));
    out[i] = fn;
    const double f0 = prev ? (double)__ldg(prev + i) : fld * er;
    const double dd = f0 - (double)fn;
    acc[0] += dd * dd;
  }
  __device__ void finish() {
    if (!grid_sum_last<1>(acc, partials, &st->counter)) return;
    if (threadIdx.x + blockDim.x * threadIdx.y != 0) return;
    const double nr = sqrt(acc[0]);
    st->nr = nr;
    const int k = st->k + 1;
    st->k = k;
    if (k < max_iter && nr <= st->eps) {
      st->done = 1;
      st->stop_at = k + 1;
    }
  }
};

// local = mask ? field - f : 0 (ismv.rs:158-164)
template <typename T>
__global__ void k_ismv_out(long long N, const double* __restrict__ field, const uint8_t* __restrict__ mask,
                           const T* __restrict__ f, double* __restrict__ out) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x)
    out[i] = mask[i] != 0 ? field[i] - (double)f[i] : 0.0;
}

template <typename T>
void ismv_impl(qsm_ctx* ctx, const GridDims& d, const double* field, const uint8_t* mask,
               const qsm_ismv_params& p, qsm_progress_fn progress, void* user, double* out_local,
               uint8_t* out_mask) {
  using C = cplx_t<T>;
  Fft3<T> f = make_fft3<T>(ctx, d);
  const size_t H = (size_t)f.g.hsize();
  const long long N = d.n;
  const std::string pre = sizeof(T) == 4 ? "ismv32." : "ismv64.";
  T* Sr = ws<T>(ctx, pre + "Sr", H);
  C* spec = ws<C>(ctx, pre + "spec", H);
  T* fb[2] = {ws<T>(ctx, pre + "f0", (size_t)N), ws<T>(ctx, pre + "f1", (size_t)N)};
  IsmvState* st = ws<IsmvState>(ctx, pre + "state", 1);
  double* partials = ws<double>(ctx, pre + "partials", x_partials(f, 1));
  QSM_CUDA(cudaMemsetAsync(st, 0, sizeof(IsmvState), ctx->stream));
  const SmvSphere sphere = smv_sphere(d, p.radius);
  smv_multiplier<T>(ctx, f, sphere, kSmvS, 0.0, Sr);
  smv_erode(ctx, d, mask, sphere, 1.0 - 1e-10, out_mask);  // ismv.rs:166-169
  {
    LaunchScope ls(ctx, "ismv_init");
    k_ismv_init<T><<<grid1d(N), 256, 0, ctx->stream>>>(N, field, out_mask, p.tol, p.max_iter, fb[0], st, partials);
    ls.done();
  }
  const int* done = &st->done;
  const T scale = (T)(1.0 / (double)N);
  const int maxi = (int)std::min<size_t>(p.max_iter, (size_t)1 << 30);
  // iteration k reads fb[(k-1) % 2] and writes fb[k % 2]
  auto iter = [&](int k) {
    const T* in = fb[(k - 1) % 2];
    StoreIsmv<T> store{fb[k % 2], k == 1 ? nullptr : in, field, mask, out_mask, d.nx, scale, st, partials, maxi,
                       {0.0}};
    run_x_r2c<T>(ctx, f, spec, LoadCast<T, T>{in, d.nx}, done);
    run_yz<T, -1, 1>(ctx, f, spec, spec, OpId<T>{}, done);
    run_z_fused_m<T>(ctx, f, spec, spec, Sr, done);
    run_yz<T, +1, 1>(ctx, f, spec, spec, OpId<T>{}, done);
    run_x_c2r<T>(ctx, f, spec, store, done);
  };
  IsmvState hs{};
  size_t reported = 0;
  auto poll = [&]() {
    d2h(ctx, &hs, st, sizeof(hs));
    sync(ctx);
    const size_t through = hs.stop_at ? (size_t)hs.stop_at : (size_t)hs.k;
    if (progress)
      for (; reported < through; ++reported) progress(user, reported + 1, p.max_iter);
    return hs.done != 0;
  };
  const bool watch = progress != nullptr || p.tol > 0.0;
  bool stopped = false;
  if (maxi >= 1) {
    iter(1);
    if (maxi >= 2) {
      if (ctx->profiling) {
        for (int k = 2; k <= maxi && !stopped; ++k) {
          iter(k);
          if (watch && k % 8 == 0) stopped = poll();
        }
      } else {
        cudaGraph_t graph = nullptr;
        const uint64_t l0 = ctx->launches;
        QSM_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
        try {
          iter(2);
          iter(3);
        } catch (...) {
          cudaStreamEndCapture(ctx->stream, &graph);
          if (graph) cudaGraphDestroy(graph);
          throw;
        }
        QSM_CUDA(cudaStreamEndCapture(ctx->stream, &graph));
        const uint64_t per = ctx->launches - l0;
        ctx->launches = l0;
        cudaGraphExec_t exec = nullptr;
        const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess)
          throw QsmError(QSM_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(ie));
        try {
          const int pairs = (maxi - 1) / 2;
          for (int q = 0; q < pairs && !stopped; ++q) {
            QSM_CUDA(cudaGraphLaunch(exec, ctx->stream));
            ctx->launches += per;
            if (watch && (q + 1) % 4 == 0) stopped = poll();
          }
          if (!stopped && (maxi - 1) % 2 == 1) iter(maxi);
        } catch (...) {
          cudaGraphExecDestroy(exec);
          throw;
        }
        cudaGraphExecDestroy(exec);
      }
    }
  }
  poll();
  const int kdone = hs.k;
  {
    LaunchScope ls(ctx, "ismv_out");
    k_ismv_out<T><<<grid1d(N), 256, 0, ctx->stream>>>(N, field, mask, fb[kdone % 2], out_local);
    ls.done();
  }
  sync(ctx);
  if (progress) {
    const size_t through = hs.stop_at ? (size_t)hs.stop_at : p.max_iter;
    for (; reported < through; ++reported) progress(user, reported + 1, p.max_iter);
    if (hs.stop_at) progress(user, (size_t)hs.stop_at, (size_t)hs.stop_at);
  }
}

template <typename T>
void unwrap_impl(qsm_ctx* ctx, const GridDims& d, const double* phase, const uint8_t* mask, double* out) {
  using C = cplx_t<T>;
  Fft3<T> f = make_fft3<T>(ctx, d);
  KSpace K = make_kspace(ctx, d, nullptr);
  C* spec = ws<C>(ctx, "spec", (size_t)f.g.hsize());
  T* lap = ws<T>(ctx, sizeof(T) == 4 ? "unwrap.lap32" : "unwrap.lap64", (size_t)d.n);
  {
    // about 24 blocks per SM
    const int gx = (d.nx + 31) / 32, gy = (d.ny + 7) / 8;
    const long long zc = std::max<long long>(1, 24LL * sm_count(ctx) / ((long long)gx * gy));
    const int zchunk = (int)((d.nz + zc - 1) / zc);
    LaunchScope ls(ctx, "wrapped_lap");
    k_wrapped_lap<T><<<dim3(gx, gy, (d.nz + zchunk - 1) / zchunk), 256, 0, ctx->stream>>>(
        d.nx, d.ny, d.nz, zchunk, 1.0 / (d.vsx * d.vsx), 1.0 / (d.vsy * d.vsy), 1.0 / (d.vsz * d.vsz), phase, mask, lap);
    ls.done();
  }
  run_x_r2c<T>(ctx, f, spec, LoadCast<T, T>{lap, d.nx}, nullptr);
  run_yz<T, -1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_z_fused<T>(ctx, f, spec, spec, OpPoisson<T>{K}, nullptr);
  run_yz<T, +1, 1>(ctx, f, spec, spec, OpId<T>{}, nullptr);
  run_x_c2r<T>(ctx, f, spec, StoreMaskedF64<T>{out, mask, d.nx, (T)(1.0 / (double)d.n)}, nullptr);
}

void check_io(const void* a, const void* m, const void* o) {
  check_ptr(a, "input");
  check_ptr(m, "mask");
  check_ptr(o, "output");
}

void unwrap_device(qsm_ctx* ctx, const double* ph, const uint8_t* m, const qsm_grid* grid, double* out) {
  GridDims d = check_grid(grid);
  check_io(ph, m, out);
  check_volume_finite(ctx, ph, d.n, "phase");
  if (ctx->precision == QSM_PRECISION_MIXED) unwrap_impl<float>(ctx, d, ph, m, out);
  else unwrap_impl<double>(ctx, d, ph, m, out);
}

void smv_device(qsm_ctx* ctx, const double* f, const uint8_t* m, const GridDims& d, double radius, double* ol,
                uint8_t* om) {
  check_finite(radius, "radius");
  check_volume_finite(ctx, f, d.n, "field");
  if (ctx->precision == QSM_PRECISION_MIXED) smv_impl<float>(ctx, d, f, m, radius, ol, om);
  else smv_impl<double>(ctx, d, f, m, radius, ol, om);
}

void ismv_device(qsm_ctx* ctx, const double* f, const uint8_t* m, const GridDims& d, const qsm_ismv_params* p,
                 qsm_progress_fn progress, void* user, double* ol, uint8_t* om) {
  check_ptr(p, "params");
  check_finite(p->radius, "radius");
  if (std::isnan(p->tol)) throw QsmError(QSM_ERR_INVALID_ARGUMENT, "tol is NaN");
  check_volume_finite(ctx, f, d.n, "field");
  if (ctx->precision == QSM_PRECISION_MIXED) ismv_impl<float>(ctx, d, f, m, *p, progress, user, ol, om);
  else ismv_impl<double>(ctx, d, f, m, *p, progress, user, ol, om);
}

void sharp_device(qsm_ctx* ctx, const double* f, const uint8_t* m, const GridDims& d, double thr, double radius,
                  double* ol, uint8_t* om) {
  check_finite(thr, "threshold");
  check_finite(radius, "radius");
  check_volume_finite(ctx, f, d.n, "field");
  if (ctx->precision == QSM_PRECISION_MIXED) sharp_impl<float>(ctx, d, f, m, thr, radius, ol, om);
  else sharp_impl<double>(ctx, d, f, m, thr, radius, ol, om);
}

void vsharp_device(qsm_ctx* ctx, const double* f, const uint8_t* m, const GridDims& d, const double* radii,
                   size_t n_radii, double thr, qsm_progress_fn progress, void* user, double* ol, uint8_t* om) {
  check_finite(thr, "threshold");
  if (n_radii > 0) check_ptr(radii, "radii");
  std::vector<double> r(radii, radii + n_radii);
  for (double v : r) check_finite(v, "radius");
  check_volume_finite(ctx, f, d.n, "field");
  const size_t N = (size_t)d.n;
  if (r.empty()) {  // src/bgremove/vsharp.rs:98-100
    QSM_CUDA(cudaMemsetAsync(ol, 0, N * sizeof(double), ctx->stream));
    QSM_CUDA(cudaMemcpyAsync(om, m, N, cudaMemcpyDeviceToDevice, ctx->stream));
    return;
  }
  if (r.size() == 1) {  // src/bgremove/vsharp.rs:102-108
    if (progress) progress(user, 1, 1);
    sharp_device(ctx, f, m, d, thr, r[0], ol, om);
    return;
  }
  std::stable_sort(r.begin(), r.end(), [](double a, double b) { return a > b; });
  if (ctx->precision == QSM_PRECISION_MIXED) vsharp_impl<float>(ctx, d, f, m, r, thr, progress, user, ol, om);
  else vsharp_impl<double>(ctx, d, f, m, r, thr, progress, user, ol, om);
}

// radii list of VsharpParams (src/bgremove/vsharp.rs:70-82)
std::vector<double> vsharp_radii(const qsm_vsharp_params& p) {
  std::vector<double> radii;
  double r = p.max_radius;
  const double step = p.min_radius;
  if (step > 0.0) {
    while (r >= step) {
      radii.push_back(r);
      r -= step;
    }
  } else if (step <= 0.0 && r >= step) {
    throw QsmError(QSM_ERR_INVALID_ARGUMENT, "min_radius must be > 0 (the radius list would never end)");
  }
  if (radii.empty()) radii.push_back(p.max_radius);
  return radii;
}

// host staging for the two-output functions
template <class Run>
void with_host_io2(qsm_ctx* ctx, const GridDims& d, const double* h_in, const uint8_t* h_mask, double* h_out,
                   uint8_t* h_mask_out, Run run) {
  const size_t N = (size_t)d.n;
  double* din = ws<double>(ctx, "io.in", N);
  uint8_t* dm = ws<uint8_t>(ctx, "io.mask", N);
  double* dout = ws<double>(ctx, "io.out", N);
  uint8_t* dmo = ws<uint8_t>(ctx, "io.mask_out", N);
  h2d(ctx, din, h_in, N * sizeof(double));
  h2d(ctx, dm, h_mask, N);
  run(din, dm, dout, dmo);
  d2h(ctx, h_out, dout, N * sizeof(double));
  d2h(ctx, h_mask_out, dmo, N);
  sync(ctx);
}

}  // namespace qsm

using namespace qsm;

extern "C" {

qsm_status qsm_laplacian_unwrap_device(qsm_ctx* ctx, const double* d_phase, const uint8_t* d_mask,
                                       const qsm_grid* grid, double* d_out) {
  return guarded(ctx, [&] {
    unwrap_device(ctx, d_phase, d_mask, grid, d_out);
    sync(ctx);
  });
}

qsm_status qsm_laplacian_unwrap(qsm_ctx* ctx, const double* phase, const uint8_t* mask, const qsm_grid* grid,
                                double* out) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_io(phase, mask, out);
    const size_t N = (size_t)d.n;
    double* din = ws<double>(ctx, "io.in", N);
    uint8_t* dm = ws<uint8_t>(ctx, "io.mask", N);
    double* dout = ws<double>(ctx, "io.out", N);
    h2d(ctx, din, phase, N * sizeof(double));
    h2d(ctx, dm, mask, N);
    unwrap_device(ctx, din, dm, grid, dout);
    d2h(ctx, out, dout, N * sizeof(double));
    sync(ctx);
  });
}

qsm_status qsm_smv(qsm_ctx* ctx, const double* field, const uint8_t* mask, const qsm_grid* grid, double radius,
                   double* out_local, uint8_t* out_mask) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_io(field, mask, out_local);
    check_ptr(out_mask, "out_mask");
    with_host_io2(ctx, d, field, mask, out_local, out_mask,
                  [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                    smv_device(ctx, f, m, d, radius, o, om);
                  });
  });
}

qsm_status qsm_sharp(qsm_ctx* ctx, const double* field, const uint8_t* mask, const qsm_grid* grid,
                     const qsm_sharp_params* p, double* out_local, uint8_t* out_mask) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_io(field, mask, out_local);
    check_ptr(out_mask, "out_mask");
    check_ptr(p, "params");
    with_host_io2(ctx, d, field, mask, out_local, out_mask,
                  [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                    sharp_device(ctx, f, m, d, p->threshold, p->radius, o, om);
                  });
  });
}

qsm_status qsm_vsharp_with_radii_device(qsm_ctx* ctx, const double* d_field, const uint8_t* d_mask,
                                        const qsm_grid* grid, const double* radii, size_t n_radii, double threshold,
                                        qsm_progress_fn progress, void* user, double* d_out_local,
                                        uint8_t* d_out_mask) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_io(d_field, d_mask, d_out_local);
    check_ptr(d_out_mask, "out_mask");
    vsharp_device(ctx, d_field, d_mask, d, radii, n_radii, threshold, progress, user, d_out_local, d_out_mask);
    sync(ctx);
  });
}

qsm_status qsm_vsharp_with_radii(qsm_ctx* ctx, const double* field, const uint8_t* mask, const qsm_grid* grid,
                                 const double* radii, size_t n_radii, double threshold, qsm_progress_fn progress,
                                 void* user, double* out_local, uint8_t* out_mask) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_io(field, mask, out_local);
    check_ptr(out_mask, "out_mask");
    with_host_io2(ctx, d, field, mask, out_local, out_mask,
                  [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                    vsharp_device(ctx, f, m, d, radii, n_radii, threshold, progress, user, o, om);
                  });
  });
}

qsm_status qsm_vsharp(qsm_ctx* ctx, const double* field, const uint8_t* mask, const qsm_grid* grid,
                      const qsm_vsharp_params* p, qsm_progress_fn progress, void* user, double* out_local,
                      uint8_t* out_mask) {
  return guarded(ctx, [&] {
    check_ptr(p, "params");
    std::vector<double> radii = vsharp_radii(*p);
    GridDims d = check_grid(grid);
    check_io(field, mask, out_local);
    check_ptr(out_mask, "out_mask");
    with_host_io2(ctx, d, field, mask, out_local, out_mask,
                  [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                    vsharp_device(ctx, f, m, d, radii.data(), radii.size(), p->threshold, progress, user, o, om);
                  });
  });
}

void qsm_ismv_params_default(qsm_ismv_params* p) {
  if (!p) return;
  // IsmvParams::default, src/bgremove/ismv.rs:31-35
  p->tol = 1e-6;
  p->max_iter = 50;
  p->radius = 5.0;
}

qsm_status qsm_ismv_device(qsm_ctx* ctx, const double* d_field, const uint8_t* d_mask, const qsm_grid* grid,
                           const qsm_ismv_params* params, qsm_progress_fn progress, void* user, double* d_out_local,
                           uint8_t* d_out_mask) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_io(d_field, d_mask, d_out_local);
    check_ptr(d_out_mask, "out_mask");
    ismv_device(ctx, d_field, d_mask, d, params, progress, user, d_out_local, d_out_mask);
    sync(ctx);
  });
}

qsm_status qsm_ismv(qsm_ctx* ctx, const double* field, const uint8_t* mask, const qsm_grid* grid,
                    const qsm_ismv_params* params, qsm_progress_fn progress, void* user, double* out_local,
                    uint8_t* out_mask) {
  return guarded(ctx, [&] {
    GridDims d = check_grid(grid);
    check_io(field, mask, out_local);
    check_ptr(out_mask, "out_mask");
    with_host_io2(ctx, d, field, mask, out_local, out_mask,
                  [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                    ismv_device(ctx, f, m, d, params, progress, user, o, om);
                  });
  });
}

void qsm_bg_removal_config_default(qsm_bg_removal_config* c) {
  if (!c) return;
  c->algorithm = QSM_BG_VSHARP;
  qsm_vsharp_params_default(&c->vsharp);
  qsm_sharp_params_default(&c->sharp);
  qsm_resharp_params_default(&c->resharp);
  qsm_ismv_params_default(&c->ismv);
}

qsm_status qsm_run_bg_removal(qsm_ctx* ctx, const double* field_ppm, size_t len, const uint8_t* mask,
                              const qsm_scan_metadata* md, const qsm_bg_removal_config* cfg,
                              qsm_progress_fn progress, void* user, double* out_local, uint8_t* out_mask) {
  return guarded(ctx, [&] {
    check_ptr(md, "metadata");
    check_ptr(cfg, "config");
    qsm_grid g{md->nx, md->ny, md->nz, md->vsx, md->vsy, md->vsz};
    const size_t n = md->nx * md->ny * md->nz;
    if (len != n)
      throw QsmError(QSM_ERR_DIMENSION_MISMATCH,
                     "dimension mismatch: expected " + std::to_string(n) + ", got " + std::to_string(len));
    GridDims d = check_grid(&g);
    check_io(field_ppm, mask, out_local);
    check_ptr(out_mask, "out_mask");
    switch (cfg->algorithm) {
      case QSM_BG_VSHARP: {
        std::vector<double> radii = vsharp_radii(cfg->vsharp);
        with_host_io2(ctx, d, field_ppm, mask, out_local, out_mask,
                      [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                        vsharp_device(ctx, f, m, d, radii.data(), radii.size(), cfg->vsharp.threshold, progress,
                                      user, o, om);
                      });
        break;
      }
      case QSM_BG_RESHARP:
        with_host_io2(ctx, d, field_ppm, mask, out_local, out_mask,
                      [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                        resharp_device(ctx, f, m, d, &cfg->resharp, progress, user, o, om);
                      });
        break;
      case QSM_BG_ISMV:
        with_host_io2(ctx, d, field_ppm, mask, out_local, out_mask,
                      [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                        ismv_device(ctx, f, m, d, &cfg->ismv, progress, user, o, om);
                      });
        break;
      case QSM_BG_SHARP:
        with_host_io2(ctx, d, field_ppm, mask, out_local, out_mask,
                      [&](const double* f, const uint8_t* m, double* o, uint8_t* om) {
                        sharp_device(ctx, f, m, d, cfg->sharp.threshold, cfg->sharp.radius, o, om);
                      });
        break;
      default:
        throw QsmError(QSM_ERR_INVALID_CONFIG, "invalid config: background removal algorithm " +
                                                   std::to_string(cfg->algorithm) + " is not provided by this library");
    }
  });
}

}  // extern "C"
