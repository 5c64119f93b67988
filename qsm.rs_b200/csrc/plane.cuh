// X and Y passes of a small in-plane matrix as one kernel.
//
// A block transforms one z plane in shared memory: rows two at a time (as k_x_r2c_fx /
// k_x_c2r_fx), then its half-spectrum columns, or the other way round, so the spectrum
// crosses L2 once instead of three times and each direction is one launch.  Both transforms
// exchange their stages in place: a row pair's two half-spectrum rows hold its full row,
// and a column its own elements.
//
// Small volumes are bound by launches and by each kernel's chain of latencies, not by
// bytes: TV-ADMM of 250 iterations at 64^3 takes 6.1 ms instead of 7.3 in float and 6.3 instead
// of 7.5 in double, TKD there 53 us instead of 63 to 70 in double.
#pragma once

#include "launch.cuh"

namespace qsm {

constexpr int kPlaneThreads = 256;
// Elements between plane rows: a row pair holds the skewed full row (and begins FX::T modulo
// the banks after the pair before it, so neighbouring pencils do not meet on a bank), a row
// the half spectrum.
template <typename T, class FX> constexpr int plane_pitch() {
  constexpr int need = FX::n + FX::n / x_pad<T, FX>() + 1, M = sizeof(T) == 8 ? 8 : 16;
  constexpr int pair = need + ((FX::T - need) % M + M) % M;
  static_assert(pair % 2 == 0, "a pair of rows");
  return pair / 2 > FX::n / 2 + 1 ? pair / 2 : FX::n / 2 + 1;
}
template <typename T, class FX, class FY> constexpr size_t plane_smem() {
  return (size_t)(x_tw_len<T>(FX::n) + FY::n + FY::n * plane_pitch<T, FX>()) * sizeof(cplx_t<T>);
}
template <int LP> struct SAColumn {
  __device__ __forceinline__ int operator()(int e) const { return e * LP; }
};
template <typename T> constexpr int plane_cols() { return sizeof(T) == 8 ? 8 : 16; }  // 128-byte row segments

template <typename T, class FX, class FY>
__device__ __forceinline__ void plane_tables(cplx_t<T>* twx, cplx_t<T>* twy, const cplx_t<T>* gx, const cplx_t<T>* gy) {
  constexpr bool TWP = x_tw_padded<T>();
  for (int i = threadIdx.x; i < FX::n; i += kPlaneThreads) twx[TWP ? tw_pad(i) : i] = gx[i];
  for (int i = threadIdx.x; i < FY::n; i += kPlaneThreads) twy[i] = gy[i];
}

// Columns of the plane through FY in place; fetch(e, col) and emit(e, col, v).
template <typename T, int DIR, class FX, class FY, class Fetch, class Emit>
__device__ __forceinline__ void plane_columns(cplx_t<T>* plane, const cplx_t<T>* twy, const Fetch& fetch, const Emit& emit) {
  using C = cplx_t<T>;
  constexpr int NXH = FX::n / 2 + 1, P = plane_cols<T>(), G = kPlaneThreads / (P * FY::T), tiles = (NXH + P - 1) / P;
  static_assert(kPlaneThreads % (P * FY::T) == 0, "whole column groups");
  const int px = threadIdx.x % P, t = threadIdx.x / P % FY::T, g = threadIdx.x / (P * FY::T);
  for (int tile0 = 0; tile0 < tiles; tile0 += G) {
    const int col = (tile0 + g) * P + px;
    const bool active = col < NXH;
    C* sp = plane + (active ? col : 0);
    SAColumn<plane_pitch<T, FX>()> sa;
    auto in = [&](int e) -> C { return fetch(e, col); };
    auto out = [&](int e, C v) { emit(e, col, v); };
    FY::template run<DIR>(t, active, sp, sa, twy, in, out);
  }
}

template <typename T, class FX, class FY, class Load>
__global__ void __launch_bounds__(kPlaneThreads)
    k_plane_fwd(Geom g, const cplx_t<T>* __restrict__ twxg, const cplx_t<T>* __restrict__ twyg,
                cplx_t<T>* __restrict__ spec, Load ld, const int* __restrict__ done) {
  using C = cplx_t<T>;
  constexpr int N = FX::n, NY = FY::n, NXH = N / 2 + 1, TX = FX::T, PX = kPlaneThreads / TX, LP = plane_pitch<T, FX>();
  constexpr int CH = (NXH + TX - 1) / TX;
  static_assert(kPlaneThreads % TX == 0 && NY % 2 == 0, "whole pencils of row pairs");
  if (done != nullptr && *done) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* twx = reinterpret_cast<C*>(smraw);
  C* twy = twx + x_tw_len<T>(N);
  C* plane = twy + NY;
  plane_tables<T, FX, FY>(twx, twy, twxg, twyg);
  const int t = threadIdx.x % TX, p = threadIdx.x / TX;
  const int row0 = blockIdx.x * NY;
  for (int q0 = 0; q0 < NY / 2; q0 += PX) {
    const int q = q0 + p;
    const bool active = q < NY / 2;
    C* sp = plane + 2 * (active ? q : 0) * LP;
    SAPadded<x_pad<T, FX>()> sa;
    auto fetch = [&](int e) -> C { return mk<C>(ld(row0 + 2 * q, e), ld(row0 + 2 * q + 1, e)); };
    auto emit = [&](int e, C v) { sp[sa(e)] = v; };
    FX::template run<-1, x_tw_padded<T>()>(t, active, sp, sa, twx, fetch, emit);
    C ra[CH], rb[CH];
    const T half = T(0.5);
    if (active) {
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int k = t + c * TX;
        if (k < NXH) {
          const C zk = sp[sa(k)];
          const C zn = sp[sa(k == 0 ? 0 : N - k)];
          ra[c] = mk<C>((zk.x + zn.x) * half, (zk.y - zn.y) * half);
          rb[c] = mk<C>((zk.y + zn.y) * half, (zn.x - zk.x) * half);
        }
      }
    }
    __syncthreads();
    if (active) {
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int k = t + c * TX;
        if (k < NXH) {
          sp[k] = ra[c];
          sp[LP + k] = rb[c];
        }
      }
    }
  }
  __syncthreads();
  C* out = spec + (long long)row0 * g.pitch;
  plane_columns<T, -1, FX, FY>(
      plane, twy, [&](int e, int col) -> C { return plane[e * LP + col]; },
      [&](int e, int col, C v) { out[(long long)e * g.pitch + col] = v; });
}

template <typename T, class FX, class FY, class Store>
__global__ void __launch_bounds__(kPlaneThreads)
    k_plane_inv(Geom g, const cplx_t<T>* __restrict__ twxg, const cplx_t<T>* __restrict__ twyg,
                const cplx_t<T>* __restrict__ spec, Store st0, const int* __restrict__ done) {
  using C = cplx_t<T>;
  constexpr int N = FX::n, NY = FY::n, TX = FX::T, PX = kPlaneThreads / TX, LP = plane_pitch<T, FX>();
  if (done != nullptr && *done) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* twx = reinterpret_cast<C*>(smraw);
  C* twy = twx + x_tw_len<T>(N);
  C* plane = twy + NY;
  plane_tables<T, FX, FY>(twx, twy, twxg, twyg);
  const int row0 = blockIdx.x * NY;
  const C* in = spec + (long long)row0 * g.pitch;
  plane_columns<T, +1, FX, FY>(
      plane, twy, [&](int e, int col) -> C { return in[(long long)e * g.pitch + col]; },
      [&](int e, int col, C v) { plane[e * LP + col] = v; });
  const int t = threadIdx.x % TX, p = threadIdx.x / TX;
  Store st = st0;
  for (int q0 = 0; q0 < NY / 2; q0 += PX) {
    const int q = q0 + p;
    const bool active = q < NY / 2;
    C* sp = plane + 2 * (active ? q : 0) * LP;
    const C* ra = sp;
    const C* rb = sp + LP;
    SAPadded<x_pad<T, FX>()> sa;
    // as in k_x_c2r_fx
    auto fetch = [&](int e) -> C {
      const bool lo = e <= N / 2;
      const int k = lo ? e : N - e;
      C xa = ra[k], xb = rb[k];
      if (k == 0 || 2 * k == N) {
        xa.y = T(0);
        xb.y = T(0);
      }
      return lo ? mk<C>(xa.x - xb.y, xa.y + xb.x) : mk<C>(xa.x + xb.y, xb.x - xa.y);
    };
    auto emit = [&](int e, C v) {
      st(row0 + 2 * q, e, v.x);
      st(row0 + 2 * q + 1, e, v.y);
    };
    FX::template run<+1, x_tw_padded<T>()>(t, active, sp, sa, twx, fetch, emit);
  }
  st.finish();
}

// In-plane lengths with plane kernels.
#define QSM_PLANE_LENGTHS(X, ...) \
  X(__VA_ARGS__, 64, 4, 16, 4, 1) X(__VA_ARGS__, 96, 8, 16, 6, 1) X(__VA_ARGS__, 128, 8, 16, 8, 1)

// With a 64-point axis the kernel is the faster one from 5 planes to 500.  Between 96 and 128
// points a block's latency is longer and the gain smaller, and it needs a wave that is mostly
// full but not more than one (TV-ADMM in double, two kernels against one: 96x96x48 9.18 and
// 9.73 ms, 96x96x90 13.05 and 12.93, 128x128x80 16.6 and 17.3, 128x128x128 21.7 and 20.3,
// 128x96x160 21.0 and 22.8).
template <typename T> inline bool plane_usable(qsm_ctx* ctx, const Fft3<T>& f) {
  if (!compiled_plans(ctx) || f.forms != PassForms::kAll) return false;
  if (f.g.nx == 64 || f.g.ny == 64) return true;
  return 5LL * f.g.nz >= 3LL * sm_count(ctx) && f.g.nz <= sm_count(ctx);
}

template <typename T, class FX, class FY, class Load>
void launch_plane_fwd(qsm_ctx* ctx, const Fft3<T>& f, cplx_t<T>* spec, const Load& ld, const int* done) {
  auto kern = k_plane_fwd<T, FX, FY, Load>;
  constexpr size_t smem = plane_smem<T, FX, FY>();
  ensure_smem(kern, smem);
  LaunchScope ls(ctx, "fft_xy_fwd");
  kern<<<(unsigned)f.g.nz, kPlaneThreads, smem, ctx->stream>>>(f.g, f.twx, f.twy, spec, ld, done);
  ls.done();
}
template <typename T, class FX, class FY, class Store>
void launch_plane_inv(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, const Store& st, const int* done) {
  auto kern = k_plane_inv<T, FX, FY, Store>;
  constexpr size_t smem = plane_smem<T, FX, FY>();
  ensure_smem(kern, smem);
  LaunchScope ls(ctx, "fft_xy_inv");
  kern<<<(unsigned)f.g.nz, kPlaneThreads, smem, ctx->stream>>>(f.g, f.twx, f.twy, spec, st, done);
  ls.done();
}

#define QSM_PLANE_Y(CALL_, FX_, N_, T_, R0_, R1_, R2_)                            \
  if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(f.py)) {                          \
    using FY = FixedPlan<N_, T_, R0_, R1_, R2_>;                                  \
    CALL_;                                                                        \
    return true;                                                                  \
  }
// The X r2c and forward Y passes; false when the volume does not take the plane kernel.
template <typename T, class FX, class Load>
bool try_plane_fwd(qsm_ctx* ctx, const Fft3<T>& f, cplx_t<T>* spec, const Load& ld, const int* done) {
  if (!FX::matches(f.px)) return false;
  QSM_PLANE_LENGTHS(QSM_PLANE_Y, (launch_plane_fwd<T, FX, FY>(ctx, f, spec, ld, done)), FX)
  return false;
}
template <typename T, class FX, class Store>
bool try_plane_inv(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, const Store& st, const int* done) {
  if (!FX::matches(f.px)) return false;
  QSM_PLANE_LENGTHS(QSM_PLANE_Y, (launch_plane_inv<T, FX, FY>(ctx, f, spec, st, done)), FX)
  return false;
}
#undef QSM_PLANE_Y
#undef QSM_PLANE_LENGTHS

// X r2c then forward Y, and inverse Y then X c2r.
template <typename T, bool W = false, bool DEAD = false, class Load>
void run_xy_fwd(qsm_ctx* ctx, const Fft3<T>& f, cplx_t<T>* spec, const Load& ld, const int* done) {
  if (plane_usable(ctx, f) && (try_plane_fwd<T, FixedPlan<64, 4, 16, 4, 1>>(ctx, f, spec, ld, done) ||
                               try_plane_fwd<T, FixedPlan<96, 8, 16, 6, 1>>(ctx, f, spec, ld, done) ||
                               try_plane_fwd<T, FixedPlan<128, 8, 16, 8, 1>>(ctx, f, spec, ld, done)))
    return;
  run_x_r2c<T, W, DEAD>(ctx, f, spec, ld, done);
  run_yz<T, -1, 1>(ctx, f, spec, spec, OpId<T>{}, done);
}
template <typename T, bool W = false, bool DEAD = false, class Store>
void run_xy_inv(qsm_ctx* ctx, const Fft3<T>& f, cplx_t<T>* spec, const Store& st, const int* done) {
  if (plane_usable(ctx, f) && (try_plane_inv<T, FixedPlan<64, 4, 16, 4, 1>>(ctx, f, spec, st, done) ||
                               try_plane_inv<T, FixedPlan<96, 8, 16, 6, 1>>(ctx, f, spec, st, done) ||
                               try_plane_inv<T, FixedPlan<128, 8, 16, 8, 1>>(ctx, f, spec, st, done)))
    return;
  run_yz<T, +1, 1>(ctx, f, spec, spec, OpId<T>{}, done);
  run_x_c2r<T, W, DEAD>(ctx, f, spec, st, done);
}

}  // namespace qsm
