// Y/Z passes without hooks and the multiplier Z pass: launchers of the compile-time kernels
// and their launch-shape tuning (declared in launch.cuh).  Included only by the
// translation units that instantiate them (plain_y32.cu, plain_y64.cu, plain_z32.cu,
// plain_z64.cu), so that no solver file compiles these kernels again.
#pragma once

#include "functors.cuh"

namespace qsm {

// One compile-time Y/Z pass (k_pass_yz_dx, FP a FixedPlan) in launch shape `shape`.
template <typename T, int DIR, int AXIS, class FP>
bool launch_yz_fx(qsm_ctx* ctx, const Fft3<T>& f, int shape, const cplx_t<T>* src, cplx_t<T>* dst, const int* done) {
  const cplx_t<T>* tw = (AXIS == 1) ? f.twy : f.twz;
  auto kern = k_pass_yz_dx<T, DIR, FP, fx_cols<T>()>;
  const size_t smem = dx_smem<T>(FP::n, fx_cols<T>());
  const TileWalk w = tile_walk(f, AXIS, fx_cols<T>(), (shape & kTuneEdge) != 0);
  unsigned grid = 0;
  if (!fx_launch_ok(ctx, kern, fx_cols<T>() * FP::T, smem, &grid, w.ntiles, (shape & kTuneBlockPerTile) != 0,
                    tune_bpsm(shape)))
    return false;
  LaunchScope ls(ctx, yz_name(AXIS, DIR));
  kern<<<grid, dim3(fx_cols<T>(), FP::T), smem, ctx->stream>>>(f.g, w, tw, src, dst, done);
  ls.done();
  return true;
}

// Compile-time Y/Z kernels (fx_cols<T>() columns per tile) for the axis lengths of
// QSM_FIXED_PLANS and QSM_FIXED_PLANS_WIDE; returns false when the plan is not
// one of them.
template <typename T, int DIR, int AXIS>
bool run_yz_fixed(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const int* done) {
  if (!compiled_plans(ctx)) return false;
  {
    const FftPlan1D& pl = (AXIS == 1) ? f.py : f.pz;
#define QSM_TRY_YZ(N_, T_, R0_, R1_, R2_)                                                         \
    if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(pl) && fx_cols<T>() * T_ <= 1024) {                   \
      using FP = FixedPlan<N_, T_, R0_, R1_, R2_>;                                                \
      const int shape = tuned_shape(ctx, yz_tune_key<T>("yz_fx", f, AXIS, DIR));                  \
      return launch_yz_fx<T, DIR, AXIS, FP>(ctx, f, shape, src, dst, done);                       \
    }
    QSM_FIXED_PLANS(QSM_TRY_YZ)
    if (f.forms == PassForms::kBase) return false;
    QSM_FIXED_PLANS_WIDE(QSM_TRY_YZ)
#undef QSM_TRY_YZ
    return false;
  }
}

template <typename T, int DIR, int AXIS>
void run_yz_plain(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const int* done) {
  if (run_yz_fixed<T, DIR, AXIS>(ctx, f, src, dst, done)) return;
  if (axis_listed(ctx, f, AXIS == 1 ? f.py : f.pz)) {
    if (more_yz_0<T, DIR, AXIS>(ctx, f, src, dst, done) || more_yz_1<T, DIR, AXIS>(ctx, f, src, dst, done) ||
        more_yz_2<T, DIR, AXIS>(ctx, f, src, dst, done) || more_yz_3<T, DIR, AXIS>(ctx, f, src, dst, done))
      return;
  }
  if (run_yz_tf<T, DIR, AXIS, false>(ctx, f, src, dst, OpId<T>{}, nullptr, nullptr, done, yz_name(AXIS, DIR))) return;
  run_yz_rt<T, DIR, AXIS>(ctx, f, src, dst, done);
}

// One compile-time multiplier Z pass (k_z_fused_m_fx, FP a FixedPlan) in launch shape
// `shape`.
template <typename T, class FP>
bool launch_zm_fx(qsm_ctx* ctx, const Fft3<T>& f, int shape, const cplx_t<T>* src, cplx_t<T>* dst, const T* mult,
                  const int* done) {
  auto kfx = k_z_fused_m_fx<T, FP, kZmCols>;
  const size_t smem = zm_smem<T>(FP::n, FP::n, kZmCols);
  const TileWalk w = tile_walk(f, 2, kZmCols, (shape & kTuneEdge) != 0);
  unsigned grid = 0;
  if (!fx_launch_ok(ctx, kfx, kZmCols * FP::T, smem, &grid, w.ntiles, (shape & kTuneBlockPerTile) != 0,
                    tune_bpsm(shape)))
    return false;
  LaunchScope ls(ctx, "fft_z_fused");
  kfx<<<grid, dim3(kZmCols, FP::T), smem, ctx->stream>>>(f.g, w, f.twz, src, dst, mult, done);
  ls.done();
  return true;
}

template <typename T, int DIR, int AXIS>
void tune_yz_fixed(qsm_ctx* ctx, const Fft3<T>& f, const std::function<void()>& chain) {
  {
    if (!compiled_plans(ctx)) return;
    const std::string key = yz_tune_key<T>("yz_fx", f, AXIS, DIR);
    if (!autotune_due(ctx, key)) return;
    const FftPlan1D& pl = (AXIS == 1) ? f.py : f.pz;
#define QSM_TUNE_YZ(N_, T_, R0_, R1_, R2_)                                                        \
    if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(pl) && fx_cols<T>() * T_ <= 1024) {                   \
      using FP = FixedPlan<N_, T_, R0_, R1_, R2_>;                                                \
      auto kern = k_pass_yz_dx<T, DIR, FP, fx_cols<T>()>;                                              \
      const size_t smem = dx_smem<T>(FP::n, fx_cols<T>());                                             \
      ensure_smem(kern, smem);                                                                    \
      const auto cands = yz_candidates(f, fx_cols<T>(), kern, fx_cols<T>() * FP::T, smem);                  \
      autotune_pick(ctx, key, cands, [&](int c) { ctx->tuned[key] = TuneRec{c, {}}; chain(); }, 3, 4); \
      return;                                                                                     \
    }
    QSM_FIXED_PLANS(QSM_TUNE_YZ)
    QSM_FIXED_PLANS_WIDE(QSM_TUNE_YZ)
#undef QSM_TUNE_YZ
  }
}

template <typename T>
void tune_z_fused_m(qsm_ctx* ctx, const Fft3<T>& f, const std::function<void()>& chain) {
  {
    if (!compiled_plans(ctx)) return;
    const std::string key = yz_tune_key<T>("zm_fx", f, 2, -1);
    if (!autotune_due(ctx, key)) return;
    const FftPlan1D& pl = f.pz;
#define QSM_TUNE_ZM(N_, T_, R0_, R1_, R2_)                                                        \
    if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(pl) && kZmCols * T_ <= 1024) {                   \
      using FP = FixedPlan<N_, T_, R0_, R1_, R2_>;                                                \
      auto kfx = k_z_fused_m_fx<T, FP, kZmCols>;                                                  \
      const size_t smem = zm_smem<T>(FP::n, FP::n, kZmCols);                                      \
      ensure_smem(kfx, smem);                                                                     \
      const auto cands = yz_candidates(f, kZmCols, kfx, kZmCols * FP::T, smem);                   \
      autotune_pick(ctx, key, cands, [&](int c) { ctx->tuned[key] = TuneRec{c, {}}; chain(); }, 3, 4); \
      return;                                                                                     \
    }
    QSM_FIXED_PLANS(QSM_TUNE_ZM)
    QSM_FIXED_PLANS_WIDE(QSM_TUNE_ZM)
#undef QSM_TUNE_ZM
  }
}

template <typename T>
void run_z_fused_m(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const T* mult,
                   const int* done) {
  if (compiled_plans(ctx)) {
    const FftPlan1D& pl = f.pz;
#define QSM_TRY_ZM(N_, T_, R0_, R1_, R2_)                                                         \
    if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(pl) && kZmCols * T_ <= 1024) {                   \
      using FP = FixedPlan<N_, T_, R0_, R1_, R2_>;                                                \
      const int shape = tuned_shape(ctx, yz_tune_key<T>("zm_fx", f, 2, -1));                      \
      if (launch_zm_fx<T, FP>(ctx, f, shape, src, dst, mult, done)) return;                       \
    }
    QSM_FIXED_PLANS(QSM_TRY_ZM)
    if (f.forms != PassForms::kBase) {
      QSM_FIXED_PLANS_WIDE(QSM_TRY_ZM)
    }
#undef QSM_TRY_ZM
    if (axis_listed(ctx, f, pl) &&
        (more_zm_0<T>(ctx, f, src, dst, mult, done) || more_zm_1<T>(ctx, f, src, dst, mult, done) ||
         more_zm_2<T>(ctx, f, src, dst, mult, done) || more_zm_3<T>(ctx, f, src, dst, mult, done)))
      return;
  }
  if (!tf_usable(ctx, f.tfz, tf_cols<T>()) && run_z_fused_m_rt<T>(ctx, f, src, dst, mult, done)) return;
  run_z_fused<T>(ctx, f, src, dst, OpMultArray<T>{mult}, done, false);
}

template <typename T>
bool x_plain_r2c(qsm_ctx* ctx, const Fft3<T>& f, const T* in, cplx_t<T>* spec, const int* done) {
  return run_x_r2c_fixed<T, true, false>(ctx, f, spec, LoadCast<T, T>{in, f.g.nx}, done) ||
         more_xr_0<T>(ctx, f, in, spec, done) || more_xr_1<T>(ctx, f, in, spec, done) ||
         more_xr_2<T>(ctx, f, in, spec, done) || more_xr_3<T>(ctx, f, in, spec, done);
}
template <typename T>
bool x_plain_c2r(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, T* out, T scale, const int* done) {
  return run_x_c2r_fixed<T, true, false>(ctx, f, spec, StoreReal<T>{out, f.g.nx, scale}, done) ||
         more_xc_0<T>(ctx, f, spec, out, scale, done) || more_xc_1<T>(ctx, f, spec, out, scale, done) ||
         more_xc_2<T>(ctx, f, spec, out, scale, done) || more_xc_3<T>(ctx, f, spec, out, scale, done);
}

}  // namespace qsm
