// Compile-time passes without functors (plain Y/Z passes, the multiplier Z pass, X passes
// between real arrays and half spectra) for the lists QSM_FIXED_PLANS_MORE_0..3.  Included by
// the translation units that instantiate one list each (more_*.cu).
//
// Why: outside the compile-time lists these lengths ran the runtime engine (FP64 231-point
// Y pass at 189x231x165: 53 us, X passes of 189: 117 and 181 us); as compile-time
// plans 31 us, and 47 and 43 us.
#pragma once

#include "plain_passes.cuh"

namespace qsm {

#define QSM_MORE_YZ(N_, T_, R0_, R1_, R2_)                                                        \
  if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(AXIS == 1 ? f.py : f.pz) && fx_cols<T>() * T_ <= 1024) \
    return launch_yz_fx<T, DIR, AXIS, FixedPlan<N_, T_, R0_, R1_, R2_>>(ctx, f, 0, src, dst, done);
#define QSM_MORE_ZM(N_, T_, R0_, R1_, R2_)                                                        \
  if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(f.pz) && kZmCols * T_ <= 1024)                     \
    return launch_zm_fx<T, FixedPlan<N_, T_, R0_, R1_, R2_>>(ctx, f, 0, src, dst, mult, done);
#define QSM_MORE_XR(N_, T_, R0_, R1_, R2_)                                                        \
  if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(f.px))                                             \
    return launch_x_r2c_fx<T, FixedPlan<N_, T_, R0_, R1_, R2_>, false>(ctx, f, spec, LoadCast<T, T>{in, f.g.nx}, done);
#define QSM_MORE_XC(N_, T_, R0_, R1_, R2_)                                                        \
  if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(f.px))                                             \
    return launch_x_c2r_fx<T, FixedPlan<N_, T_, R0_, R1_, R2_>, false>(ctx, f, spec, StoreReal<T>{out, f.g.nx, scale}, \
                                                                      done);

#define QSM_MORE_DEFINE(G_)                                                                                       \
  template <typename T, int DIR, int AXIS>                                                                        \
  bool more_yz_##G_(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const int* done) {       \
    QSM_FIXED_PLANS_MORE_##G_(QSM_MORE_YZ) return false;                                                          \
  }                                                                                                               \
  template <typename T>                                                                                           \
  bool more_zm_##G_(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const T* mult,           \
                    const int* done) {                                                                            \
    QSM_FIXED_PLANS_MORE_##G_(QSM_MORE_ZM) return false;                                                          \
  }                                                                                                               \
  template <typename T>                                                                                           \
  bool more_xr_##G_(qsm_ctx* ctx, const Fft3<T>& f, const T* in, cplx_t<T>* spec, const int* done) {               \
    QSM_FIXED_PLANS_MORE_##G_(QSM_MORE_XR) return false;                                                          \
  }                                                                                                               \
  template <typename T>                                                                                           \
  bool more_xc_##G_(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, T* out, T scale, const int* done) {     \
    QSM_FIXED_PLANS_MORE_##G_(QSM_MORE_XC) return false;                                                          \
  }
#define QSM_MORE_INSTANTIATE(G_, T)                                                                               \
  template bool more_yz_##G_<T, -1, 1>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);        \
  template bool more_yz_##G_<T, +1, 1>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);        \
  template bool more_yz_##G_<T, -1, 2>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);        \
  template bool more_yz_##G_<T, +1, 2>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);        \
  template bool more_zm_##G_<T>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const T*, const int*);     \
  template bool more_xr_##G_<T>(qsm_ctx*, const Fft3<T>&, const T*, cplx_t<T>*, const int*);                       \
  template bool more_xc_##G_<T>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, T*, T, const int*);

}  // namespace qsm
