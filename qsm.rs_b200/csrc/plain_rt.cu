// Runtime Stockham engine over plain arrays: the passes of contexts in QSM_PLANS_RUNTIME
// and of lengths outside the compile-time lists and the two-factor form.
#include "launch.cuh"

namespace qsm {

// Tile width for a Y/Z pass: 128-byte rows, halved while the block (P x T threads)
// does not fit on an SM (long axes: many threads, registers, shared memory).
template <typename T, class K> int yz_tile_width(K kernel, int n, int Tn) {
  constexpr int kMinP = 16 / (int)sizeof(cplx_t<T>) > 0 ? 16 / (int)sizeof(cplx_t<T>) : 1;
  for (int P = yz_cols<T>(); P >= kMinP; P /= 2) {
    if (P * Tn > 1024) continue;
    const size_t smem = yz_smem<T>(n, P);
    if (smem > 227u * 1024u) continue;
    ensure_smem(kernel, smem);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, P * Tn, smem) != cudaSuccess) {
      (void)cudaGetLastError();
      continue;
    }
    if (per_sm >= 1) return P;
  }
  throw QsmError(QSM_ERR_UNSUPPORTED_SIZE, "axis of length " + std::to_string(n) + " does not fit one tile");
}

template <typename T, int DIR, int AXIS>
void run_yz_rt(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const int* done) {
  const FftPlan1D& pl = (AXIS == 1) ? f.py : f.pz;
  const cplx_t<T>* tw = (AXIS == 1) ? f.twy : f.twz;
  auto kern = pl.m != pl.n ? k_pass_yz<T, DIR, true> : k_pass_yz<T, DIR, false>;
  const int P = yz_tile_width<T>(kern, pl.m, pl.T);
  const size_t smem = yz_smem<T>(pl.m, P);
  const TileWalk w = tile_walk(f, AXIS, P);
  const unsigned grid = persistent_grid(ctx, kern, P * pl.T, smem, w.ntiles);
  LaunchScope ls(ctx, yz_name(AXIS, DIR));
  kern<<<grid, dim3(P, pl.T), smem, ctx->stream>>>(f.g, pl, w, tw, src, dst, done);
  ls.done();
}

// Tile width of the multiplier Z pass, 0 when no width fits (long axes).
template <typename T, class K> int zm_tile_width(K kernel, int n, int m, int Tn) {
  for (int p = yz_cols<T>(); p >= 16 / (int)sizeof(T); p /= 2) {
    if (p * Tn > 1024 || zm_smem<T>(n, m, p) > 227u * 1024u) continue;
    ensure_smem(kernel, zm_smem<T>(n, m, p));
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, p * Tn, zm_smem<T>(n, m, p)) != cudaSuccess) {
      (void)cudaGetLastError();
      continue;
    }
    if (per_sm >= 1) return p;
  }
  return 0;
}

template <typename T> bool z_mult_fits(const FftPlan1D& pl) {
  auto kern = pl.m != pl.n ? k_z_fused_m<T, true> : k_z_fused_m<T, false>;
  return zm_tile_width<T>(kern, pl.n, pl.m, pl.T) > 0;
}

template <typename T>
bool run_z_fused_m_rt(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const T* mult,
                      const int* done) {
  const FftPlan1D& pl = f.pz;
  auto kern = pl.m != pl.n ? k_z_fused_m<T, true> : k_z_fused_m<T, false>;
  const int P = zm_tile_width<T>(kern, pl.n, pl.m, pl.T);
  if (P == 0) return false;
  const size_t smem = zm_smem<T>(pl.n, pl.m, P);
  const TileWalk w = tile_walk(f, 2, P);
  const unsigned grid = persistent_grid(ctx, kern, P * pl.T, smem, w.ntiles);
  LaunchScope ls(ctx, "fft_z_fused");
  kern<<<grid, dim3(P, pl.T), smem, ctx->stream>>>(f.g, pl, w, f.twz, src, dst, mult, done);
  ls.done();
  return true;
}

template <typename T>
void run_x_r2c_rt(qsm_ctx* ctx, const Fft3<T>& f, const T* in, cplx_t<T>* spec, const int* done) {
  const int Tt = x_block_t(f.px.T);
  const int P = x_pencils_per_block<T>(f.px.T);
  const size_t smem = (size_t)(f.px.m + P * x_rowlen<T>(f.px.m)) * sizeof(cplx_t<T>);
  auto kern = f.px.m != f.px.n ? k_x_r2c<T, true> : k_x_r2c<T, false>;
  ensure_smem(kern, smem);
  LaunchScope ls(ctx, "fft_x_r2c");
  kern<<<(unsigned)x_blocks(f), dim3(Tt, P), smem, ctx->stream>>>(f.g, f.px, f.twx, spec, in, done);
  ls.done();
}

template <typename T>
void run_x_c2r_rt(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, T* out, T scale, const int* done) {
  const int Tt = x_block_t(f.px.T);
  const int P = x_pencils_per_block<T>(f.px.T);
  const size_t smem = (size_t)(f.px.m + P * x_rowlen<T>(f.px.m)) * sizeof(cplx_t<T>);
  auto kern = f.px.m != f.px.n ? k_x_c2r<T, true> : k_x_c2r<T, false>;
  ensure_smem(kern, smem);
  LaunchScope ls(ctx, "fft_x_c2r");
  kern<<<(unsigned)x_blocks(f), dim3(Tt, P), smem, ctx->stream>>>(f.g, f.px, f.twx, spec, out, scale, done);
  ls.done();
}

bool plan_listed(const FftPlan1D& pl) {
#define QSM_LISTED(N_, T_, R0_, R1_, R2_) \
  if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(pl)) return true;
  QSM_FIXED_PLANS(QSM_LISTED)
  QSM_FIXED_PLANS_WIDE(QSM_LISTED)
  QSM_FIXED_PLANS_MORE_0(QSM_LISTED)
  QSM_FIXED_PLANS_MORE_1(QSM_LISTED)
  QSM_FIXED_PLANS_MORE_2(QSM_LISTED)
  QSM_FIXED_PLANS_MORE_3(QSM_LISTED)
#undef QSM_LISTED
  return false;
}

#define QSM_RT(T)                                                                                             \
  template void run_yz_rt<T, -1, 1>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);       \
  template void run_yz_rt<T, +1, 1>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);       \
  template void run_yz_rt<T, -1, 2>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);       \
  template void run_yz_rt<T, +1, 2>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);       \
  template bool z_mult_fits<T>(const FftPlan1D&);                                                             \
  template bool run_z_fused_m_rt<T>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const T*, const int*); \
  template void run_x_r2c_rt<T>(qsm_ctx*, const Fft3<T>&, const T*, cplx_t<T>*, const int*);                   \
  template void run_x_c2r_rt<T>(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, T*, T, const int*);
QSM_RT(float)
QSM_RT(double)
#undef QSM_RT

}  // namespace qsm
