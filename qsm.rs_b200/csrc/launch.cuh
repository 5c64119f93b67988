// Host launchers for the pass kernels, the per-grid transform bundle and the
// double-precision k-space geometry shared by every spectral multiplier.
#pragma once

#include "internal.h"
#include "passes.cuh"
#include "two_factor.cuh"

namespace qsm {

// Kernels that a grid's passes may take.  kAll: the fastest form of each length.  kBase and
// kBaseWide: the compile-time passes of QSM_FIXED_PLANS (and QSM_FIXED_PLANS_WIDE) and
// otherwise the run-time engine, whatever faster forms are added.  The forms of a length
// differ in their roundings, so a solver whose single-precision map must not move by them
// (restrict_forms) keeps to these.
enum class PassForms { kAll, kBase, kBaseWide };

template <typename T> struct Fft3 {
  Geom g;
  FftPlan1D px, py, pz;
  const cplx_t<T>* twx;
  const cplx_t<T>* twy;
  const cplx_t<T>* twz;
  TwoFactor<T> tfx{}, tfy{}, tfz{};  // two-factor passes of each axis (n = 0: none)
  T* xstage = nullptr;  // buffer of the runtime-engine X passes (null: the context's own)
  T* zstage = nullptr;  // multiplier array of run_z_fused (null: the context's own)
  PassForms forms = PassForms::kAll;
};

template <typename T> void restrict_forms(Fft3<T>& f, PassForms forms) {
  f.forms = forms;
  f.tfx = f.tfy = f.tfz = TwoFactor<T>{};
}

// The two-factor form of a length on axis 0, 1 or 2 (two_factor.cu), n = 0 when it does not
// take one.
template <typename T> TwoFactor<T> make_two_factor(qsm_ctx* ctx, int n, int axis);
// Its radices and blocks, and its host table (tw).
template <typename T> TwoFactor<T> plan_two_factor(int n, int axis);
template <typename T> std::vector<cplx_t<T>> two_factor_table(const TwoFactor<T>& ax);

// Point each Bluestein plan at the chirp and kernel spectrum that follow the stage
// twiddles in its table.
template <typename T> void attach_tables(Fft3<T>& f) {
  f.px.ext = f.px.m != f.px.n ? (const void*)(f.twx + f.px.m) : nullptr;
  f.py.ext = f.py.m != f.py.n ? (const void*)(f.twy + f.py.m) : nullptr;
  f.pz.ext = f.pz.m != f.pz.n ? (const void*)(f.twz + f.pz.m) : nullptr;
}

template <typename T> Fft3<T> make_fft3(qsm_ctx* ctx, const GridDims& d) {
  Fft3<T> f;
  f.g.nx = d.nx;
  f.g.ny = d.ny;
  f.g.nz = d.nz;
  f.g.nxh = d.nx / 2 + 1;
  // rows start on 32-byte boundaries in both precisions, and float and double
  // spectra of one grid share a layout (mixed-precision ops index both)
  f.g.pitch = (f.g.nxh + 3) / 4 * 4;
  f.px = plan_or_throw(d.nx);
  f.py = plan_or_throw(d.ny);
  f.pz = plan_or_throw(d.nz);
  const bool dbl = sizeof(T) == 8;
  f.twx = (const cplx_t<T>*)twiddle_table(ctx, f.px, dbl);
  f.twy = (const cplx_t<T>*)twiddle_table(ctx, f.py, dbl);
  f.twz = (const cplx_t<T>*)twiddle_table(ctx, f.pz, dbl);
  attach_tables(f);
  f.tfx = make_two_factor<T>(ctx, d.nx, 0);
  f.tfy = make_two_factor<T>(ctx, d.ny, 1);
  f.tfz = make_two_factor<T>(ctx, d.nz, 2);
  return f;
}

// Raise a kernel's dynamic shared-memory limit when a launch needs more than the
// default 48 KB (tracked per kernel function and device, under a lock).
void raise_smem_limit(const void* func, int device, size_t bytes);
template <class K> void ensure_smem(K kernel, size_t bytes) {
  if (bytes > 227u * 1024u) throw QsmError(QSM_ERR_UNSUPPORTED_SIZE, "transform tile exceeds shared memory");
  int dev = 0;
  QSM_CUDA(cudaGetDevice(&dev));
  raise_smem_limit(reinterpret_cast<const void*>(kernel), dev, bytes);
}

// False when the context runs every pass on the runtime engine (QSM_PLANS_RUNTIME).
inline bool compiled_plans(const qsm_ctx* ctx) { return ctx->plan_mode == QSM_PLANS_COMPILED; }

inline void after_launch(qsm_ctx* ctx) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw QsmError(QSM_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  ctx->launches++;
}

// Threads per pencil in the X passes: the plan's T rounded up to a divisor of 32
// (T <= 32) or to a multiple of 32, so that a block is a whole number of warps.
inline int x_block_t(int T_) {
  if (T_ <= 32) {
    int b = 1;
    while (b < T_) b <<= 1;
    return b;
  }
  return (T_ + 31) / 32 * 32;
}

template <typename T> inline int x_pencils_per_block(int T_) {
  int P = 256 / x_block_t(T_);
  if (P < 1) P = 1;
  return P;
}

template <typename T> inline long long x_blocks(const Fft3<T>& f) {
  // the X kernels hold a row's elements (<= kFftEmax) and half-spectrum entries
  // (<= kXHalfMax) per thread in fixed register arrays
  if ((f.px.n + f.px.T - 1) / f.px.T > kFftEmax || (f.g.nxh + f.px.T - 1) / f.px.T > kXHalfMax)
    throw QsmError(QSM_ERR_UNSUPPORTED_SIZE, "x length outside the per-thread register budget");
  const int P = x_pencils_per_block<T>(f.px.T);
  const long long npairs = ((long long)f.g.nrows() + 1) / 2;
  return (npairs + P - 1) / P;
}

constexpr int kMaxPersistentBlocks = 4096;

// ------------------------------------------------------- two-factor launches --
// Two buffers of a tile (rows of `stride` elements) and the twiddle table.
template <typename T> inline size_t tf_smem(int n, int stride) { return (2 * (size_t)stride + 1) * n * sizeof(cplx_t<T>); }
// Whether a pass over this axis takes the two-factor kernels (stride: tf_cols, or
// tf_x_stride for X passes).
template <typename T> inline bool tf_usable(const qsm_ctx* ctx, const TwoFactor<T>& ax, int stride) {
  return compiled_plans(ctx) && ax.n > 0 && tf_smem<T>(ax.n, stride) <= 227u * 1024u;
}
template <typename T> inline unsigned tf_x_grid(long long rows) {
  const long long b = (rows + tf_cols<T>() - 1) / tf_cols<T>();
  return (unsigned)(b < kMaxPersistentBlocks ? b : kMaxPersistentBlocks);
}
// Multiplier array as a Z-pass operator (spectrum layout).
template <typename T> struct OpMultArray {
  using C = cplx_t<T>;
  const T* m;
  __device__ __forceinline__ C mid(C v, int, int, int, long long idx) const { return cscale(v, __ldg(m + idx)); }
};

// Doubles that K sums per block of an X pass may fill (grid_sum_last), whichever kernel runs.
template <typename T> inline size_t x_partials(const Fft3<T>& f, int K) {
  // blocks of the runtime engine; a compile-time block holds at least 64 threads of pencils
  // (x_fx_pencils) to the engine's 256, so four times as many is the bound
  const long long b = 4 * x_blocks(f);
  return (size_t)(b > kMaxPersistentBlocks ? b : kMaxPersistentBlocks) * K;
}

int sm_count_of(int device);  // multiprocessor count, cached per device under a lock
inline int sm_count(qsm_ctx* ctx) { return sm_count_of(ctx->device); }

// Threads a block of the compile-time X passes aims at.  Blocks of 128 overlap each other's
// barriers better than blocks of 256 (double: r2c at 189x231x165 47.0 to 42.8 us, c2r 43.5 to
// 38.8 us, at 160x192x160 25.9 to 23.0 and 24.9 to 20.9 us; float c2r at 256x256x176 24.9 to
// 23.4 us, r2c unchanged); at 64 the twiddle table of each block costs that again (43.6 and
// 39.7 us, 23.4 and 21.3 us).
constexpr int kXThreads = 128;
// Pencils per block: as many whole pencils as kXThreads threads hold, halved (down to two
// warps) while the grid is under two blocks per SM: at 64^3 a block of 64 four-thread pencils
// left 32 blocks for 148 SMs.  A pencil's threads are not rounded up to a divisor of a warp
// (as the runtime engine's are): at 21 threads per pencil (length 189) a third of each block
// idled.
template <class FP> inline int x_fx_pencils(qsm_ctx* ctx, long long pencils) {
  int P = FP::T >= kXThreads ? 1 : kXThreads / FP::T;
  while (P > 1 && P / 2 * FP::T >= 64 && (pencils + P - 1) / P < 2LL * sm_count(ctx)) P /= 2;
  return P;
}
inline unsigned x_fx_blocks(long long pencils, int P) { return (unsigned)((pencils + P - 1) / P); }

// One compile-time X pass (k_x_r2c_fx / k_x_c2r_fx, FP a FixedPlan).
template <typename T, class FP, bool DEAD, class Load>
bool launch_x_r2c_fx(qsm_ctx* ctx, const Fft3<T>& f, cplx_t<T>* spec, const Load& ld, const int* done) {
  const int P = x_fx_pencils<FP>(ctx, ((long long)f.g.nrows() + 1) / 2);
  const size_t smem = (size_t)(x_tw_len<T>(FP::n) + P * x_rowlen<T>(FP::n)) * sizeof(cplx_t<T>);
  auto kern = k_x_r2c_fx<T, FP, Load, DEAD>;
  ensure_smem(kern, smem);
  LaunchScope ls(ctx, "fft_x_r2c");
  kern<<<x_fx_blocks(((long long)f.g.nrows() + 1) / 2, P), dim3(FP::T, P), smem, ctx->stream>>>(f.g, f.twx, spec, ld, done);
  ls.done();
  return true;
}
template <typename T, class FP, bool DEAD, class Store>
bool launch_x_c2r_fx(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, const Store& st, const int* done) {
  const int P = x_fx_pencils<FP>(ctx, ((long long)f.g.nrows() + 1) / 2);
  const size_t smem = (size_t)(x_tw_len<T>(FP::n) + P * x_rowlen<T>(FP::n)) * sizeof(cplx_t<T>);
  auto kern = k_x_c2r_fx<T, FP, Store, DEAD>;
  ensure_smem(kern, smem);
  LaunchScope ls(ctx, "fft_x_c2r");
  kern<<<x_fx_blocks(((long long)f.g.nrows() + 1) / 2, P), dim3(FP::T, P), smem, ctx->stream>>>(f.g, f.twx, spec, st, done);
  ls.done();
  return true;
}

// Compile-time X kernels with the functor inside: in float for the lengths of
// QSM_FIXED_PLANS, and with W in both precisions for QSM_FIXED_PLANS_WIDE too; false when
// the plan is not one of them.
template <typename T, bool W, bool DEAD, class Load>
bool run_x_r2c_fixed(qsm_ctx* ctx, const Fft3<T>& f, cplx_t<T>* spec, const Load& ld, const int* done) {
  if (!compiled_plans(ctx)) return false;
#define QSM_TRY_XR(N_, T_, R0_, R1_, R2_)                                                          \
  if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(f.px))                                             \
    return launch_x_r2c_fx<T, FixedPlan<N_, T_, R0_, R1_, R2_>, DEAD>(ctx, f, spec, ld, done);
  if constexpr (std::is_same<T, float>::value || W) {
    QSM_FIXED_PLANS(QSM_TRY_XR)
  }
  if constexpr (W) {
    QSM_FIXED_PLANS_WIDE(QSM_TRY_XR)
  }
#undef QSM_TRY_XR
  return false;
}

template <typename T, bool W, bool DEAD, class Store>
bool run_x_c2r_fixed(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, const Store& st, const int* done) {
  if (!compiled_plans(ctx)) return false;
#define QSM_TRY_XC(N_, T_, R0_, R1_, R2_)                                                          \
  if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(f.px))                                             \
    return launch_x_c2r_fx<T, FixedPlan<N_, T_, R0_, R1_, R2_>, DEAD>(ctx, f, spec, st, done);
  if constexpr (std::is_same<T, float>::value || W) {
    QSM_FIXED_PLANS(QSM_TRY_XC)
  }
  if constexpr (W) {
    QSM_FIXED_PLANS_WIDE(QSM_TRY_XC)
  }
#undef QSM_TRY_XC
  return false;
}

// Compile-time X passes between a real array and a half spectrum for every listed length
// (plain_x32.cu, plain_x64.cu, more_*.cu); axis_listed says whether the axis is one of them.
template <typename T>
bool x_plain_r2c(qsm_ctx* ctx, const Fft3<T>& f, const T* in, cplx_t<T>* spec, const int* done);
template <typename T>
bool x_plain_c2r(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, T* out, T scale, const int* done);
bool plan_listed(const FftPlan1D& pl);
// Whether the axis takes the compile-time passes of some list.
template <typename T> inline bool axis_listed(const qsm_ctx* ctx, const Fft3<T>& f, const FftPlan1D& pl) {
  return compiled_plans(ctx) && f.forms == PassForms::kAll && plan_listed(pl);
}
// Loaders and stores that are just such arrays (functors.cuh).
template <typename T, class Load> struct PlainLoad : std::false_type {};
template <typename T, class Store> struct PlainStore : std::false_type {};

// Runtime-engine X passes over plain arrays (real rows and half spectra),
// compiled once (plain_rt.cu).
template <typename T>
void run_x_r2c_rt(qsm_ctx* ctx, const Fft3<T>& f, const T* in, cplx_t<T>* spec, const int* done);
template <typename T>
void run_x_c2r_rt(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, T* out, T scale, const int* done);

// Buffers of the runtime-engine X passes, between the caller's functor and the engine.
template <typename T> T* x_stage(qsm_ctx* ctx, const Fft3<T>& f) {
  return f.xstage ? f.xstage : ws_scratch<T>(ctx, sizeof(T) == 4 ? "x.stage32" : "x.stage64", (size_t)f.g.nvox());
}
template <typename T> cplx_t<T>* x_stage_c(qsm_ctx* ctx, const Fft3<T>& f) {
  return ws_scratch<cplx_t<T>>(ctx, sizeof(T) == 4 ? "x.stagec32" : "x.stagec64", (size_t)f.g.hsize());
}
// A listed length with a functor that no compile-time kernel carries: the functor as a pass
// of its own around the plain kernel, except in small volumes, where the launch costs more
// than the two-factor kernel (functor inside) loses.  TKD in double, functor inside against
// its own pass: 49.8 and 55.3 us at 64x48x40, 68.0 and 69.3 at 96x90x88, 78.1 and 75.4 at
// 100x100x110, 85.1 and 80.6 at 160x96x90, 192 and 167 at 256x160x120; iSMV, 50 iterations:
// 2.12 and 2.08 ms at 72x64x60, 4.09 and 3.82 at 100x100x110, 13.8 and 11.7 at 256x160x120.
template <typename T> inline bool x_use_stage(const Fft3<T>& f) { return f.g.nvox() > (1LL << 20); }
// Persistent grid: as many CTAs as fit on the device at once, capped by the work.
template <class K> unsigned persistent_grid(qsm_ctx* ctx, K kernel, int threads, size_t smem, long long work) {
  int per_sm = 0;
  QSM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  if (per_sm < 1) throw QsmError(QSM_ERR_UNSUPPORTED_SIZE, "transform tile does not fit on an SM");
  long long g = (long long)per_sm * sm_count(ctx);
  if (g > work) g = work;
  if (g < 1) g = 1;
  return (unsigned)g;
}

// Grid of 256-thread blocks of an elementwise kernel over n elements: one full wave.  A grid
// fixed at 16 blocks per SM left the last of three to four waves of the register-heavy
// kernels mostly idle (48 registers: five blocks per SM, adjoint update at 160x192x160 111.6
// us, 92.3 in one wave).
template <class K> unsigned wave_grid(qsm_ctx* ctx, K kernel, long long n) {
  return persistent_grid(ctx, kernel, 256, 0, (n + 255) / 256);
}

// One full wave: with 47 registers five blocks fit on an SM, and a fixed eight per SM ran
// them in two waves, the second mostly idle.
template <class K> unsigned x_rows_grid(qsm_ctx* ctx, K kernel, const Geom& g) {
  return persistent_grid(ctx, kernel, 256, 0, ((long long)g.nrows() + 7) / 8);
}

// DEAD (compile-time kernels only): the pass reads ld's rows for the last time and drops
// their L2 lines (k_x_r2c_fx); ld then provides row_begin.
template <typename T, bool W = false, bool DEAD = false, class Load>
void run_x_r2c(qsm_ctx* ctx, const Fft3<T>& f, cplx_t<T>* spec, const Load& ld, const int* done) {
  if (run_x_r2c_fixed<T, W, DEAD>(ctx, f, spec, ld, done)) return;
  const bool listed = axis_listed(ctx, f, f.px);
  if constexpr (PlainLoad<T, Load>::value) {
    if (listed) {
      x_plain_r2c<T>(ctx, f, ld.p, spec, done);
      return;
    }
  }
  if (tf_usable(ctx, f.tfx, tf_x_stride<T>()) && !(listed && x_use_stage(f))) {
    const size_t smem = tf_smem<T>(f.tfx.n, tf_x_stride<T>());
    auto kern = k_x_r2c_tf<T, Load>;
    ensure_smem(kern, smem);
    LaunchScope ls(ctx, "fft_x_r2c");
    kern<<<tf_x_grid<T>(((long long)f.g.nrows() + 1) / 2), kTfThreads, smem, ctx->stream>>>(f.g, f.tfx, spec, ld, done);
    ls.done();
    return;
  }
  if constexpr (PlainLoad<T, Load>::value) {
    run_x_r2c_rt<T>(ctx, f, ld.p, spec, done);
    return;
  }
  T* st = x_stage(ctx, f);
  {
    LaunchScope ls(ctx, "x_load");
    k_x_load<T, T, Load><<<x_rows_grid(ctx, k_x_load<T, T, Load>, f.g), 256, 0, ctx->stream>>>(f.g, f.g.nx, ld, st, done);
    ls.done();
  }
  if (listed) x_plain_r2c<T>(ctx, f, st, spec, done);
  else run_x_r2c_rt<T>(ctx, f, st, spec, done);
}

// DEAD (compile-time kernels only): the pass reads the half spectrum for the last time and
// drops its L2 lines (k_x_c2r_fx).
template <typename T, bool W = false, bool DEAD = false, class Store>
void run_x_c2r(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* spec, const Store& st, const int* done) {
  if (run_x_c2r_fixed<T, W, DEAD>(ctx, f, spec, st, done)) return;
  const bool listed = axis_listed(ctx, f, f.px);
  if constexpr (PlainStore<T, Store>::value) {
    if (listed) {
      x_plain_c2r<T>(ctx, f, spec, st.out, st.scale, done);
      return;
    }
  }
  if (tf_usable(ctx, f.tfx, tf_x_stride<T>()) && !(listed && x_use_stage(f))) {
    const size_t smem = tf_smem<T>(f.tfx.n, tf_x_stride<T>());
    auto kern = k_x_c2r_tf<T, Store>;
    ensure_smem(kern, smem);
    LaunchScope ls(ctx, "fft_x_c2r");
    kern<<<tf_x_grid<T>(((long long)f.g.nrows() + 1) / 2), kTfThreads, smem, ctx->stream>>>(f.g, f.tfx, spec, st, done);
    ls.done();
    return;
  }
  if constexpr (PlainStore<T, Store>::value) {
    run_x_c2r_rt<T>(ctx, f, spec, st.out, st.scale, done);
    return;
  }
  T* buf = x_stage(ctx, f);
  if (listed) x_plain_c2r<T>(ctx, f, spec, buf, T(1), done);
  else run_x_c2r_rt<T>(ctx, f, spec, buf, T(1), done);
  LaunchScope ls(ctx, "x_store");
  k_x_store<T, T, Store><<<x_rows_grid(ctx, k_x_store<T, T, Store>, f.g), 256, 0, ctx->stream>>>(f.g, f.g.nx, buf, st, done);
  ls.done();
}

template <typename T> inline int yz_cols() { return sizeof(T) == 4 ? 16 : 8; }

// Tile walk of a Y (axis 1) or Z (axis 2) pass with P-column tiles.  edge: walk a
// narrow column remainder (at most P/4 columns) as edge tiles (TileWalk); only the
// compile-time kernels read edge tiles.
template <typename T> TileWalk tile_walk(const Fft3<T>& f, int axis, int P, bool edge = false) {
  TileWalk w;
  w.ntx = (f.g.nxh + P - 1) / P;
  w.nouter = axis == 1 ? f.g.nz : f.g.ny;
  if (axis == 1) {  // Y: outer = z
    w.ostride = (long long)f.g.pitch * f.g.ny;
    w.estride = f.g.pitch;
  } else {  // Z: outer = y
    w.ostride = f.g.pitch;
    w.estride = (long long)f.g.pitch * f.g.ny;
  }
  const int rem = f.g.nxh % P;
  w.nedge = 0;
  w.col_edge = f.g.nxh;
  if (edge && rem > 0 && 4 * rem <= P) {
    w.ntx = f.g.nxh / P;
    w.nedge = rem;
    w.col_edge = w.ntx * P;
  }
  w.nmain = w.ntx * w.nouter;
  w.ntiles = w.nmain + w.nedge * ((w.nouter + P - 1) / P);
  return w;
}
// True when tile_walk(..., edge = true) has edge tiles.
template <typename T> bool has_edge_tiles(const Fft3<T>& f, int P) {
  const int rem = f.g.nxh % P;
  return rem > 0 && 4 * rem <= P;
}

// shared memory of the direct-fetch kernels: twiddles + one tile (the stage exchange)
template <typename T> inline size_t dx_smem(int n, int P) {
  return (size_t)(((n + 7) & ~7) + (size_t)n * P) * sizeof(cplx_t<T>);
}

template <typename T> inline size_t yz_smem(int n, int P) {
  return (size_t)(((n + 7) & ~7) + 2 * (size_t)n * P) * sizeof(cplx_t<T>);
}

// shared memory of the multiplier Z pass: n multiplier rows, m tile-buffer rows (m = n except
// for Bluestein plans)
template <typename T> inline size_t zm_smem(int n, int m, int P) {
  return yz_smem<T>(m, P) + 2 * (((size_t)n * P + 3) & ~(size_t)3) * sizeof(T);
}

// Columns per tile of the compile-time Y/Z passes: 128-byte tile rows (16 float or 8
// double complex values).
template <typename T> constexpr int fx_cols() { return sizeof(T) == 4 ? 16 : 8; }
constexpr int kZmCols = 8;  // columns per tile of the fused Z pass

// ----------------------------------------------------------------- autotuner --
// Launch shapes of the compile-time Y/Z passes, as fields of a candidate number:
//   kTuneEdge         edge tiles for a narrow column remainder (TileWalk)
//   kTuneBlockPerTile one block per tile, scheduled by the hardware, instead of a
//                     persistent grid of resident blocks walking the tiles
//   bits 2..5         persistent grid: resident blocks per SM (0 = as many as fit)
// Every shape runs the same arithmetic on every column, so results do not depend on the
// choice.  The choice is made per context by timing each candidate once on scratch
// buffers (autotune_pick) and cached under a key naming the pass and its geometry;
// launches whose key is not cached use shape 0, the persistent grid without edge tiles.
constexpr int kTuneEdge = 1, kTuneBlockPerTile = 2, kTuneBpsmShift = 2;  // kTuneMaxShape: internal.h
inline int tune_bpsm(int shape) { return (shape >> kTuneBpsmShift) & 15; }
bool stream_capturing(qsm_ctx* ctx);
// Time launch(c) for every candidate c on ctx->stream (after one warm-up launch each,
// `rounds` rounds of `reps` launches; the best round counts) and cache the fastest under key.
void autotune_pick(qsm_ctx* ctx, const std::string& key, const std::vector<int>& cands,
                   const std::function<void(int)>& launch, int rounds = 3, int reps = 5);
inline int tuned_shape(const qsm_ctx* ctx, const std::string& key) {
  if (ctx->forced_shape >= 0) return ctx->forced_shape;
  if (!ctx->autotune) return 0;
  auto it = ctx->tuned.find(key);
  return it == ctx->tuned.end() ? 0 : it->second.choice;
}
// Whether a tuning run for key should happen now (autotuner on, key not cached, stream
// not capturing).
inline bool autotune_due(qsm_ctx* ctx, const std::string& key) {
  return ctx->autotune && ctx->forced_shape < 0 && ctx->tuned.find(key) == ctx->tuned.end() && !stream_capturing(ctx);
}
template <typename T> std::string yz_tune_key(const char* pass, const Fft3<T>& f, int axis, int dir) {
  return std::string(pass) + (axis == 1 ? ":y" : ":z") + (dir < 0 ? "-" : "+") + ":" + std::to_string(f.g.nx) +
         "x" + std::to_string(f.g.ny) + "x" + std::to_string(f.g.nz) + (sizeof(T) == 4 ? ":f32" : ":f64");
}
// Candidates: persistent grids of the occupancy limit and of one block per SM fewer,
// and one block per tile, each with and without edge tiles where the grid has them.
template <typename T, class K>
std::vector<int> yz_candidates(const Fft3<T>& f, int P, K kern, int threads, size_t smem) {
  int per_sm = 0;
  QSM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
  std::vector<int> base{0, kTuneBlockPerTile};
  if (per_sm >= 2 && per_sm - 1 <= 15) base.push_back((per_sm - 1) << kTuneBpsmShift);
  std::vector<int> c = base;
  if (has_edge_tiles(f, P))
    for (int b : base) c.push_back(b | kTuneEdge);
  return c;
}

// Grid of a compile-time Y/Z pass over `work` tiles: resident blocks (persistent) or one
// block per tile; false when the block does not fit on an SM.
template <class K>
bool fx_launch_ok(qsm_ctx* ctx, K kern, int threads, size_t smem, unsigned* grid, long long work,
                  bool per_tile = false, int bpsm = 0) {
  if (smem > 227u * 1024u) return false;
  ensure_smem(kern, smem);
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  if (per_sm < 1) return false;
  if (bpsm > 0 && bpsm < per_sm) per_sm = bpsm;
  long long g = per_tile ? work : (long long)per_sm * sm_count(ctx);
  if (g > work) g = work;
  *grid = (unsigned)(g < 1 ? 1 : g);
  return true;
}

// One compile-time operator pass: k_pass_yz_dx_old when the op's epilogue reads a second
// array (ACC only), k_pass_yz_st_op when its pre hook wants a staged tile, else
// k_pass_yz_dx_op.  False when the block does not fit.
template <typename T, int DIR, int AXIS, bool ACC, class FP, class Op>
bool launch_yz_op_fx(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* tw, const cplx_t<T>* src, cplx_t<T>* dst,
                     const Op& op, double* partials, unsigned* counter, const int* done, const char* name) {
  constexpr int P = fx_cols<T>();
  const TileWalk w = tile_walk(f, AXIS, P);
  unsigned grid = 0;
  if constexpr (ACC && ReadsOld<Op>::value) {
    auto kern = k_pass_yz_dx_old<T, DIR, AXIS, FP, P, Op>;
    const size_t smem = dx_smem<T>(FP::n, P) + (size_t)FP::n * P * sizeof(cplx_t<T>);
    if (!fx_launch_ok(ctx, kern, P * FP::T, smem, &grid, w.ntiles)) return false;
    if (grid > (unsigned)kMaxPersistentBlocks) return false;
    LaunchScope ls(ctx, name);
    kern<<<grid, dim3(P, FP::T), smem, ctx->stream>>>(f.g, w, tw, src, dst, op, partials, counter, done);
    ls.done();
  } else {
    auto kern = k_pass_yz_dx_op<T, DIR, AXIS, FP, P, Op, ACC>;
    const size_t smem = dx_smem<T>(FP::n, P);
    if (!fx_launch_ok(ctx, kern, P * FP::T, smem, &grid, w.ntiles)) return false;
    if (ACC && grid > (unsigned)kMaxPersistentBlocks) return false;
    LaunchScope ls(ctx, name);
    kern<<<grid, dim3(P, FP::T), smem, ctx->stream>>>(f.g, w, tw, src, dst, op, partials, counter, done);
    ls.done();
  }
  return true;
}

// Compile-time Y/Z pass that carries an operator (k_pass_yz_dx_op), lengths of
// QSM_FIXED_PLANS; ACC as in run_yz_acc.  Returns false when the plan is not one of them.
template <typename T, int DIR, int AXIS, bool ACC, class Op>
bool run_yz_op_fixed(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const Op& op,
                     double* partials, unsigned* counter, const int* done, const char* name) {
  if (!compiled_plans(ctx)) return false;
  {
    const FftPlan1D& pl = (AXIS == 1) ? f.py : f.pz;
    const cplx_t<T>* tw = (AXIS == 1) ? f.twy : f.twz;
#define QSM_TRY_YZO(N_, T_, R0_, R1_, R2_)                                                         \
    if (FixedPlan<N_, T_, R0_, R1_, R2_>::matches(pl) && fx_cols<T>() * T_ <= 1024)                \
      return launch_yz_op_fx<T, DIR, AXIS, ACC, FixedPlan<N_, T_, R0_, R1_, R2_>>(ctx, f, tw, src, dst, op, partials, \
                                                                                counter, done, name);
    QSM_FIXED_PLANS(QSM_TRY_YZO)
#undef QSM_TRY_YZO
    return false;
  }
}

// Two-factor Y/Z pass; false when the axis does not use it.
template <typename T, int DIR, int AXIS, bool ACC, class Op>
bool run_yz_tf(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const Op& op, double* partials,
               unsigned* counter, const int* done, const char* name) {
  const TwoFactor<T>& ax = AXIS == 1 ? f.tfy : f.tfz;
  if (!tf_usable(ctx, ax, tf_cols<T>())) return false;
  const size_t smem = tf_smem<T>(ax.n, tf_cols<T>());
  auto kern = k_pass_yz_tf<T, DIR, AXIS, Op, ACC>;
  ensure_smem(kern, smem);
  const TileWalk w = tile_walk(f, AXIS, tf_cols<T>());
  unsigned grid = persistent_grid(ctx, kern, kTfThreads, smem, w.ntiles);
  if (ACC && grid > (unsigned)kMaxPersistentBlocks) grid = kMaxPersistentBlocks;
  LaunchScope ls(ctx, name);
  kern<<<grid, kTfThreads, smem, ctx->stream>>>(f.g, ax, w, src, dst, op, partials, counter, done);
  ls.done();
  return true;
}
// Two-factor fused Z pass; false when the axis does not use it.
template <typename T, class Op>
bool run_z_fused_tf(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const Op& op,
                    const int* done) {
  if (!tf_usable(ctx, f.tfz, tf_cols<T>())) return false;
  const size_t smem = tf_smem<T>(f.tfz.n, tf_cols<T>());
  auto kern = k_z_fused_tf<T, Op>;
  ensure_smem(kern, smem);
  const TileWalk w = tile_walk(f, 2, tf_cols<T>());
  const unsigned grid = persistent_grid(ctx, kern, kTfThreads, smem, w.ntiles);
  LaunchScope ls(ctx, "fft_z_fused");
  kern<<<grid, kTfThreads, smem, ctx->stream>>>(f.g, f.tfz, w, src, dst, op, done);
  ls.done();
  return true;
}

// Plain passes (plain_y*.cu, plain_z*.cu, plain_rt.cu: instantiated once): the compile-time
// kernel for the lengths of QSM_FIXED_PLANS and QSM_FIXED_PLANS_WIDE, the two-factor
// kernel, or the runtime engine.
template <typename T, int DIR, int AXIS>
void run_yz_plain(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const int* done);
template <typename T, int DIR, int AXIS>
void run_yz_rt(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const int* done);
// The run-time engine's multiplier Z pass in one kernel; false when no tile of it fits an SM,
// which z_mult_fits says beforehand.
template <typename T> bool z_mult_fits(const FftPlan1D& pl);
template <typename T>
bool run_z_fused_m_rt(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const T* mult,
                      const int* done);
// Z forward -> precomputed real multiplier array (spectrum layout) -> Z inverse.
template <typename T>
void run_z_fused_m(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const T* mult,
                   const int* done);

// Tune the launch shape of the compile-time Y/Z pass (DIR, AXIS) and of the multiplier Z
// pass for grid f: each candidate is timed inside `chain`, the solver's own sequence of
// passes (which looks the shape up under the same key), so that it is judged where it runs:
// after the pass that fills the L2-resident spectrum, not back to back with itself.  No-op
// when the lengths have no compile-time pass, the shapes are cached, the autotuner is off or
// the stream is capturing.
template <typename T, int DIR, int AXIS>
void tune_yz_fixed(qsm_ctx* ctx, const Fft3<T>& f, const std::function<void()>& chain);
template <typename T> void tune_z_fused_m(qsm_ctx* ctx, const Fft3<T>& f, const std::function<void()>& chain);

#define QSM_MORE_DECLARE(G_)                                                                                      \
  template <typename T, int DIR, int AXIS>                                                                        \
  bool more_yz_##G_(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const int*);                           \
  template <typename T>                                                                                           \
  bool more_zm_##G_(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, cplx_t<T>*, const T*, const int*);                 \
  template <typename T> bool more_xr_##G_(qsm_ctx*, const Fft3<T>&, const T*, cplx_t<T>*, const int*);             \
  template <typename T> bool more_xc_##G_(qsm_ctx*, const Fft3<T>&, const cplx_t<T>*, T*, T, const int*);
QSM_MORE_DECLARE(0)
QSM_MORE_DECLARE(1)
QSM_MORE_DECLARE(2)
QSM_MORE_DECLARE(3)
#undef QSM_MORE_DECLARE

inline const char* yz_name(int axis, int dir) {
  return axis == 1 ? (dir < 0 ? "fft_y_fwd" : "fft_y_inv") : (dir < 0 ? "fft_z_fwd" : "fft_z_inv");
}
inline unsigned spec_grid(const Geom& g) { return (unsigned)(g.nrows() < 2368 ? g.nrows() : 2368); }

// The hooks of a pass as elementwise passes (those that do something) around the plain
// transform.
template <typename T, int DIR, int AXIS, class Op>
void run_yz_hooks(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const Op& op, const int* done) {
  if constexpr (!NoPre<Op>::value) {
    LaunchScope ls(ctx, "yz_pre");
    k_spec_pre<T, Op><<<spec_grid(f.g), 128, 0, ctx->stream>>>(f.g, src, dst, op, done);
    ls.done();
    src = dst;
  }
  run_yz_plain<T, DIR, AXIS>(ctx, f, src, dst, done);
  if constexpr (!NoPost<Op>::value) {
    LaunchScope ls(ctx, "yz_post");
    k_spec_post<T, Op><<<spec_grid(f.g), 128, 0, ctx->stream>>>(f.g, dst, op, done);
    ls.done();
  }
}

// AXIS 1 = y, 2 = z; DIR -1 forward, +1 inverse.  Passes with hooks take the compile-time
// operator kernel when W (QSM_FIXED_PLANS); at other listed lengths the hooks run as passes
// of their own around the compile-time transform, and elsewhere inside the two-factor kernel.
template <typename T, int DIR, int AXIS, bool W = false, class Op>
void run_yz(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const Op& op, const int* done) {
  if constexpr (IsPlainOp<Op>::value) {
    run_yz_plain<T, DIR, AXIS>(ctx, f, src, dst, done);
  } else {
    if constexpr (W) {
      if (run_yz_op_fixed<T, DIR, AXIS, false>(ctx, f, src, dst, op, nullptr, nullptr, done, yz_name(AXIS, DIR))) return;
    }
    const bool listed = axis_listed(ctx, f, AXIS == 1 ? f.py : f.pz);
    if (!listed && run_yz_tf<T, DIR, AXIS, false>(ctx, f, src, dst, op, nullptr, nullptr, done, yz_name(AXIS, DIR))) return;
    run_yz_hooks<T, DIR, AXIS>(ctx, f, src, dst, op, done);
  }
}

// Y/Z pass with an FP64 accumulation in its post hook (as k_pass_yz_tf, ACC).  `partials`
// holds at least kMaxPersistentBlocks doubles; `counter` is 0 between launches.
template <typename T, int DIR, int AXIS, bool W = false, class Op>
void run_yz_acc(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const Op& op,
                double* partials, unsigned* counter, const int* done, const char* name) {
  if constexpr (W) {
    if (run_yz_op_fixed<T, DIR, AXIS, true>(ctx, f, src, dst, op, partials, counter, done, name)) return;
  }
  const bool listed = axis_listed(ctx, f, AXIS == 1 ? f.py : f.pz);
  if (!listed && run_yz_tf<T, DIR, AXIS, true>(ctx, f, src, dst, op, partials, counter, done, name)) return;
  // dst may be the op's old vector: the transform goes through a buffer of its own
  cplx_t<T>* t = x_stage_c(ctx, f);
  if constexpr (!NoPre<Op>::value) {
    LaunchScope ls(ctx, "yz_pre");
    k_spec_pre<T, Op><<<spec_grid(f.g), 128, 0, ctx->stream>>>(f.g, src, t, op, done);
    ls.done();
    src = t;
  }
  run_yz_plain<T, DIR, AXIS>(ctx, f, src, t, done);
  LaunchScope ls(ctx, name);
  k_spec_post_acc<T, Op><<<spec_grid(f.g), 128, 0, ctx->stream>>>(f.g, t, dst, op, partials, counter, done);
  ls.done();
}

// The real multiplier of op.mid as an array (spectrum layout).
template <typename T, class Op>
void spec_multiplier(qsm_ctx* ctx, const Fft3<T>& f, const Op& op, T* out, const int* done) {
  LaunchScope ls(ctx, "z_mult");
  k_spec_mult<T, Op><<<dim3((unsigned)f.g.ny, (unsigned)f.g.nz), 128, 0, ctx->stream>>>(f.g, op, out, done);
  ls.done();
}

// Z forward -> op.mid -> Z inverse, op.mid a real multiplier (v -> m v).  The two-factor kernel
// evaluates it in the pass; other lengths evaluate it once into an array for the multiplier
// pass (`array` false where no buffer may be allocated).
template <typename T, class Op>
void run_z_fused(qsm_ctx* ctx, const Fft3<T>& f, const cplx_t<T>* src, cplx_t<T>* dst, const Op& op,
                 const int* done, bool array = true) {
  if (array && (axis_listed(ctx, f, f.pz) || !tf_usable(ctx, f.tfz, tf_cols<T>()))) {
    T* m = f.zstage ? f.zstage : ws_scratch<T>(ctx, sizeof(T) == 4 ? "z.mult32" : "z.mult64", (size_t)f.g.hsize());
    spec_multiplier<T>(ctx, f, op, m, done);
    if (f.forms == PassForms::kAll) {
      run_z_fused_m<T>(ctx, f, src, dst, m, done);
      return;
    }
    if (run_z_fused_m_rt<T>(ctx, f, src, dst, m, done)) return;
  }
  if (run_z_fused_tf(ctx, f, src, dst, op, done)) return;
  const bool rt = f.forms != PassForms::kAll;
  if (rt) run_yz_rt<T, -1, 2>(ctx, f, src, dst, done);
  else run_yz_plain<T, -1, 2>(ctx, f, src, dst, done);
  {
    LaunchScope ls(ctx, "z_mid");
    k_spec_mid<T, Op><<<spec_grid(f.g), 128, 0, ctx->stream>>>(f.g, dst, op, done);
    ls.done();
  }
  if (rt) run_yz_rt<T, +1, 2>(ctx, f, dst, dst, done);
  else run_yz_plain<T, +1, 2>(ctx, f, dst, dst, done);
}

// ---------------------------------------------------------------------------
// k-space geometry in double: fftfreq per axis (src/fft.rs:544-566), per-axis
// eigenvalues of the negative 7-point Laplacian (the FFT of
// laplacian_kernel(negative=true), src/kernels/laplacian.rs:20-61, which is a sum of
// per-axis terms), the Poisson eigenvalues of the unwrapping solver
// (src/unwrap/laplacian.rs:91-105), and the normalised B0 direction.
// ---------------------------------------------------------------------------
template <typename S> struct KSpaceT {
  const S* fx;
  const S* fy;
  const S* fz;
  const S* lx;
  const S* ly;
  const S* lz;
  const S* qx;
  const S* qy;
  const S* qz;
  int nyqx, nyqy, nyqz;  // index n/2 for even n, else -1
  S bx, by, bz;

  __device__ __forceinline__ S dipole(S kx, S ky, S kz) const {
    const S kdb = kx * bx + ky * by + kz * bz;
    const S k2 = kx * kx + ky * ky + kz * kz;
    return k2 > S(1e-20) ? S(1.0 / 3.0) - (kdb * kdb) / k2 : S(0);
  }
  __device__ __forceinline__ S lapneg(int ix, int iy, int iz) const {
    return (__ldg(lx + ix) + __ldg(ly + iy)) + __ldg(lz + iz);
  }
  __device__ __forceinline__ S poisson(int ix, int iy, int iz) const {
    return (__ldg(qx + ix) + __ldg(qy + iy)) + __ldg(qz + iz);
  }
  __device__ __forceinline__ bool on_nyquist(int ix, int iy, int iz) const {
    return ix == nyqx || iy == nyqy || iz == nyqz;
  }
  // Evaluate a multiplier M(kx,ky,kz,ix,iy,iz) symmetrised over k -> -k: the C2C
  // reference keeps Re(IFFT(F * M)), which equals IFFT(F * (M(k) + M(-k))/2) for real
  // input.  M(-k) differs from M(k) only on even-length Nyquist planes, where the
  // mirrored index keeps its frequency -n/2 while the other coordinates flip sign.
  template <class F>
  __device__ __forceinline__ S sym(int ix, int iy, int iz, const F& m) const {
    const S kx = __ldg(fx + ix), ky = __ldg(fy + iy), kz = __ldg(fz + iz);
    S v = m(kx, ky, kz, ix, iy, iz);
    if (on_nyquist(ix, iy, iz)) {
      const S v2 = m(ix == nyqx ? -kx : kx, iy == nyqy ? -ky : ky, iz == nyqz ? -kz : kz, ix, iy, iz);
      v = S(0.5) * (v + v2);
    }
    return v;
  }
};
using KSpace = KSpaceT<double>;

template <typename S> KSpaceT<S> make_kspace_t(qsm_ctx* ctx, const GridDims& d, const double bdir[3]);
KSpace make_kspace(qsm_ctx* ctx, const GridDims& d, const double bdir[3]);

}  // namespace qsm
