// Two-factor DFT passes: any axis length n = ra * rb as two dense DFTs of run-time radix.
//
// The Stockham engine needs one codelet per radix (2..16), so a length with another prime
// factor had to run as a Bluestein convolution of twice its length, and lengths outside
// the compile-time lists run codelets behind a run-time switch.  Here a transform is
//   y[k1 + ra k2] = sum_j W_rb^(j k2) W_n^(j k1) sum_r W_ra^(r k1) x[j + rb r],
// two dense DFTs whose radices are plain loop counts: a thread takes 16 bytes of columns (or
// row pairs), one j and a block of KT output frequencies, keeps their sums in registers
// and walks the inputs, so one small kernel serves every length.  A pair of inputs r, ra - r
// and a pair of outputs k, ra - k share cos and sin: with s = x_r + x_{ra-r} and
// d = x_r - x_{ra-r},
//   y_k, y_{ra-k} = (x_0 + sum cos s) +- i DIR (sum sin d),
// which costs ra + rb fused multiply-adds per complex element in all: 32 at 256 = 16 * 16
// and 111 at 218 = 2 * 109, against some 28 for codelets and 240 for the 441-point
// Bluestein convolution of 218.
#pragma once

#include "passes.cuh"

namespace qsm {

constexpr int kTfThreads = 256;
constexpr int kTfMaxKT = 3;  // output frequencies a thread holds
// Resident blocks the kernels are compiled for (64 registers in float, 80 in double).
template <typename T> constexpr int tf_min_blocks() { return sizeof(T) == 4 ? 4 : 3; }

// One axis of the two-factor passes; n = 0: this axis does not use them.
template <typename T> struct TwoFactor {
  int n;         // ra * rb
  int ra, rb;    // ra <= rb; ra = 1: a single dense DFT
  int kta, ktb;  // output frequencies held per thread
  int nka, nkb;  // sets of 4 * kt frequencies covering 0..r/2
  const cplx_t<T>* tw;  // W_n^k, k in [0, n)
};

// Columns of a tile: a warp is 8 lanes of 16-byte column vectors (two float or one double
// complex value) times four frequency blocks, so a data read is one 128-byte row whose
// words the four blocks share.
template <typename T> constexpr int tf_nc() { return 16 / (int)sizeof(cplx_t<T>); }
template <typename T> constexpr int tf_cols() { return 8 * tf_nc<T>(); }

template <typename T> struct alignas(16) TfVec {
  cplx_t<T> c[tf_nc<T>()];
};

// One dense stage over `groups` DFTs of radix R: a warp per (set of frequencies, group).
// from(g) is the lane's first input of group g (the others st elements apart); put(g, k, v)
// takes output k of the lane's columns.  tab holds W_n^i in shared memory; W_R^(m k) sits at
// i = (m k n / R) mod n, stepped by one add and a wrap per input pair.  (A matrix of all
// (m, k) read through L1 took 140 us for a 218-point FP64 Y pass at 182x218x182, L1-bound
// with 53 KB of matrix beside the tiles.)
template <typename T, int DIR, int KT, class From, class Put>
__device__ __forceinline__ void tf_stage_kt(int n, int R, int groups, int nk, const cplx_t<T>* tab, int st,
                                            const From& from, const Put& put) {
  using C = cplx_t<T>;
  using V = TfVec<T>;
  constexpr int NC = tf_nc<T>();
  const int kq = (threadIdx.x & 31) >> 3;
  const int H = (R - 1) / 2;
  for (int set = 0, g = threadIdx.x >> 5;; g += kTfThreads / 32) {
    while (g >= groups) {
      g -= groups;
      ++set;
    }
    if (set >= nk) break;
    const C* p = from(g);
    const int k0 = (set * 4 + kq) * KT;
    unsigned idx[KT], inc[KT];
#pragma unroll
    for (int q = 0; q < KT; ++q) {
      inc[q] = (unsigned)((2 * (k0 + q) <= R ? k0 + q : 0) * groups);  // groups = n / R
      idx[q] = inc[q];
    }
    C A[KT][NC], B[KT][NC];
    {
      const V x0 = *reinterpret_cast<const V*>(p);
#pragma unroll
      for (int q = 0; q < KT; ++q)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          A[q][c] = x0.c[c];
          B[q][c] = mk<C>(T(0), T(0));
        }
    }
    const C* pa = p + st;
    const C* pb = p + (R - 1) * st;
#pragma unroll 2
    for (int m = 0; m < H; ++m) {
      const V a = *reinterpret_cast<const V*>(pa), b = *reinterpret_cast<const V*>(pb);
      C w[KT];
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        w[q] = tab[idx[q]];
        const unsigned t = idx[q] + inc[q];
        idx[q] = min(t, t - (unsigned)n);  // t < 2 n: wraps to t - n once t >= n
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const C s = cadd(a.c[c], b.c[c]), d = csub(a.c[c], b.c[c]);
#pragma unroll
        for (int q = 0; q < KT; ++q) {
          A[q][c].x += w[q].x * s.x;
          A[q][c].y += w[q].x * s.y;
          B[q][c].x += w[q].y * d.x;  // w.y = -sin
          B[q][c].y += w[q].y * d.y;
        }
      }
      pa += st;
      pb -= st;
    }
    if ((R & 1) == 0) {
      const V a = *reinterpret_cast<const V*>(pa);
#pragma unroll
      for (int q = 0; q < KT; ++q) {
        const bool odd = (k0 + q) & 1;  // cos(pi k)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          A[q][c].x += odd ? -a.c[c].x : a.c[c].x;
          A[q][c].y += odd ? -a.c[c].y : a.c[c].y;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < KT; ++q) {
      const int k = k0 + q;
      if (2 * k <= R) {
        V y, z;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const C iB = (DIR < 0) ? cmul_i(B[q][c]) : cmul_mi(B[q][c]);
          y.c[c] = cadd(A[q][c], iB);
          z.c[c] = csub(A[q][c], iB);
        }
        put(g, k, y);
        if (k > 0 && 2 * k < R) put(g, R - k, z);
      }
    }
  }
}

template <typename T, int DIR, class From, class Put>
__device__ __forceinline__ void tf_stage(int n, int R, int kt, int groups, int nk, const cplx_t<T>* tab, int st,
                                         const From& from, const Put& put) {
  switch (kt) {
    case 1: tf_stage_kt<T, DIR, 1>(n, R, groups, nk, tab, st, from, put); break;
    case 2: tf_stage_kt<T, DIR, 2>(n, R, groups, nk, tab, st, from, put); break;
    default: tf_stage_kt<T, DIR, 3>(n, R, groups, nk, tab, st, from, put); break;
  }
}

// The stages of a tile in dynamic shared memory (element e of column px at offset
// e * S + px of a buffer; buffers are given as offsets in elements, so that the compiler
// sees shared-memory accesses; the twiddle table follows the two buffers).  Out of line: each is compiled once per direction and
// precision.

// First stage: `out` receives the twiddled values, a group's outputs in place of its inputs.
template <typename T, int DIR>
__device__ __noinline__ void tf_first(const TwoFactor<T>& ax, int S, int in, int out) {
  using C = cplx_t<T>;
  using V = TfVec<T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int px = (threadIdx.x & 7) * tf_nc<T>();
  const C* src = reinterpret_cast<const C*>(smraw) + in + px;
  C* dst = reinterpret_cast<C*>(smraw) + out + px;
  const int st = ax.rb * S;
  const C* tab = reinterpret_cast<const C*>(smraw) + 2 * ax.n * S;
  auto from = [&](int g) -> const C* { return src + g * S; };
  auto put = [&](int g, int k, V v) {
    const C w = tab[g * k];
#pragma unroll
    for (int c = 0; c < tf_nc<T>(); ++c) v.c[c] = (DIR < 0) ? cmul(v.c[c], w) : cmulc(v.c[c], w);
    *reinterpret_cast<V*>(dst + g * S + k * st) = v;
  };
  tf_stage<T, DIR>(ax.n, ax.ra, ax.kta, ax.rb, ax.nka, tab, st, from, put);
}

// Second stage into shared memory, natural order.
template <typename T, int DIR>
__device__ __noinline__ void tf_second(const TwoFactor<T>& ax, int S, int in, int out) {
  using C = cplx_t<T>;
  using V = TfVec<T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int px = (threadIdx.x & 7) * tf_nc<T>();
  const C* src = reinterpret_cast<const C*>(smraw) + in + px;
  C* dst = reinterpret_cast<C*>(smraw) + out + px;
  const int gs = ax.rb * S, ks = ax.ra * S;
  const C* tab = reinterpret_cast<const C*>(smraw) + 2 * ax.n * S;
  auto from = [&](int g) -> const C* { return src + g * gs; };
  auto put = [&](int g, int k, V v) { *reinterpret_cast<V*>(dst + g * S + k * ks) = v; };
  tf_stage<T, DIR>(ax.n, ax.rb, ax.ktb, ax.ra, ax.nkb, tab, S, from, put);
}

// Second stage to global memory: element e of column px < ncols at dst[e * estride + px].
template <typename T, int DIR>
__device__ __noinline__ void tf_second_g(const TwoFactor<T>& ax, int S, int in, cplx_t<T>* __restrict__ dst, int ncols,
                                         long long estride) {
  using C = cplx_t<T>;
  using V = TfVec<T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int px = (threadIdx.x & 7) * tf_nc<T>();
  const C* src = reinterpret_cast<const C*>(smraw) + in + px;
  const int gs = ax.rb * S;
  const C* tab = reinterpret_cast<const C*>(smraw) + 2 * ax.n * S;
  const long long ks = ax.ra * estride;
  C* out = dst + px;
  const int mine = ncols - px;  // valid columns of this lane
  auto from = [&](int g) -> const C* { return src + g * gs; };
  auto put = [&](int g, int k, V v) {
    C* o = out + g * estride + k * ks;
    if (mine >= tf_nc<T>()) *reinterpret_cast<V*>(o) = v;
    else if (mine > 0) *o = v.c[0];
  };
  tf_stage<T, DIR>(ax.n, ax.rb, ax.ktb, ax.ra, ax.nkb, tab, S, from, put);
}

// Whole transform in shared memory, natural order, from buffer a; returns the buffer that
// holds it (a, or b when ra = 1).  Ends with a block barrier.
template <typename T, int DIR>
__device__ __forceinline__ int tf_transform(const TwoFactor<T>& ax, int S, int a, int b) {
  int r = b;
  if (ax.ra > 1) {
    tf_first<T, DIR>(ax, S, a, b);
    __syncthreads();
    tf_second<T, DIR>(ax, S, b, a);
    r = a;
  } else {
    tf_second<T, DIR>(ax, S, a, b);
  }
  __syncthreads();
  return r;
}

// Stage a tile of tf_cols() columns at one outer index (as issue_tile, 128-byte rows).
template <typename C>
__device__ __forceinline__ void tf_issue(const C* __restrict__ src, C* buf, const Geom& g, const TileWalk& w, int tile,
                                         int n) {
  constexpr int NC = 16 / (int)sizeof(C), P = 8 * NC;
  const int tx = tile % w.ntx, outer = tile / w.ntx;
  const int ch = (threadIdx.x & 7) * NC;
  const bool ok = tx * P + ch < g.nxh;
  const C* gp = src + tx * P + (long long)outer * w.ostride + (ok ? ch : 0);
  for (int e = threadIdx.x >> 3; e < n; e += kTfThreads / 8) cp_async16(buf + e * P + ch, gp + e * w.estride, ok);
}

template <typename T> __device__ __forceinline__ void tf_load_table(const TwoFactor<T>& ax, cplx_t<T>* tab) {
  for (int i = threadIdx.x; i < ax.n; i += kTfThreads) tab[i] = __ldg(ax.tw + i);
}

// f(i) -> value for i in [0, total) step kTfThreads from tid, written by put(i, v): the
// values of U elements are formed before any is stored, so that their loads overlap.
template <int U, class F, class Put>
__device__ __forceinline__ void tf_each(int first, int step, int total, const F& f, const Put& put) {
  using V = decltype(f(0));
  int i = first;
  for (; i + (U - 1) * step < total; i += U * step) {
    V v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = f(i + u * step);
#pragma unroll
    for (int u = 0; u < U; ++u) put(i + u * step, v[u]);
  }
#pragma unroll 1
  for (; i < total; i += step) put(i, f(i));
}

// Y/Z pass (IsPlainOp: no hooks; ACC: the post hook also sums one FP64
// value per element, which the last block hands to op.last).  The
// tile is staged by cp.async; the next tile's copy starts as soon as the first stage has
// read this one, under the second stage and the stores.
template <typename T, int DIR, int AXIS, class Op, bool ACC>
__global__ void __launch_bounds__(kTfThreads, tf_min_blocks<T>())
    k_pass_yz_tf(Geom g, const __grid_constant__ TwoFactor<T> ax, TileWalk w, const cplx_t<T>* src,
                 cplx_t<T>* dst, Op op, double* __restrict__ partials, unsigned* counter,
                 const int* __restrict__ done) {
  using C = cplx_t<T>;
  if (done != nullptr && *done) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  constexpr int P = tf_cols<T>(), lp = P == 16 ? 4 : 3;
  const int n = ax.n;
  int a = 0, b = n * P;
  double acc[1] = {0.0};
  tf_load_table(ax, sm + 2 * n * P);
  int tile = blockIdx.x;
  if (tile < w.ntiles) tf_issue(src, sm + a, g, w, tile, n);
  cp_async_commit();
  for (; tile < w.ntiles; tile += gridDim.x) {
    const int next = tile + gridDim.x;
    const int tx = tile % w.ntx, outer = tile / w.ntx;
    const int ncols = min(P, g.nxh - (tx << lp));
    const long long base = (tx << lp) + (long long)outer * w.ostride;
    cp_async_wait<0>();
    __syncthreads();
    if constexpr (!IsPlainOp<Op>::value) {
      tf_each<2>(
          threadIdx.x, kTfThreads, n << lp,
          [&](int i) -> C {
            const int e = i >> lp, px = i & (P - 1);
            const C v = sm[a + i];
            if (px >= ncols) return v;
            const long long idx = base + px + (long long)e * w.estride;
            return (AXIS == 1) ? op.pre(v, (tx << lp) + px, e, outer, idx) : op.pre(v, (tx << lp) + px, outer, e, idx);
          },
          [&](int i, C v) { sm[a + i] = v; });
      __syncthreads();
    }
    if (ax.ra > 1) {
      tf_first<T, DIR>(ax, P, a, b);
    } else {
      const int t = a;
      a = b;
      b = t;
    }
    __syncthreads();
    if constexpr (IsPlainOp<Op>::value) {
      if (next < w.ntiles) tf_issue(src, sm + a, g, w, next, n);
      cp_async_commit();
      tf_second_g<T, DIR>(ax, P, b, dst + base, ncols, w.estride);
    } else {
      tf_second<T, DIR>(ax, P, b, a);
      __syncthreads();
      tf_each<2>(
          threadIdx.x, kTfThreads, n << lp,
          [&](int i) -> C {
            const int e = i >> lp, px = i & (P - 1);
            const C v = sm[a + i];
            if (px >= ncols) return v;
            const long long idx = base + px + (long long)e * w.estride;
            if constexpr (ACC)
              return (AXIS == 1) ? op.post(v, (tx << lp) + px, e, outer, idx, acc[0])
                                 : op.post(v, (tx << lp) + px, outer, e, idx, acc[0]);
            else
              return (AXIS == 1) ? op.post(v, (tx << lp) + px, e, outer, idx)
                                 : op.post(v, (tx << lp) + px, outer, e, idx);
          },
          [&](int i, C v) {
            const int px = i & (P - 1);
            if (px < ncols) dst[base + px + (long long)(i >> lp) * w.estride] = v;
          });
      __syncthreads();
      if (next < w.ntiles) tf_issue(src, sm + a, g, w, next, n);
      cp_async_commit();
    }
    __syncthreads();  // b is free for the next tile
  }
  cp_async_wait<0>();
  if constexpr (ACC) {
    if (grid_sum_last<1>(acc, partials, counter) && threadIdx.x == 0) op.last(acc[0]);
  }
}

// Z forward -> op.mid -> Z inverse, tiled and staged as k_pass_yz_tf.
template <typename T, class Op>
__global__ void __launch_bounds__(kTfThreads, tf_min_blocks<T>())
    k_z_fused_tf(Geom g, const __grid_constant__ TwoFactor<T> ax, TileWalk w, const cplx_t<T>* src,
                 cplx_t<T>* dst, Op op, const int* __restrict__ done) {
  using C = cplx_t<T>;
  if (done != nullptr && *done) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  constexpr int P = tf_cols<T>(), lp = P == 16 ? 4 : 3;
  const int n = ax.n;
  const int a = 0, b = n * P;
  tf_load_table(ax, sm + 2 * n * P);
  int tile = blockIdx.x;
  if (tile < w.ntiles) tf_issue(src, sm + a, g, w, tile, n);
  cp_async_commit();
  for (; tile < w.ntiles; tile += gridDim.x) {
    const int next = tile + gridDim.x;
    const int tx = tile % w.ntx, iy = tile / w.ntx;
    const int ncols = min(P, g.nxh - (tx << lp));
    const long long base = (tx << lp) + (long long)iy * w.ostride;
    cp_async_wait<0>();
    __syncthreads();
    int f = tf_transform<T, -1>(ax, P, a, b);
    tf_each<2>(
        threadIdx.x, kTfThreads, n << lp,
        [&](int i) -> C {
          const int e = i >> lp, px = i & (P - 1);
          const C v = sm[f + i];
          return px < ncols ? op.mid(v, (tx << lp) + px, iy, e, base + px + (long long)e * w.estride) : v;
        },
        [&](int i, C v) { sm[f + i] = v; });
    __syncthreads();
    if (ax.ra > 1) {  // f is a
      tf_first<T, +1>(ax, P, a, b);
      f = b;
      __syncthreads();
    }
    // a is free: read by the stage above, or (ra = 1) the first transform's input
    if (next < w.ntiles) tf_issue(src, sm + a, g, w, next, n);
    cp_async_commit();
    tf_second_g<T, +1>(ax, P, f, dst + base, ncols, w.estride);
    __syncthreads();
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------- X passes --
// tf_cols() pencils per block, element e of pencil p at e * S + p with S = 144 bytes, so
// that the coalesced row loops (lanes along e) spread over the banks and the stages read
// aligned 128-byte rows.  A warp owns whole rows in the row loops.  Blocks walk the pencils
// with stride gridDim.x (the launcher bounds the grid, for stores that reduce over it).
template <typename T> constexpr int tf_x_stride() { return tf_cols<T>() + tf_nc<T>(); }

// Real rows (two per pencil) -> half spectrum.
template <typename T, class Load>
__global__ void __launch_bounds__(kTfThreads, tf_min_blocks<T>())
    k_x_r2c_tf(Geom g, const __grid_constant__ TwoFactor<T> ax, cplx_t<T>* __restrict__ spec, Load ld,
               const int* __restrict__ done) {
  using C = cplx_t<T>;
  if (done != nullptr && *done) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  constexpr int P = tf_cols<T>(), S = tf_x_stride<T>();
  const int n = ax.n;
  tf_load_table(ax, sm + 2 * n * S);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nrows = g.nrows();
  const int npairs = (nrows + 1) >> 1;
  for (int q0 = blockIdx.x * P; q0 < npairs; q0 += gridDim.x * P) {
    for (int p = wid; p < P; p += kTfThreads / 32) {
      const int r0 = 2 * (q0 + p), r1 = r0 + 1;
      const bool h0 = r0 < nrows, h1 = r1 < nrows;
      tf_each<4>(
          lane, 32, n, [&](int e) -> C { return mk<C>(h0 ? ld(r0, e) : T(0), h1 ? ld(r1, e) : T(0)); },
          [&](int e, C v) { sm[e * S + p] = v; });
    }
    __syncthreads();
    const int z = tf_transform<T, -1>(ax, S, 0, n * S);
    for (int p = wid; p < P; p += kTfThreads / 32) {
      const int r0 = 2 * (q0 + p), r1 = r0 + 1;
      if (r0 >= nrows) break;
      C* ra = spec + (long long)r0 * g.pitch;
      C* rb = spec + (long long)r1 * g.pitch;
      const T half = T(0.5);
#pragma unroll 2
      for (int k = lane; k < g.nxh; k += 32) {
        const C zk = sm[z + k * S + p];
        const C zn = sm[z + (k == 0 ? 0 : n - k) * S + p];
        ra[k] = mk<C>((zk.x + zn.x) * half, (zk.y - zn.y) * half);
        if (r1 < nrows) rb[k] = mk<C>((zk.y + zn.y) * half, (zn.x - zk.x) * half);
      }
    }
    __syncthreads();
  }
}

// Half spectrum -> real rows handed to the store functor.
template <typename T, class Store>
__global__ void __launch_bounds__(kTfThreads, tf_min_blocks<T>())
    k_x_c2r_tf(Geom g, const __grid_constant__ TwoFactor<T> ax, const cplx_t<T>* __restrict__ spec, Store st0,
               const int* __restrict__ done) {
  using C = cplx_t<T>;
  if (done != nullptr && *done) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  constexpr int P = tf_cols<T>(), S = tf_x_stride<T>();
  const int n = ax.n;
  tf_load_table(ax, sm + 2 * n * S);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nrows = g.nrows();
  const int npairs = (nrows + 1) >> 1;
  struct Two {
    C a, b;
  };
  Store st = st0;
  for (int q0 = blockIdx.x * P; q0 < npairs; q0 += gridDim.x * P) {
    if constexpr (RowFilter<Store>::value) {
      const int r = 2 * q0 + (int)threadIdx.x;
      if (!__syncthreads_or(threadIdx.x < 2 * P && r < nrows && st0.wants_row(r))) continue;
    }
    for (int p = wid; p < P; p += kTfThreads / 32) {
      const int r0 = 2 * (q0 + p), r1 = r0 + 1;
      const bool h0 = r0 < nrows, h1 = r1 < nrows;
      const C* ra = spec + (long long)r0 * g.pitch;
      const C* rb = spec + (long long)r1 * g.pitch;
      tf_each<4>(
          lane, 32, g.nxh,
          [&](int k) -> Two {
            return Two{h0 ? ra[k] : mk<C>(T(0), T(0)), h1 ? rb[k] : mk<C>(T(0), T(0))};
          },
          [&](int k, Two v) {
            const bool selfm = (k == 0) || (2 * k == n);
            if (selfm) {
              v.a.y = T(0);
              v.b.y = T(0);
            }
            sm[k * S + p] = mk<C>(v.a.x - v.b.y, v.a.y + v.b.x);
            if (!selfm) sm[(n - k) * S + p] = mk<C>(v.a.x + v.b.y, v.b.x - v.a.y);
          });
    }
    __syncthreads();
    const int z = tf_transform<T, +1>(ax, S, 0, n * S);
    for (int p = wid; p < P; p += kTfThreads / 32) {
      const int r0 = 2 * (q0 + p), r1 = r0 + 1;
      if (r0 >= nrows) break;
#pragma unroll 4
      for (int e = lane; e < n; e += 32) {
        const C v = sm[z + e * S + p];
        st(r0, e, v.x);
        if (r1 < nrows) st(r1, e, v.y);
      }
    }
    __syncthreads();
  }
  st.finish();
}

}  // namespace qsm
