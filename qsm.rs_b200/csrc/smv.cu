// Spherical-mean-value kernels without transforms: the sphere's spectrum from its own
// run lengths, and mask erosion by exact counts.
//
// Spectrum.  The kernel is real, even and supported on a few thousand voxels, so its
// transform is a short cosine sum per axis:
//   X_L(kx) = sum_{|d| <= L} cos(2 pi kx d / nx)                 (a prefix sum over L)
//   A(dz, ky, kx) = sum_dy w(dy) cos(2 pi ky dy / ny) X_{L(dy, dz)}(kx)
//   S(kz, ky, kx) = norm sum_dz w(dz) cos(2 pi kz dz / nz) A(dz, ky, kx)
// (offsets >= 0, w = 2 except at 0 and n/2).  At radius 12 voxels that is 13 FP64
// multiply-adds per spectrum element, one write, no reads worth counting: three FP64
// transform passes over the zero-padded volume before.  The multiplier that a solver needs
// (S, 1 - S or its thresholded inverse) is formed in double and stored in working
// precision.
//
// Erosion.  mean(mask over the sphere) > delta with delta just below 1 allows a fixed
// number of missing voxels (2 of 7153 at radius 12, none below radius 10), so for a 0/1
// mask the decision is a count.  One exact distance transform to the nearest zero voxel
// serves every sphere: a voxel further from all zeros than the radius (compared with the
// sphere's own rounding, (dx^2 + dy^2) + dz^2) misses nothing.  Only where a sphere
// tolerates missing voxels are the others counted: up to two on bit planes, 32 voxels a
// thread; more (spheres from about 9500 voxels, 13 voxels of radius) and masks with values
// above 1 by the sphere's sums of the mask through FP64 transforms, rounded to the whole
// numbers that they are, whose cost depends neither on the radius nor on the values.  (Counting
// voxel by voxel along the sphere's rows, V-SHARP of radii 12..1 mm took 33.9 ms at
// 384x384x256 and 0.6 mm in double and 12.5 ms at 192x192x128 and 0.4 mm, now 14.2 and 2.9;
// on a mask of threes 44.8 ms at 256x256x176 and 1 mm, now 5.2.)
#include "functors.cuh"
#include "smv.h"

#include <algorithm>
#include <cmath>

#include "solvers.h"

namespace qsm {

namespace {

double axis_coord(int c, double vs) { return (double)c * vs; }

constexpr unsigned kNoZero = 0xffffu;  // no zero voxel within the window

// ------------------------------------------------------------------- spectrum --
// cos(2 pi i / n), i in [0, n)
const double* cos_table(qsm_ctx* ctx, int n) {
  const std::string key = "cos:" + std::to_string(n);
  auto it = ctx->tables.find(key);
  if (it != ctx->tables.end()) return static_cast<const double*>(it->second);
  std::vector<double> c((size_t)n);
  for (int i = 0; i < n; ++i) c[(size_t)i] = cos2pi(i, n);
  return static_cast<const double*>(upload_table(ctx, key, c.data(), c.size() * sizeof(double)));
}

// Half-widths of the runs, [dz + 1][dy + 1], as a kernel parameter where they fit.
constexpr int kHalfMax = 1800;
struct HalfTable {
  short h[kHalfMax];
};

// A(dz, ky, kx), with the weight of dz.  Runs widen as |dy| shrinks, so X_L is one prefix
// sum extended on the way from the largest dy to 0.
__global__ void __launch_bounds__(128)
    k_smv_y(int nx, int ny, int nz, int nxh, int dy, const __grid_constant__ HalfTable tab,
            const int* __restrict__ half, const double* __restrict__ cx, const double* __restrict__ cy,
            double* __restrict__ A) {
  const int kx = blockIdx.x * blockDim.x + threadIdx.x;
  const int ky = blockIdx.y, z = blockIdx.z;
  if (kx >= nxh) return;
  double s = 0.0, X = 0.0;
  int have = -1, ix = 0;  // X holds offsets 0..have; ix = (have + 1) kx mod nx
  int iy = (int)((long long)dy * ky % ny);
  for (int y = dy; y >= 0; --y) {
    const int at = z * (dy + 1) + y;
    const int L = half ? __ldg(half + at) : (int)tab.h[at];
    while (have < L) {
      ++have;
      X += (have == 0 || 2 * have == nx ? 1.0 : 2.0) * __ldg(cx + ix);
      ix += kx;
      if (ix >= nx) ix -= nx;
    }
    if (L >= 0) s += (y == 0 || 2 * y == ny ? 1.0 : 2.0) * __ldg(cy + iy) * X;
    iy -= ky;
    if (iy < 0) iy += ny;
  }
  A[((size_t)z * ny + ky) * nxh + kx] = (z == 0 || 2 * z == nz ? 1.0 : 2.0) * s;
}

// The normalised sphere's image (src/kernels/smv.rs:19-67) as an X-pass input; the inclusion
// test without fused multiply-adds, as the reference's.
struct LoadSphere {
  int nx, ny, nz;
  double vsx, vsy, vsz, r2, norm;
  static __device__ __forceinline__ double coord(int i, int n, double vs) { return (double)(i <= n / 2 ? i : i - n) * vs; }
  __device__ __forceinline__ double operator()(int row, int e) const {
    const int k = row / ny, j = row - k * ny;
    const double dx = coord(e, nx, vsx), dy = coord(j, ny, vsy), dz = coord(k, nz, vsz);
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)) <= r2 ? norm : 0.0;
  }
};
__global__ void k_one_minus_re(long long H, const double2* __restrict__ S, float* __restrict__ out) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < H; i += (long long)gridDim.x * blockDim.x)
    out[i] = (float)(1.0 - S[i].x);
}

constexpr int kSmvZ = 16;   // kz per thread
constexpr int kSmvZc = 32;  // planes of dz per shared-memory cosine table

// S over kSmvZ values of kz per thread; the multiplier of `kind` in working precision
template <typename T>
__global__ void __launch_bounds__(256)
    k_smv_z(Geom g, int dz, double norm, const double* __restrict__ cz, const double* __restrict__ A, int kind,
            double thr, T* __restrict__ out) {
  __shared__ double cs[kSmvZc * kSmvZ];
  const int k0 = blockIdx.y * kSmvZ;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int ky = i / g.pitch, kx = i - ky * g.pitch;
  const bool in = i < g.ny * g.pitch;
  double acc[kSmvZ];
#pragma unroll
  for (int q = 0; q < kSmvZ; ++q) acc[q] = 0.0;
  for (int z0 = 0; z0 <= dz; z0 += kSmvZc) {
    const int zn = min(kSmvZc, dz + 1 - z0);
    __syncthreads();
    for (int t = threadIdx.x; t < zn * kSmvZ; t += blockDim.x) {
      const int z = t / kSmvZ, q = t - z * kSmvZ;
      cs[t] = cz[(int)((long long)(k0 + q) * (z0 + z) % g.nz)];
    }
    __syncthreads();
    if (in && kx < g.nxh)
#pragma unroll 4
      for (int z = 0; z < zn; ++z) {
        const double a = A[((size_t)(z0 + z) * g.ny + ky) * g.nxh + kx];
#pragma unroll
        for (int q = 0; q < kSmvZ; ++q) acc[q] += a * cs[z * kSmvZ + q];
      }
  }
  if (!in) return;
#pragma unroll
  for (int q = 0; q < kSmvZ; ++q) {
    if (k0 + q >= g.nz) break;
    double v = acc[q] * norm;
    if (kind != kSmvS) v = 1.0 - v;
    if (kind == kSmvDeconv) v = fabs(v) < thr ? 0.0 : 1.0 / v;
    out[((size_t)(k0 + q) * g.ny + ky) * g.pitch + kx] = kx < g.nxh ? (T)v : T(0);
  }
}

// -------------------------------------------------------------------- erosion --
struct ErodeState {
  int weighted;  // the mask holds a value above 1
};

// One warp per row: distance in x to the row's nearest zero voxel (periodic, up to rx;
// kNoZero beyond).
__global__ void __launch_bounds__(256)
    k_smv_rows(int nx, int nrows, int rx, const uint8_t* __restrict__ mask, uint16_t* __restrict__ gx,
               ErodeState* st) {
  extern __shared__ unsigned bits_all[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ext = nx + 2 * rx, words = (ext + 31) >> 5;
  unsigned* bits = bits_all + wid * words;
  bool weighted = false;
  for (int row = blockIdx.x * 8 + wid; row < nrows; row += gridDim.x * 8) {
    const uint8_t* m = mask + (long long)row * nx;
    for (int w = 0; w < words; ++w) {
      const int j = w * 32 + lane;
      int x = j - rx;
      x = x < 0 ? x + nx : (x >= nx ? x - nx : x);
      const unsigned b = __ballot_sync(0xffffffffu, j < ext && m[x] == 0);
      if (lane == 0) bits[w] = b;
    }
    __syncwarp();
    for (int x0 = 0; x0 < nx; x0 += 32) {
      const int x = x0 + lane;
      if (x < nx) {
        weighted |= m[x] > 1;
        const int j = x + rx, w0 = j >> 5, b0 = j & 31;
        int best = rx + 1;
        unsigned u = bits[w0] >> b0;  // zeros at or right of x
        for (int w = w0;;) {
          if (u) {
            best = min(best, w * 32 + (w == w0 ? b0 : 0) + __ffs(u) - 1 - j);
            break;
          }
          if (++w >= words || w * 32 - j > rx) break;
          u = bits[w];
        }
        u = bits[w0] << (31 - b0);  // zeros at or left of x
        for (int w = w0;;) {
          if (u) {
            best = min(best, j - (w * 32 + (w == w0 ? b0 : 31) - __clz(u)));
            break;
          }
          if (--w < 0 || j - (w * 32 + 31) > rx) break;
          u = bits[w];
        }
        gx[(long long)row * nx + x] = best <= rx ? (uint16_t)best : (uint16_t)kNoZero;
      }
    }
    __syncwarp();
  }
  if (__any_sync(0xffffffffu, weighted) && lane == 0) atomicOr(&st->weighted, 1);
}

constexpr int kEdtU = 8;  // outputs per thread along the pass's axis

// min over |dy| <= ry of dx^2 + dy^2 (double, the sphere test's rounding)
__global__ void __launch_bounds__(256)
    k_smv_edt_y(int nx, int ny, int nz, int rx, int ry, double vsx, double vsy, const uint16_t* __restrict__ gx,
                double* __restrict__ d2) {
  extern __shared__ __align__(16) double tab[];
  double* sx = tab;           // dx^2, dx in [0, rx]
  double* sy = tab + rx + 1;  // dy^2, dy in [0, ry]
  for (int i = threadIdx.x; i <= rx; i += blockDim.x) {
    const double c = (double)i * vsx;
    sx[i] = __dmul_rn(c, c);
  }
  for (int i = threadIdx.x; i <= ry; i += blockDim.x) {
    const double c = (double)i * vsy;
    sy[i] = __dmul_rn(c, c);
  }
  __syncthreads();
  const int x = blockIdx.x * 32 + (threadIdx.x & 31);
  const int y0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * kEdtU;
  const int z = blockIdx.z;
  if (x >= nx || y0 >= ny) return;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  double m[kEdtU];
  const uint16_t* col = gx + (long long)z * ny * nx + x;
  unsigned any = 0u;  // zero voxels are done: distance 0
#pragma unroll
  for (int u = 0; u < kEdtU; ++u) {
    m[u] = inf;
    any |= y0 + u < ny ? col[(long long)(y0 + u) * nx] : 0u;
  }
  if (any == 0u) {
#pragma unroll
    for (int u = 0; u < kEdtU; ++u)
      if (y0 + u < ny) d2[((long long)z * ny + y0 + u) * nx + x] = 0.0;
    return;
  }
  for (int t = -ry; t < ry + kEdtU; ++t) {
    int y = y0 + t;
    y = y < 0 ? y + ny : y;
    while (y >= ny) y -= ny;
    const unsigned d = col[(long long)y * nx];
    if (d == kNoZero) continue;
    const double a = sx[d];
#pragma unroll
    for (int u = 0; u < kEdtU; ++u) {
      const int dy = t > u ? t - u : u - t;
      if (dy <= ry) m[u] = fmin(m[u], __dadd_rn(a, sy[dy]));
    }
  }
#pragma unroll
  for (int u = 0; u < kEdtU; ++u)
    if (y0 + u < ny) d2[((long long)z * ny + y0 + u) * nx + x] = m[u];
}

// min over |dz| <= rz of d2 + dz^2, then the first sphere whose radius it exceeds
__global__ void __launch_bounds__(256)
    k_smv_edt_z(int nx, int ny, int nz, int rz, double vsz, const double* __restrict__ d2, int ns,
                const double* __restrict__ r2, uint8_t* __restrict__ first) {
  extern __shared__ __align__(16) double tab[];
  double* sz = tab;           // dz^2
  double* sr = tab + rz + 1;  // r^2
  for (int i = threadIdx.x; i <= rz; i += blockDim.x) {
    const double c = (double)i * vsz;
    sz[i] = __dmul_rn(c, c);
  }
  for (int i = threadIdx.x; i < ns; i += blockDim.x) sr[i] = r2[i];
  __syncthreads();
  const long long p = (long long)blockIdx.x * 256 + threadIdx.x, sxy = (long long)nx * ny;
  const int z0 = blockIdx.y * kEdtU;
  if (p >= sxy) return;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  double m[kEdtU];
  double any = 0.0;
#pragma unroll
  for (int u = 0; u < kEdtU; ++u) {
    m[u] = inf;
    any = fmax(any, z0 + u < nz ? d2[(z0 + u) * sxy + p] : 0.0);
  }
  if (any == 0.0) {  // zero voxels: no sphere keeps them whole
#pragma unroll
    for (int u = 0; u < kEdtU; ++u)
      if (z0 + u < nz) first[(z0 + u) * sxy + p] = 255;
    return;
  }
  for (int t = -rz; t < rz + kEdtU; ++t) {
    int z = z0 + t;
    z = z < 0 ? z + nz : z;
    while (z >= nz) z -= nz;
    const double a = d2[z * sxy + p];
    if (a == inf) continue;
#pragma unroll
    for (int u = 0; u < kEdtU; ++u) {
      const int dz = t > u ? t - u : u - t;
      if (dz <= rz) m[u] = fmin(m[u], __dadd_rn(a, sz[dz]));
    }
  }
#pragma unroll
  for (int u = 0; u < kEdtU; ++u) {
    if (z0 + u >= nz) break;
    int f = 255;
    for (int s = 0; s < ns; ++s)
      if (m[u] > sr[s]) {
        f = s;
        break;
      }
    first[(z0 + u) * sxy + p] = (uint8_t)f;
  }
}

// Rows of one sphere and its decision: at least `need` of its `total` voxels (a 0/1 mask:
// at most total - need missing).
struct ErodeSphere {
  int begin, count;  // rows in the row list
  long long total, need;
};

// Zeros of the mask as bits, 32 voxels of a row per word with a margin of `pad` words on
// either side (periodic): bit j of word w of a row is voxel 32 (w - pad) + j.
__global__ void __launch_bounds__(256)
    k_smv_bits(int nx, int nrows, int words, int pad, const uint8_t* __restrict__ mask, unsigned* __restrict__ bits) {
  const int lane = threadIdx.x & 31;
  const long long total = (long long)nrows * words;
  for (long long t = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); t < total; t += (long long)gridDim.x * 8) {
    const long long row = t / words;
    int x = ((int)(t - row * words) - pad) * 32 + lane;
    if (x < 0) x += nx;
    if (x >= nx) x -= nx;
    const bool ok = x >= 0 && x < nx;
    const unsigned b = __ballot_sync(0xffffffffu, ok && mask[row * nx + x] == 0);
    if (lane == 0) bits[t] = b;
  }
}

// Saturating counts of the zeros within L of each voxel along its row, L = 0..lmax:
// planes[(3 * L + c) * nrows * wpr + row * wpr + w] has a voxel's bit set when there are at
// least c + 1.
__global__ void __launch_bounds__(256)
    k_smv_planes(int nx, int nrows, int wpr, int words, int pad, int lmax, const unsigned* __restrict__ bits,
                 unsigned* __restrict__ planes) {
  const long long plane = (long long)nrows * wpr;
  const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
  if (t >= plane) return;
  const long long row = t / wpr;
  const unsigned* r = bits + row * words + pad + (int)(t - row * wpr);  // the voxels' own word
  unsigned c1 = 0u, c2 = 0u, c3 = 0u;
  auto take = [&](int off) {  // zeros at distance off
    const int w = off >> 5;   // floor
    const unsigned z = __funnelshift_r(__ldg(r + w), __ldg(r + w + 1), off & 31);
    c3 |= c2 & z;
    c2 |= c1 & z;
    c1 |= z;
  };
  for (int L = 0; L <= lmax; ++L) {
    take(-L);
    if (L > 0 && 2 * L != nx) take(L);  // offset n/2 is one voxel
    unsigned* o = planes + 3LL * L * plane + t;
    o[0] = c1;
    o[plane] = c2;
    o[2 * plane] = c3;
  }
}

// Sums of a sphere's rows over the bit planes, NP planes (counts up to NP), eight rows at a
// time: their loads are in flight together, and the exit test (no open voxel can still have
// fewer than NP zeros) sees them all.
template <int NP>
__device__ __forceinline__ void smv_row_sum(const ErodeSphere& E, int y, int z, int ny, int nz, int wpr, int w,
                                            long long plane, const int4* __restrict__ rows,
                                            const unsigned* __restrict__ planes, unsigned open, unsigned& c1,
                                            unsigned& c2, unsigned& c3) {
  constexpr int U = 8;
  for (int r0 = 0; r0 < E.count; r0 += U) {
    unsigned a[U][3];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = min(r0 + u, E.count - 1);
      const int4 q = __ldg(rows + E.begin + r);
      int yy = y + q.x, zz = z + q.y;
      yy = yy < 0 ? yy + ny : (yy >= ny ? yy - ny : yy);
      zz = zz < 0 ? zz + nz : (zz >= nz ? zz - nz : zz);
      const unsigned* p = planes + 3LL * q.z * plane + ((long long)zz * ny + yy) * wpr + w;
#pragma unroll
      for (int c = 0; c < NP; ++c) a[u][c] = __ldg(p + c * plane);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (r0 + u >= E.count) break;
      if (NP == 3) c3 |= a[u][2] | (c1 & a[u][1]) | (c2 & a[u][0]);
      c2 |= a[u][1] | (c1 & a[u][0]);
      c1 |= a[u][0];
    }
    if ((open & ~(NP == 2 ? c2 : c3)) == 0u) break;
  }
}

// Tolerances of one or two missing voxels, 32 voxels per thread: saturating counts of the
// sphere's zeros in three bit planes, summed over its rows.  (A count per voxel took 2.2 ms
// at 256x256x176 for V-SHARP's three tolerant radii: every warp along a boundary walked all
// 450 rows.)
__global__ void __launch_bounds__(128)
    k_smv_count_bits(int nx, int ny, int nz, int wpr, int ns, const ErodeSphere* __restrict__ spheres,
                     const int4* __restrict__ rows, const unsigned* __restrict__ planes,
                     uint8_t* __restrict__ first) {
  const long long nrows = (long long)ny * nz, plane = nrows * wpr;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= plane) return;
  const int w = (int)(t % wpr);
  const long long row = t / wpr;
  const int y = (int)(row % ny), z = (int)(row / ny);
  const int x0 = w * 32, xn = min(32, nx - x0);
  uint8_t* f = first + row * nx + x0;
  for (int s = 0; s < ns; ++s) {
    const ErodeSphere E = spheres[s];
    const long long tol = E.total - E.need;
    if (tol < 1 || tol > 2) continue;
    unsigned open = 0u;  // voxels no earlier sphere keeps
    for (int b = 0; b < xn; ++b) open |= (f[b] > s ? 1u : 0u) << b;
    if (open == 0u) continue;
    unsigned c1 = 0u, c2 = 0u, c3 = 0u;
    if (tol == 1) smv_row_sum<2>(E, y, z, ny, nz, wpr, w, plane, rows, planes, open, c1, c2, c3);
    else smv_row_sum<3>(E, y, z, ny, nz, wpr, w, plane, rows, planes, open, c1, c2, c3);
    const unsigned keep = open & ~(tol == 1 ? c2 : c3);
    if (keep)
      for (int b = 0; b < xn; ++b)
        if ((keep >> b) & 1u) f[b] = (uint8_t)s;
  }
}

// The voxels that a sphere keeps by its sum of the mask (v / N times the sphere's voxels, a
// whole number), where no earlier sphere does.
struct StoreErode {
  uint8_t* first;
  int nx, index;
  double scale, need;
  __device__ __forceinline__ void operator()(int row, int e, double v) {
    const long long i = (long long)row * nx + e;
    if (rint(v * scale) >= need && (int)first[i] > index) first[i] = (uint8_t)index;
  }
  __device__ __forceinline__ void finish() {}
};

}  // namespace

SmvSphere smv_sphere(const GridDims& d, double radius) {
  SmvSphere s;
  s.nx = d.nx;
  s.ny = d.ny;
  s.nz = d.nz;
  s.r2 = radius * radius;
  auto sq = [](int c, double vs) {
    volatile double v = axis_coord(c, vs);
    volatile double w = v * v;
    return (double)w;
  };
  auto inside = [&](double x2, double y2, double z2) {
    volatile double xy = x2 + y2;
    volatile double d2 = xy + z2;
    return (double)d2 <= s.r2;
  };
  auto reach = [&](int n, double vs) {
    int m = 0;
    while (m + 1 <= n / 2 && sq(m + 1, vs) <= s.r2) ++m;
    return m;
  };
  const int dx = reach(d.nx, d.vsx);
  s.dy = reach(d.ny, d.vsy);
  s.dz = reach(d.nz, d.vsz);
  s.half.assign((size_t)(s.dy + 1) * (s.dz + 1), -1);
  s.total = 0.0;
  for (int z = 0; z <= s.dz; ++z) {
    int L = dx;
    for (int y = 0; y <= s.dy; ++y) {
      const double y2 = sq(y, d.vsy), z2 = sq(z, d.vsz);
      while (L >= 0 && !inside(sq(L, d.vsx), y2, z2)) --L;
      if (L < 0) break;
      s.half[(size_t)z * (s.dy + 1) + y] = L;
      const double wy = (y == 0 || 2 * y == d.ny) ? 1.0 : 2.0, wz = (z == 0 || 2 * z == d.nz) ? 1.0 : 2.0;
      s.total += wy * wz * (double)std::min(2 * L + 1, d.nx);
    }
  }
  return s;
}

template <typename T>
void smv_multiplier(qsm_ctx* ctx, const Fft3<T>& f, const SmvSphere& s, SmvMult kind, double threshold, T* out) {
  const int nxh = f.g.nxh;
  double* A = ws_scratch<double>(ctx, "smv.A", (size_t)(f.g.nz / 2 + 1) * f.g.ny * nxh);
  HalfTable tab;
  int* half = nullptr;
  if (s.half.size() <= (size_t)kHalfMax) {
    for (size_t i = 0; i < s.half.size(); ++i) tab.h[i] = (short)s.half[i];
  } else {
    half = ws_scratch<int>(ctx, "smv.half", (size_t)(f.g.ny / 2 + 1) * (f.g.nz / 2 + 1));
    h2d(ctx, half, s.half.data(), s.half.size() * sizeof(int));
  }
  LaunchScope ls(ctx, "smv_spectrum");
  k_smv_y<<<dim3((nxh + 127) / 128, f.g.ny, s.dz + 1), 128, 0, ctx->stream>>>(
      f.g.nx, f.g.ny, f.g.nz, nxh, s.dy, tab, half, cos_table(ctx, f.g.nx), cos_table(ctx, f.g.ny), A);
  k_smv_z<T><<<dim3((unsigned)((f.g.ny * f.g.pitch + 255) / 256), (f.g.nz + kSmvZ - 1) / kSmvZ), 256, 0,
               ctx->stream>>>(f.g, s.dz, s.total > 0.0 ? 1.0 / s.total : 0.0, cos_table(ctx, f.g.nz), A, (int)kind,
                              threshold, out);
  ls.done();
}
template void smv_multiplier<float>(qsm_ctx*, const Fft3<float>&, const SmvSphere&, SmvMult, double, float*);
template void smv_multiplier<double>(qsm_ctx*, const Fft3<double>&, const SmvSphere&, SmvMult, double, double*);

void smv_one_minus_transform(qsm_ctx* ctx, const GridDims& d, const SmvSphere& s, float* out) {
  Fft3<double> f = make_fft3<double>(ctx, d);
  restrict_forms(f, PassForms::kBase);
  const long long H = f.g.hsize();
  double2* S = ws<double2>(ctx, "smv.S", (size_t)H);
  run_x_r2c<double>(ctx, f, S, LoadSphere{d.nx, d.ny, d.nz, d.vsx, d.vsy, d.vsz, s.r2, s.total > 0.0 ? 1.0 / s.total : 0.0},
                    nullptr);
  run_yz<double, -1, 1>(ctx, f, S, S, OpId<double>{}, nullptr);
  run_yz<double, -1, 2>(ctx, f, S, S, OpId<double>{}, nullptr);
  LaunchScope ls(ctx, "smv_spectrum");
  k_one_minus_re<<<grid1d(H), 256, 0, ctx->stream>>>(H, S, out);
  ls.done();
}

// Spheres of `es` in `list` on top of what `first` holds, by transforms.
static void erode_by_transform(qsm_ctx* ctx, const GridDims& d, const uint8_t* mask,
                               const std::vector<SmvSphere>& spheres, const std::vector<ErodeSphere>& es,
                               const std::vector<int>& list, uint8_t* first) {
  Fft3<double> f = make_fft3<double>(ctx, d);
  const size_t H = (size_t)f.g.hsize();
  double2* F = ws<double2>(ctx, "smv.F", H);
  double2* t = ws<double2>(ctx, "smv.S", H);
  double* m = ws<double>(ctx, "smv.m64", H);
  run_x_r2c<double>(ctx, f, F, LoadCast<uint8_t, double>{mask, d.nx}, nullptr);
  run_yz<double, -1, 1>(ctx, f, F, F, OpId<double>{}, nullptr);
  run_yz<double, -1, 2>(ctx, f, F, F, OpId<double>{}, nullptr);
  for (int s : list) {
    const ErodeSphere& e = es[(size_t)s];
    smv_multiplier<double>(ctx, f, spheres[(size_t)s], kSmvS, 0.0, m);
    run_yz<double, +1, 2, true>(ctx, f, F, t, OpPreMult<double>{m}, nullptr);
    run_yz<double, +1, 1>(ctx, f, t, t, OpId<double>{}, nullptr);
    run_x_c2r<double>(ctx, f, t, StoreErode{first, d.nx, s, (double)e.total / (double)d.n, (double)e.need}, nullptr);
  }
}

void smv_erode_first(qsm_ctx* ctx, const GridDims& d, const uint8_t* mask, const std::vector<SmvSphere>& spheres,
                     double delta, uint8_t* first) {
  const int ns = (int)spheres.size();
  if (ns < 1 || ns > 254) throw QsmError(QSM_ERR_INVALID_ARGUMENT, "smv_erode_first: 1 to 254 spheres");
  const long long N = d.n;
  const int nrows = d.ny * d.nz;
  int rx = 0, ry = 0, rz = 0, lbits = -1;
  std::vector<double> r2;
  std::vector<ErodeSphere> es;
  std::vector<int4> rows;        // of the spheres that bit planes count
  std::vector<int> all, tolerant;  // spheres; those tolerating more than two missing voxels
  for (const SmvSphere& s : spheres) {
    rx = std::max(rx, s.half[0]);
    ry = std::max(ry, s.dy);
    rz = std::max(rz, s.dz);
    r2.push_back(s.r2);
    ErodeSphere e;
    e.total = (long long)s.total;
    // smallest count whose mean exceeds delta
    long long need = (long long)std::floor(delta * s.total);
    while (need > 0 && (double)(need - 1) / s.total > delta) --need;
    while (!((double)need / s.total > delta)) ++need;
    e.need = need;
    e.begin = (int)rows.size();
    e.count = 0;
    const long long tol = e.total - e.need;
    all.push_back((int)es.size());
    if (tol > 2) tolerant.push_back((int)es.size());
    if (tol == 1 || tol == 2) {
      lbits = std::max(lbits, s.half[0]);
      for (int z = 0; z <= s.dz; ++z)
        for (int y = 0; y <= s.dy; ++y) {
          const int L = s.half[(size_t)z * (s.dy + 1) + y];
          if (L < 0) break;  // the same for larger |y|
          for (int sy = 0; sy < ((y == 0 || 2 * y == d.ny) ? 1 : 2); ++sy)
            for (int sz = 0; sz < ((z == 0 || 2 * z == d.nz) ? 1 : 2); ++sz)
              rows.push_back(make_int4(sy ? -y : y, sz ? -z : z, L, 0));
        }
      e.count = (int)rows.size() - e.begin;
      // a fixed shuffle, so that the rows cut by a nearby boundary come up early: xorshift64
      // with its author's example seed (G. Marsaglia, Xorshift RNGs, 2003)
      unsigned long long rnd = 88172645463325252ull;
      for (int i = e.count - 1; i > 0; --i) {
        rnd ^= rnd << 13;
        rnd ^= rnd >> 7;
        rnd ^= rnd << 17;
        std::swap(rows[(size_t)(e.begin + i)], rows[(size_t)(e.begin + (int)(rnd % (unsigned long long)(i + 1)))]);
      }
    }
    es.push_back(e);
  }
  uint16_t* gx = ws<uint16_t>(ctx, "smv.gx", (size_t)N);
  ErodeState* st = ws<ErodeState>(ctx, "smv.state", 1);
  QSM_CUDA(cudaMemsetAsync(st, 0, sizeof(ErodeState), ctx->stream));
  {
    const size_t smem = (size_t)8 * ((d.nx + 2 * rx + 31) / 32) * sizeof(unsigned);
    const int blocks = std::min((nrows + 7) / 8, 8 * sm_count(ctx));
    LaunchScope ls(ctx, "smv_rows");
    k_smv_rows<<<blocks, 256, smem, ctx->stream>>>(d.nx, nrows, rx, mask, gx, st);
    ls.done();
  }
  ErodeState h{};
  d2h(ctx, &h, st, sizeof(h));
  sync(ctx);
  if (h.weighted) {
    QSM_CUDA(cudaMemsetAsync(first, 255, (size_t)N, ctx->stream));
    erode_by_transform(ctx, d, mask, spheres, es, all, first);
    return;
  }
  double* d2 = ws<double>(ctx, "smv.d2", (size_t)N);
  double* dr2 = ws<double>(ctx, "smv.r2", 254);
  h2d(ctx, dr2, r2.data(), r2.size() * sizeof(double));
  {
    const size_t smem = (size_t)(rx + ry + 2) * sizeof(double);
    LaunchScope ls(ctx, "smv_edt_y");
    k_smv_edt_y<<<dim3((d.nx + 31) / 32, (d.ny + 8 * kEdtU - 1) / (8 * kEdtU), d.nz), 256, smem, ctx->stream>>>(
        d.nx, d.ny, d.nz, rx, ry, d.vsx, d.vsy, gx, d2);
    ls.done();
  }
  {
    const size_t smem = (size_t)(rz + 1 + ns) * sizeof(double);
    LaunchScope ls(ctx, "smv_edt_z");
    k_smv_edt_z<<<dim3((unsigned)(((long long)d.nx * d.ny + 255) / 256), (d.nz + kEdtU - 1) / kEdtU), 256, smem,
                  ctx->stream>>>(d.nx, d.ny, d.nz, rz, d.vsz, d2, ns, dr2, first);
    ls.done();
  }
  if (lbits >= 0) {
    const int wpr = (d.nx + 31) / 32, pad = (lbits + 31) / 32, words = wpr + 2 * pad + 1;
    const long long total = (long long)nrows * wpr;
    unsigned* bits = ws_scratch<unsigned>(ctx, "smv.bits", (size_t)nrows * words);
    unsigned* planes = ws_scratch<unsigned>(ctx, "smv.planes", (size_t)3 * (lbits + 1) * total);
    ErodeSphere* des = ws<ErodeSphere>(ctx, "smv.spheres", 254);
    int4* drows = ws_scratch<int4>(ctx, "smv.rows", rows.size());
    h2d(ctx, des, es.data(), es.size() * sizeof(ErodeSphere));
    h2d(ctx, drows, rows.data(), rows.size() * sizeof(int4));
    {
      LaunchScope ls(ctx, "smv_planes");
      k_smv_bits<<<16 * sm_count(ctx), 256, 0, ctx->stream>>>(d.nx, nrows, words, pad, mask, bits);
      k_smv_planes<<<(unsigned)((total + 255) / 256), 256, 0, ctx->stream>>>(d.nx, nrows, wpr, words, pad, lbits, bits,
                                                                             planes);
      ls.done();
    }
    LaunchScope ls(ctx, "smv_count_bits");
    k_smv_count_bits<<<(unsigned)((total + 127) / 128), 128, 0, ctx->stream>>>(d.nx, d.ny, d.nz, wpr, ns, des, drows,
                                                                               planes, first);
    ls.done();
  }
  if (!tolerant.empty()) erode_by_transform(ctx, d, mask, spheres, es, tolerant, first);
}

}  // namespace qsm
