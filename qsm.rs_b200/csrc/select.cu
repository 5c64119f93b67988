// Selection of order statistics (see select.h).
//
// Each double maps to a 64-bit key whose unsigned order is the numeric order
// (negative values: all bits flipped; others: sign bit set).  A rank is narrowed by
// sampled brackets: 2048 sampled keys are sorted by one block, the two sample keys some
// standard deviations around the rank's place bracket its value, and one pass over the
// data counts the keys below and at the bracket's ends and collects those strictly
// between them (about a tenth).  The next level does the same to what was collected, until it
// fits one block's sort, which reads the rank off.  The counts decide exactly whether the
// rank lies below, at or between the bracket's ends, so the result is the order statistic
// itself whatever the sample was; a bracket that misses it (or collects more than its
// buffer holds) sends the call to the radix passes below.  One pass reads the values once,
// where the radix selection reads them six times with its shared-memory histograms
// contended (few distinct leading digits): 37.7 M values, one rank, 1.80 ms -> 0.25 ms.
//
// Radix passes: six passes fix the key 11 bits at a time (the last pass 9 bits): a
// histogram kernel counts, per requested rank, the selected values whose higher bits equal
// the rank's prefix so far, binned by the current digit (shared-memory histograms, merged
// with global atomics); a scan kernel then picks the digit whose cumulative count covers
// the remaining rank.
#include "select.h"

#include "common.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "solvers.h"

namespace qsm {

void raise_smem_limit(const void* func, int device, size_t bytes);
int sm_count_of(int device);

namespace {

constexpr int kSelMaxRanks = 4;
constexpr int kSelBins = 2048;  // 11-bit digits
constexpr int kSelThreads = 256;

struct SelState {
  unsigned long long prefix[kSelMaxRanks];
  unsigned long long rem[kSelMaxRanks];
};

__device__ __forceinline__ unsigned long long order_key(double v) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

double key_to_double(unsigned long long k) {
  const unsigned long long u = (k >> 63) ? (k ^ 0x8000000000000000ull) : ~k;
  double d;
  std::memcpy(&d, &u, sizeof(d));
  return d;
}

__global__ void __launch_bounds__(kSelThreads)
    k_sel_hist(const double* __restrict__ vals, const uint8_t* __restrict__ mask, long long n, int nr, int shift,
               int width, const SelState* __restrict__ st, unsigned* __restrict__ hist) {
  __shared__ unsigned sh[kSelMaxRanks * kSelBins];
  for (int i = threadIdx.x; i < nr * kSelBins; i += blockDim.x) sh[i] = 0u;
  unsigned long long pre[kSelMaxRanks];
#pragma unroll
  for (int r = 0; r < kSelMaxRanks; ++r) pre[r] = r < nr ? st->prefix[r] : 0ull;
  __syncthreads();
  const int hs = shift + width;  // bits above the current digit
  const unsigned dmask = (1u << width) - 1u;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (mask != nullptr && mask[i] == 0) continue;
    const unsigned long long k = order_key(vals[i]);
    const unsigned bin = (unsigned)(k >> shift) & dmask;
#pragma unroll
    for (int r = 0; r < kSelMaxRanks; ++r) {
      if (r >= nr) break;
      const bool match = hs >= 64 || (k >> hs) == (pre[r] >> hs);
      if (match) atomicAdd(&sh[r * kSelBins + bin], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nr * kSelBins; i += blockDim.x)
    if (sh[i] != 0u) atomicAdd(&hist[i], sh[i]);
}

// One warp per rank: find the digit whose cumulative count covers the remaining rank.
__global__ void k_sel_scan(int nr, int shift, int width, SelState* st, const unsigned* __restrict__ hist) {
  const int r = threadIdx.y, lane = threadIdx.x;
  if (r >= nr) return;
  const int per = (1 << width) / 32;
  const unsigned* h = hist + r * kSelBins;
  const unsigned long long rem = st->rem[r];
  unsigned long long s = 0;
  for (int b = lane * per; b < (lane + 1) * per; ++b) s += h[b];
  unsigned long long incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const unsigned long long excl = incl - s;
  if (rem >= excl && rem < incl) {
    unsigned long long c = excl;
    for (int b = lane * per; b < (lane + 1) * per; ++b) {
      if (rem < c + h[b]) {
        st->prefix[r] |= (unsigned long long)b << shift;
        st->rem[r] = rem - c;
        break;
      }
      c += h[b];
    }
  }
}

// Bytes != 0 among mask[0, n): 16 bytes per thread and step, one atomic per block.
__global__ void __launch_bounds__(256) k_count_selected(const uint8_t* __restrict__ mask, long long n,
                                                        unsigned long long* out) {
  __shared__ unsigned long long total;
  if (threadIdx.x == 0) total = 0ull;
  __syncthreads();
  const long long head = imin((int)((16 - (reinterpret_cast<uintptr_t>(mask) & 15)) & 15), (int)(n < 16 ? n : 16));
  const long long chunks = (n - head) / 16;
  const uint4* v = reinterpret_cast<const uint4*>(mask + head);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  auto nz = [](unsigned w) { return 4 - __popc(__vcmpeq4(w, 0u) & 0x01010101u); };
  unsigned long long c = 0;
  for (long long i = t; i < chunks; i += step) {
    const uint4 q = __ldg(v + i);
    c += (unsigned)(nz(q.x) + nz(q.y) + nz(q.z) + nz(q.w));
  }
  const long long tail = head + 16 * chunks;
  if (t < head) c += mask[t] != 0;
  if (t < n - tail) c += mask[tail + t] != 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(&total, c);
  __syncthreads();
  if (threadIdx.x == 0 && total) atomicAdd(out, total);
}

// ------------------------------------------------------------ sampled brackets --
constexpr int kBrkSample = 2048;   // keys sorted by one block, a pair per thread
constexpr int kBrkThreads = kBrkSample / 2;
constexpr int kBrkMaxGroups = 2;   // rank groups per call (neighbouring ranks share one)
constexpr int kBrkStage = 2048;    // keys a block collects in shared memory before a flush

// One rank group: ranks[0..nr) among the keys of the current level.
struct BrkGroup {
  unsigned long long rank[kSelMaxRanks];
  unsigned long long value[kSelMaxRanks];  // keys found
  int found[kSelMaxRanks];
  int nr;
  int failed;
  int open;  // a bracket is set: the next pass counts and collects
  unsigned long long lo, hi;
  unsigned long long n_lt, n_lo, n_hi, n_mid;  // counted by the pass over the keys
  unsigned long long n_src;                    // keys of the level (the values at level 0)
};

struct BrkState {
  BrkGroup g[kBrkMaxGroups];
};

// lowbias32, a published 32-bit integer hash (C. Wellons, hash-prospector, 2018)
__device__ __forceinline__ unsigned hash32(unsigned x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// Ascending bitonic sort of kBrkSample keys in shared memory by the whole block, a pair of
// keys per thread and step.  For strides up to 32 a warp's pairs stay within its own 64
// keys, so only the 21 steps of stride 32 and more meet at a block barrier (all 91 steps of
// an 8192-key sort did: 90 us per bracket against 23 us).
__device__ __forceinline__ void bitonic_sort(unsigned long long* a) {
  const int t = threadIdx.x;
  for (int size = 2; size <= kBrkSample; size <<= 1)
    for (int j = size >> 1; j > 0; j >>= 1) {
      if (j >= 32) __syncthreads();
      else __syncwarp();
      const int i = 2 * t - (t & (j - 1));
      const unsigned long long x = a[i], y = a[i + j];
      const bool up = (i & size) == 0;
      if ((x > y) == up) {
        a[i] = y;
        a[i + j] = x;
      }
    }
  __syncthreads();
}

// One block per group.  Settles the ranks of the pass before (open groups), then either
// sorts all m remaining keys and reads the ranks off, or samples and sets a bracket.
// level 0: the keys are those of vals[i], mask[i] != 0 (count of them given); later
// levels: the group's collected keys.
__global__ void __launch_bounds__(kBrkThreads)
    k_sel_bracket(const double* __restrict__ vals, const uint8_t* __restrict__ mask, long long n, long long count,
                  const unsigned long long* __restrict__ keys, long long cap, int level, BrkState* st) {
  extern __shared__ __align__(16) unsigned long long srt[];
  __shared__ int ns;
  BrkGroup& G = st->g[blockIdx.x];
  keys += (long long)blockIdx.x * cap;
  if (threadIdx.x == 0) {
    ns = 0;
    if (level > 0 && G.open) {
      if (G.n_mid > (unsigned long long)cap) G.failed = 1;
      for (int r = 0; r < G.nr; ++r) {
        if (G.found[r]) continue;
        const unsigned long long k = G.rank[r];
        const unsigned long long a = G.n_lt, b = a + G.n_lo, c = b + G.n_mid, d = c + G.n_hi;
        if (k < a || k >= d) {
          G.failed = 1;
        } else if (k < b) {
          G.value[r] = G.lo;
          G.found[r] = 1;
        } else if (k < c) {
          G.rank[r] = k - b;
        } else {
          G.value[r] = G.hi;
          G.found[r] = 1;
        }
      }
    }
    int left = 0;
    for (int r = 0; r < G.nr; ++r) left += G.found[r] == 0;
    G.open = left > 0 && !G.failed;
  }
  __syncthreads();
  if (!G.open) return;
  const unsigned long long m = level > 0 ? G.n_mid : (unsigned long long)count;
  const bool all = level > 0 && m <= kBrkSample;
  if (all) {
    for (int i = threadIdx.x; i < kBrkSample; i += kBrkThreads) srt[i] = i < (int)m ? keys[i] : ~0ull;
  } else if (level == 0 && m <= kBrkSample) {
    // few values selected: collect them all, the next level sorts them
    __syncthreads();
    if (threadIdx.x == 0) {
      G.lo = 0ull;
      G.hi = ~0ull;
      G.n_lt = G.n_lo = G.n_hi = G.n_mid = 0ull;
    }
    return;
  } else {
    const unsigned long long total = level > 0 ? m : (unsigned long long)n;
    for (int s = threadIdx.x; s < kBrkSample; s += kBrkThreads) {
      // a hashed place in the s-th of kBrkSample equal stretches; a few tries where the
      // mask leaves some out
      const unsigned long long b0 = (unsigned long long)s * total / kBrkSample;
      const unsigned long long b1 = (unsigned long long)(s + 1) * total / kBrkSample;
      for (unsigned t = 0; t < 8; ++t) {
        const unsigned long long i = b0 + hash32((unsigned)s * 8u + t + 77u * (unsigned)level) % (b1 - b0);
        if (level == 0 && mask != nullptr && mask[i] == 0) continue;
        srt[atomicAdd(&ns, 1)] = level > 0 ? keys[i] : order_key(vals[i]);
        break;
      }
    }
    __syncthreads();
    for (int i = ns + threadIdx.x; i < kBrkSample; i += kBrkThreads) srt[i] = ~0ull;
  }
  __syncthreads();
  bitonic_sort(srt);
  if (threadIdx.x != 0) return;
  if (all) {
    for (int r = 0; r < G.nr; ++r)
      if (!G.found[r]) {
        G.value[r] = srt[G.rank[r]];
        G.found[r] = 1;
      }
    G.open = 0;
    return;
  }
  if (ns < 64) {
    G.failed = 1;
    G.open = 0;
    return;
  }
  unsigned long long first = ~0ull, last = 0ull;
  for (int r = 0; r < G.nr; ++r)
    if (!G.found[r]) {
      first = G.rank[r] < first ? G.rank[r] : first;
      last = G.rank[r] > last ? G.rank[r] : last;
    }
  const double f0 = (double)first / (double)m, f1 = (double)(last + 1) / (double)m;
  const double w0 = 5.0 * sqrt(ns * f0 * (1.0 - f0)) + 2.0, w1 = 5.0 * sqrt(ns * fmax(f1 * (1.0 - f1), 0.0)) + 2.0;
  const double p0 = floor(ns * f0 - w0), p1 = ceil(ns * f1 + w1);
  G.lo = p0 < 0.0 ? 0ull : srt[(int)p0];
  G.hi = p1 >= (double)ns ? ~0ull : srt[(int)p1];
  G.n_src = m;
  G.n_lt = G.n_lo = G.n_hi = G.n_mid = 0ull;
}

// Count the keys below and at the ends of every open group's bracket and collect those
// strictly inside.  Level 0 reads the values; later levels one group's keys per blockIdx.y.
template <bool VALUES>
__global__ void __launch_bounds__(256)
    k_sel_collect(const double* __restrict__ vals, const uint8_t* __restrict__ mask, long long n,
                  const unsigned long long* __restrict__ keys, unsigned long long* __restrict__ out, long long cap,
                  int ngroups, BrkState* st) {
  __shared__ unsigned long long stage[kBrkMaxGroups][kBrkStage];
  __shared__ unsigned fill[kBrkMaxGroups];
  __shared__ unsigned long long place;
  const int g0 = VALUES ? 0 : blockIdx.y, g1 = VALUES ? ngroups : blockIdx.y + 1;
  unsigned long long lo[kBrkMaxGroups], hi[kBrkMaxGroups];
  unsigned lt[kBrkMaxGroups], el[kBrkMaxGroups], eh[kBrkMaxGroups];
  bool open[kBrkMaxGroups], any = false;
#pragma unroll
  for (int g = 0; g < kBrkMaxGroups; ++g) {
    open[g] = g >= g0 && g < g1 && st->g[g].open;
    any |= open[g];
    lo[g] = open[g] ? st->g[g].lo : ~0ull;
    hi[g] = open[g] ? st->g[g].hi : 0ull;
    lt[g] = el[g] = eh[g] = 0u;
  }
  if (!any) return;
  if (threadIdx.x < kBrkMaxGroups) fill[threadIdx.x] = 0u;
  __syncthreads();
  auto flush = [&](int g) {  // whole block
    const unsigned have = fill[g] < (unsigned)kBrkStage ? fill[g] : (unsigned)kBrkStage;
    if (threadIdx.x == 0) place = atomicAdd(&st->g[g].n_mid, (unsigned long long)have);
    __syncthreads();
    const unsigned long long p = place;
    for (unsigned i = threadIdx.x; i < have; i += blockDim.x)
      if (p + i < (unsigned long long)cap) out[g * cap + (long long)(p + i)] = stage[g][i];
    __syncthreads();
    if (threadIdx.x == 0) fill[g] = 0u;
    __syncthreads();
  };
  const long long total = VALUES ? n : (long long)st->g[g0].n_src;
  constexpr int U = 4;
  const long long span = (long long)blockDim.x * U;
  for (long long base = (long long)blockIdx.x * span; base < total; base += (long long)gridDim.x * span) {
    unsigned long long k[U];
    bool ok[U];
    if constexpr (VALUES) {
      uint8_t mk_[U];
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long i = base + u * (long long)blockDim.x + threadIdx.x;
        mk_[u] = i < total ? (mask != nullptr ? mask[i] : (uint8_t)1) : (uint8_t)0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long i = base + u * (long long)blockDim.x + threadIdx.x;
        v[u] = mk_[u] ? vals[i] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        ok[u] = mk_[u] != 0;
        k[u] = order_key(v[u]);
      }
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long i = base + u * (long long)blockDim.x + threadIdx.x;
        ok[u] = i < total;
        k[u] = ok[u] ? keys[g0 * cap + i] : 0ull;
      }
    }
#pragma unroll
    for (int g = 0; g < kBrkMaxGroups; ++g) {
      if (!open[g]) continue;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!ok[u]) continue;
        lt[g] += k[u] < lo[g];
        el[g] += k[u] == lo[g];
        eh[g] += k[u] == hi[g] && hi[g] != lo[g];
        if (k[u] > lo[g] && k[u] < hi[g]) {
          const unsigned at = atomicAdd(&fill[g], 1u);
          stage[g][at] = k[u];  // at < kBrkStage: flushed below while a whole step still fits
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < kBrkMaxGroups; ++g)
      if (open[g] && fill[g] + (unsigned)span > (unsigned)kBrkStage) flush(g);
    __syncthreads();
  }
#pragma unroll
  for (int g = 0; g < kBrkMaxGroups; ++g) {
    if (!open[g]) continue;
    if (fill[g] > 0) flush(g);
    for (int o = 16; o > 0; o >>= 1) {
      lt[g] += __shfl_down_sync(0xffffffffu, lt[g], o);
      el[g] += __shfl_down_sync(0xffffffffu, el[g], o);
      eh[g] += __shfl_down_sync(0xffffffffu, eh[g], o);
    }
    if ((threadIdx.x & 31) == 0) {
      if (lt[g]) atomicAdd(&st->g[g].n_lt, (unsigned long long)lt[g]);
      if (el[g]) atomicAdd(&st->g[g].n_lo, (unsigned long long)el[g]);
      if (eh[g]) atomicAdd(&st->g[g].n_hi, (unsigned long long)eh[g]);
    }
  }
}

}  // namespace

long long count_selected(qsm_ctx* ctx, const uint8_t* mask, long long n) {
  if (mask == nullptr) return n;
  unsigned long long* d = ws<unsigned long long>(ctx, "sel.count", 1);
  QSM_CUDA(cudaMemsetAsync(d, 0, sizeof(unsigned long long), ctx->stream));
  {
    LaunchScope ls(ctx, "count_selected");
    k_count_selected<<<grid1d((n + 15) / 16), 256, 0, ctx->stream>>>(mask, n, d);
    ls.done();
  }
  unsigned long long h = 0;
  d2h(ctx, &h, d, sizeof(h));
  sync(ctx);
  return (long long)h;
}

namespace {

// The sampled brackets; false when a bracket missed its rank or their key buffers (4 bytes a
// value) cannot be had: the caller then runs the radix passes.  count: values selected by the
// mask.
bool bracket_ranks(qsm_ctx* ctx, const double* vals, const uint8_t* mask, long long n, long long count,
                   const std::vector<long long>& ranks, std::vector<double>& out) {
  BrkState h{};
  int ng = 0;
  std::vector<std::pair<int, int>> at;  // (group, place) of each rank
  for (size_t r = 0; r < ranks.size(); ++r) {
    if (r == 0 || ranks[r] < ranks[r - 1] || ranks[r] > ranks[r - 1] + 1) {
      if (ng == kBrkMaxGroups) return false;
      ++ng;
    }
    BrkGroup& G = h.g[ng - 1];
    at.emplace_back(ng - 1, G.nr);
    G.rank[G.nr++] = (unsigned long long)ranks[r];
  }
  const long long cap = std::max<long long>(kBrkSample, n / 8);
  BrkState* st = ws<BrkState>(ctx, "sel.brk", 1);
  unsigned long long* buf[2];
  try {
    for (int i = 0; i < 2; ++i)
      buf[i] = ws<unsigned long long>(ctx, i ? "sel.keys1" : "sel.keys0", (size_t)cap * kBrkMaxGroups);
  } catch (const QsmError& e) {  // the radix passes need no such buffers
    if (e.code != QSM_ERR_ALLOC) throw;
    return false;
  }
  h2d(ctx, st, &h, sizeof(h));
  const size_t smem = kBrkSample * sizeof(unsigned long long);
  raise_smem_limit(reinterpret_cast<const void*>(k_sel_bracket), ctx->device, smem);
  // passes until what a bracket is expected to hold fits one sort with a third to spare: its
  // width at the ranks' place (of the sample, the stretches outside the mask give nothing),
  // then at the middle, where the ranks lie among collected keys.  A count that still does
  // not fit leaves the ranks to the radix passes; an extra pass over a few thousand keys
  // costs 30 us, the radix passes over 37.7 M voxels 600 us.
  auto width = [](double p, double ns) { return std::min(1.0, 2.2 * (5.0 * std::sqrt(ns * p * (1.0 - p)) + 2.0) / ns); };
  const double ns0 = std::max(64.0, (double)kBrkSample * (double)count / (double)std::max(n, 1LL));
  double left = 0.0;
  for (long long r : ranks) left = std::max(left, (double)count * width((double)r / (double)std::max(count, 1LL), ns0));
  int passes = 1;
  for (; left > 0.67 * kBrkSample && count > kBrkSample && passes < 12; left *= width(0.5, kBrkSample)) ++passes;
  for (int level = 0; level <= passes; ++level) {
    {
      LaunchScope ls(ctx, "select_bracket");
      k_sel_bracket<<<ng, kBrkThreads, smem, ctx->stream>>>(vals, mask, n, count, buf[(level + 1) & 1], cap, level, st);
      ls.done();
    }
    if (level == passes) break;
    LaunchScope ls(ctx, "select_collect");
    if (level == 0) {
      const long long blocks = std::min<long long>((n + 1023) / 1024, 8LL * sm_count_of(ctx->device));
      k_sel_collect<true><<<(unsigned)std::max(blocks, 1LL), 256, 0, ctx->stream>>>(vals, mask, n, nullptr, buf[0], cap,
                                                                                    ng, st);
    } else {
      k_sel_collect<false><<<dim3((unsigned)sm_count_of(ctx->device), ng), 256, 0, ctx->stream>>>(
          nullptr, nullptr, 0, buf[(level + 1) & 1], buf[level & 1], cap, ng, st);
    }
    ls.done();
  }
  d2h(ctx, &h, st, sizeof(h));
  sync(ctx);
  out.resize(ranks.size());
  for (size_t r = 0; r < ranks.size(); ++r) {
    const BrkGroup& G = h.g[at[r].first];
    if (G.failed || !G.found[at[r].second]) return false;
    out[r] = key_to_double(G.value[at[r].second]);
  }
  return true;
}

}  // namespace

std::vector<double> select_ranks(qsm_ctx* ctx, const double* vals, const uint8_t* mask, long long n, long long count,
                                 const std::vector<long long>& ranks) {
  const int nr = (int)ranks.size();
  if (nr < 1 || nr > kSelMaxRanks) throw QsmError(QSM_ERR_INVALID_ARGUMENT, "select_ranks: 1 to 4 ranks");
  for (long long r : ranks)
    if (r < 0) throw QsmError(QSM_ERR_INVALID_ARGUMENT, "select_ranks: negative rank");
  std::vector<double> got;
  if (bracket_ranks(ctx, vals, mask, n, count, ranks, got)) return got;
  SelState h{};
  for (int r = 0; r < nr; ++r) h.rem[r] = (unsigned long long)ranks[r];
  SelState* st = ws<SelState>(ctx, "sel.state", 1);
  unsigned* hist = ws<unsigned>(ctx, "sel.hist", (size_t)kSelMaxRanks * kSelBins);
  h2d(ctx, st, &h, sizeof(h));
  int sm = 0;
  QSM_CUDA(cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, ctx->device));
  long long blocks = (n + kSelThreads - 1) / kSelThreads;
  if (blocks > 2LL * sm) blocks = 2LL * sm;
  if (blocks < 1) blocks = 1;
  static const int kShift[6] = {53, 42, 31, 20, 9, 0};
  static const int kWidth[6] = {11, 11, 11, 11, 11, 9};
  for (int p = 0; p < 6; ++p) {
    QSM_CUDA(cudaMemsetAsync(hist, 0, sizeof(unsigned) * nr * kSelBins, ctx->stream));
    {
      LaunchScope ls(ctx, "select_hist");
      k_sel_hist<<<(unsigned)blocks, kSelThreads, 0, ctx->stream>>>(vals, mask, n, nr, kShift[p], kWidth[p], st,
                                                                    hist);
      ls.done();
    }
    {
      LaunchScope ls(ctx, "select_scan");
      k_sel_scan<<<1, dim3(32, nr), 0, ctx->stream>>>(nr, kShift[p], kWidth[p], st, hist);
      ls.done();
    }
  }
  d2h(ctx, &h, st, sizeof(h));
  sync(ctx);
  std::vector<double> out(nr);
  for (int r = 0; r < nr; ++r) out[r] = key_to_double(h.prefix[r]);
  return out;
}

std::vector<double> percentiles(qsm_ctx* ctx, const double* vals, const uint8_t* mask, long long n,
                                long long count, const std::vector<double>& p) {
  if (count <= 0) throw QsmError(QSM_ERR_INVALID_ARGUMENT, "percentiles of an empty selection");
  if (p.size() > 2) throw QsmError(QSM_ERR_INVALID_ARGUMENT, "percentiles: at most two per call");
  std::vector<double> out(p.size());
  if (count == 1) {
    const std::vector<double> v = select_ranks(ctx, vals, mask, n, count, {0});
    for (size_t i = 0; i < p.size(); ++i) out[i] = v[0];
    return out;
  }
  std::vector<long long> ranks;
  std::vector<double> frac;
  for (double pi : p) {
    const double hpos = (pi / 100.0) * (double)(count - 1);
    const long long lo = (long long)std::floor(hpos);
    const long long hi = std::min(lo + 1, count - 1);
    ranks.push_back(lo);
    ranks.push_back(hi);
    frac.push_back(hpos - (double)lo);
  }
  const std::vector<double> v = select_ranks(ctx, vals, mask, n, count, ranks);
  for (size_t i = 0; i < p.size(); ++i) {
    const double lo = v[2 * i], hi = v[2 * i + 1];
    out[i] = lo + frac[i] * (hi - lo);
  }
  return out;
}

}  // namespace qsm

using namespace qsm;

extern "C" qsm_status qsm_prctile_device(qsm_ctx* ctx, const double* d_vals, const uint8_t* d_mask, size_t n,
                                         const double* p, size_t np, double* out) {
  return guarded(ctx, [&] {
    if (np == 0) return;
    check_ptr(p, "p");
    check_ptr(out, "out");
    if (n > 0) check_ptr(d_vals, "vals");
    const long long count = n == 0 ? 0 : count_selected(ctx, d_mask, (long long)n);
    for (size_t i = 0; i < np; i += 2) {
      std::vector<double> pi(p + i, p + std::min(np, i + 2));
      for (double v : pi)
        if (!(v >= 0.0 && v <= 100.0)) throw QsmError(QSM_ERR_INVALID_ARGUMENT, "percent outside [0, 100]");
      if (count == 0) {
        for (size_t k = 0; k < pi.size(); ++k) out[i + k] = 0.0;
        continue;
      }
      const std::vector<double> r = percentiles(ctx, d_vals, d_mask, (long long)n, count, pi);
      for (size_t k = 0; k < r.size(); ++k) out[i + k] = r[k];
    }
  });
}
