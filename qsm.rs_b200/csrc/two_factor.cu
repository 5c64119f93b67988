// Host planner and tables of the two-factor passes (two_factor.cuh).
#include "internal.h"
#include "two_factor.cuh"

#include <cstring>

namespace qsm {

namespace {

// Lengths that take the dense passes, n = ra * rb with rb the larger radix.
//
// Lengths with prime factors up to 13 have the run-time Stockham engine (and 32..384 a
// compile-time plan, so the dense form carries only their functors in small volumes): above
// 384 the dense passes lose to it (n x 128 x 128, us, dense against Stockham, X r2c / Y / Z:
// 448 double 107/87/197 and 72/60/127, float 78/59/140 and 39/45/79; 512 double 117/108/247
// and 83/66/140; 400 float 61/39/87 and 39/43/78).
//
// For the others the alternative is a Bluestein convolution, and the dense sum's error and
// time both grow with rb.  Float: the relative error against 80-bit transforms passes
// Bluestein's between rb = 139 (1.90e-7 and 1.91e-7) and 173 (2.05e-7 and 1.94e-7; 1.12 times
// at 197, 1.3 at 367); up to 139 every pass is also the faster one at all lengths measured to
// 867, but Z at 508 (274 us against 248).  Double: the error stays below Bluestein's up to
// rb = 367 (0.97 times; 1.02 at 373), and the passes are faster up to there (353: X 187 and
// 238, Y 205 and 319, Z 435 and 447) while two blocks fit an SM (n <= 427).  Beyond, the Z
// pass falls back with rb over 139 (447: 491 against 464, 478: 698 against 501) and the X
// passes over 241 (482: 286 against 312, 526: 292 against 271); Y keeps its lead (706: 542
// against 633).
template <typename T> bool tf_takes(int n, int rb, int axis) {
  int m = n;
  for (int p : {2, 3, 5, 7, 11, 13})
    while (m % p == 0) m /= p;
  if (m == 1) return n <= 384;
  if (sizeof(T) == 4) return rb <= 139;
  return rb <= (n <= 427 || axis == 1 ? 367 : axis == 0 ? 241 : 139);
}

// Sets of output frequencies of a radix-r DFT: nk sets of 4 * kt cover 0..r/2.
void tf_blocks(int r, int* kt, int* nk) {
  const int k = r / 2 + 1;
  *nk = (k + 4 * kTfMaxKT - 1) / (4 * kTfMaxKT);
  *kt = (k + 4 * *nk - 1) / (4 * *nk);
}

// Floating-point work per element of a dense stage (sums and differences once per set and
// frequency block, two multiply-adds per frequency slot) plus its fixed work.
int tf_cost(int r) {
  if (r == 1) return 0;
  int kt, nk;
  tf_blocks(r, &kt, &nk);
  return 8 * nk + 8 * kt * nk + 10;
}

template <typename T> std::vector<cplx_t<T>> tf_twiddles(int n) {
  using C = cplx_t<T>;
  std::vector<C> w((size_t)n);
  for (int k = 0; k < n; ++k) w[(size_t)k] = mk<C>((T)cos2pi(k, n), (T)-sin2pi(k, n));
  return w;
}

}  // namespace

template <typename T> TwoFactor<T> plan_two_factor(int n, int axis) {
  TwoFactor<T> ax{};
  if (n < 2) return ax;
  int best = 0, cost = 0;
  for (int a = 1; a * a <= n; ++a) {
    if (n % a != 0) continue;
    const int c = tf_cost(a) + tf_cost(n / a);
    if (best == 0 || c < cost) {
      best = a;
      cost = c;
    }
  }
  if (!tf_takes<T>(n, n / best, axis)) return ax;
  ax.n = n;
  ax.ra = best;
  ax.rb = n / best;
  tf_blocks(ax.ra, &ax.kta, &ax.nka);
  tf_blocks(ax.rb, &ax.ktb, &ax.nkb);
  return ax;
}

template <typename T> std::vector<cplx_t<T>> two_factor_table(const TwoFactor<T>& ax) { return tf_twiddles<T>(ax.n); }

template <typename T> TwoFactor<T> make_two_factor(qsm_ctx* ctx, int n, int axis) {
  TwoFactor<T> ax = plan_two_factor<T>(n, axis);
  if (ax.n == 0) return ax;
  const std::string key = "tf:" + std::to_string(n) + (sizeof(T) == 4 ? ":f" : ":d");
  auto it = ctx->tables.find(key);
  if (it != ctx->tables.end()) {
    ax.tw = static_cast<const cplx_t<T>*>(it->second);
    return ax;
  }
  const std::vector<cplx_t<T>> h = two_factor_table(ax);
  ax.tw = static_cast<const cplx_t<T>*>(upload_table(ctx, key, h.data(), h.size() * sizeof(cplx_t<T>)));
  return ax;
}

template TwoFactor<float> make_two_factor<float>(qsm_ctx*, int, int);
template TwoFactor<double> make_two_factor<double>(qsm_ctx*, int, int);
template TwoFactor<double> plan_two_factor<double>(int, int);
template std::vector<double2> two_factor_table<double>(const TwoFactor<double>&);

}  // namespace qsm
