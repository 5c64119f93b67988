// Host planner and tables of the two-factor passes (two_factor.cuh).
#include "internal.h"
#include "two_factor.cuh"

#include <cstring>

namespace qsm {

namespace {

// Largest radix run as one dense DFT.
constexpr int kTfMaxRadix = 512;

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

template <typename T> TwoFactor<T> plan_two_factor(int n) {
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
  if (n / best > kTfMaxRadix) return ax;
  ax.n = n;
  ax.ra = best;
  ax.rb = n / best;
  tf_blocks(ax.ra, &ax.kta, &ax.nka);
  tf_blocks(ax.rb, &ax.ktb, &ax.nkb);
  return ax;
}

template <typename T> std::vector<cplx_t<T>> two_factor_table(const TwoFactor<T>& ax) { return tf_twiddles<T>(ax.n); }

template <typename T> TwoFactor<T> make_two_factor(qsm_ctx* ctx, int n) {
  TwoFactor<T> ax = plan_two_factor<T>(n);
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

template TwoFactor<float> make_two_factor<float>(qsm_ctx*, int);
template TwoFactor<double> make_two_factor<double>(qsm_ctx*, int);
template TwoFactor<double> plan_two_factor<double>(int);
template std::vector<double2> two_factor_table<double>(const TwoFactor<double>&);

}  // namespace qsm
