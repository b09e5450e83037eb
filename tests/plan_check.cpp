/* Host check of the launch sizes (p3x_plan.hpp): prints the number of broken
 * rules over random calls, capacities and limits. */
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "p3x_plan.hpp"

using namespace p3x;

struct Call {
  int nwork, nlev_max, pool_cols, npools, pool_end[dev::kPoolTiers - 1];
  const void* work;
};

int main() {
  std::mt19937 g(11);
  long bad = 0;
  for (int i = 0; i < 20000; ++i) {
    Call kp{};
    const int lanes = 8 << (g() % 3), num_sms = 1 + int(g() % 160), per_sm = 1 + int(g() % 4), warps_cta = 1 + int(g() % 8);
    const int limit = g() % 2 ? 0 : 1 + int(g() % 6);
    const int percent = g() % 2 ? 100 : 1 + int(g() % 100);
    const double frac = 0.01 * percent;
    kp.nwork = 1 + int(std::exp(double(g() % 1100) / 100.0));
    kp.nlev_max = 1 + int(g() % (g() % 2 ? 200 : 2903));
    kp.work = g() % 2 ? &kp : nullptr;
    /* the capacity: never more than the SMs hold, the limit and the share allow */
    const long long ctas = resident_ctas(per_sm, limit, num_sms, frac);
    bad += ctas < 1 || ctas > (long long)per_sm * num_sms;
    bad += limit && ctas > (long long)limit * num_sms;
    bad += ctas > 1 && ctas * 100 > (long long)percent * per_sm * num_sms;
    bad += !limit && frac >= 1 && ctas != (long long)per_sm * num_sms;
    /* a CTA per column only where all of them may be resident */
    bad += part12_wide_fits<double>(kp.nwork, limit, num_sms, frac) != (kp.nwork <= resident_ctas(2, limit, num_sms, frac));
    bad += part12_wide_fits<float>(kp.nwork, limit, num_sms, frac) != (kp.nwork <= resident_ctas(4, limit, num_sms, frac));
    /* pools hold every column once, in order, none larger than the list's room */
    const long long warps = ctas * warps_cta;
    plan_pools(kp, lanes, warps);
    bad += kp.pool_cols < 1 || kp.pool_cols > pool_columns(kp.nlev_max, lanes);
    int next = 0;
    for (int p = 0; p < kp.npools; ++p) {
      int w0, w1;
      dev::pool_range(kp, p, w0, w1);
      bad += w0 != next || w1 <= w0 || w1 - w0 > kp.pool_cols;
      next = w1;
    }
    bad += next != kp.nwork;
    /* few enough columns for one pool a warp, of the warps that may be resident */
    const long long share = (kp.nwork + warps - 1) / warps;
    if (!kp.work && share <= pool_columns(kp.nlev_max, lanes)) bad += kp.npools > warps || kp.pool_cols != share;
  }
  std::printf("%ld\n", bad);
}
