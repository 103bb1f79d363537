// Which of the batched domains that fit in an SM's shared memory stay there.
//
// A domain in shared memory is stepped by one SM and is the fastest way to
// step many (148 domains of 100x100 in FP16: 14.7 us a step, 100 GLUPS, over
// every SM 20.9).  It cannot be split, though: one of 100x100 alone takes the
// same time, and 3.0 us over every SM.  So the largest ones go wide as long as
// that shortens the estimated step, the longer of
//
//   the busiest SM: a domain of n nodes takes one(n) = 0.4 us + 1.38 ns n, and
//   1.2 us more beside wide launches; domains are taken largest first, so the
//   one that starts round j is no larger than any of rounds 1 .. j;
//   the work: one(n) of those that stay, over all SMs, and 2.7 us + 1/78 ns a
//   node for the wide launches.
//
// Measured (us a step, all in shared memory / the largest wide as chosen / all
// wide): 100 of 48x48 FP32 3.9 / 3.9 / 5.7, 130 of 78x78 FP16 8.8 / 8.8 / 13.1,
// 170 of 100x100 FP16 27.4 / 18.9 / 25.5, 20 of 110x110 FP16 16.8 / 6.0 / 6.0,
// 1 of 48x48 3.8 / 2.8 / 2.8, 250 of 32..128 FP16 18.3 / 15.0 / 19.2.  A batch
// that needs no wide launches yet gets them for a tenth and more only.
#pragma once

#include <algorithm>
#include <vector>

namespace lbmc {

// fit: nodes of the domains that fit, largest first; rest: nodes of the
// others, which are stepped from HBM whatever is chosen; share: 3/4 of an SM's
// share of all nodes.  Returns how many of the largest go wide.
inline size_t wide_of_fitting(const std::vector<long long> &fit, long long rest, long long share, int sms) {
  constexpr double ONE_BASE = 400, NODE = 1.38, BESIDE_WIDE = 1200, WIDE_BASE = 2700, WIDE_NODE = 1.0 / 78;
  constexpr double MARGIN = 1.1, SHARE_MARGIN = 1.15;
  auto one = [](long long n) { return ONE_BASE + NODE * (double)n; };
  const size_t count = fit.size();
  std::vector<double> stay(count + 1, 0.0), go(count + 1, (double)rest);  // of the first i gone wide
  for (size_t i = count; i-- > 0;) stay[i] = stay[i + 1] + one(fit[i]);
  for (size_t i = 0; i < count; i++) go[i + 1] = go[i] + (double)fit[i];
  auto work = [&](size_t i) { return stay[i] / sms + (go[i] > 0 ? WIDE_BASE + WIDE_NODE * go[i] : 0); };
  auto busiest = [&](size_t i) {
    double t = 0;
    for (size_t j = 0; i + j * sms < count; j++) t = std::max(t, (double)(j + 1) * one(fit[i + j * sms]));
    return t > 0 && go[i] > 0 ? t + BESIDE_WIDE : t;
  };
  auto step = [&](size_t i) { return std::max(busiest(i), work(i)); };
  size_t chosen = 0;
  double best = rest > 0 ? step(0) : step(0) / MARGIN;
  // Once the work is the longer part, it only grows.
  for (size_t i = 0; i < count && !(go[i] > 0 && work(i) >= busiest(i)); i++)
    if (step(i + 1) < best) {
      best = step(i + 1);
      chosen = i + 1;
    }
  // Beside larger domains, which are wide, the share is the better line where
  // the estimates are close (40 of 32..512 FP16: 15.1 us a step, 16.6 by the
  // estimate).
  if (rest > 0) {
    size_t above = 0;
    while (above < count && fit[above] > share) above++;
    if (step(above) <= SHARE_MARGIN * best) chosen = above;
  }
  return chosen;
}

}  // namespace lbmc
