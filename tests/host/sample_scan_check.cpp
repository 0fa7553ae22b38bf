// Model of sample_scan_kernel (its lanes, warps and runs) on sparse sums: the scanned
// values never decrease, stay where a sum is zero, and end at the total.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "rbk_sample_scan.h"

constexpr int kThreads = 1024;

static void scan(std::vector<double>& v)
{
  const uint64_t count = v.size(), per = (count + kThreads - 1) / kThreads;
  std::vector<double> incl(kThreads), end(kThreads);
  std::vector<uint64_t> last(kThreads);
  auto lo = [&](int t) { return std::min<uint64_t>(count, uint64_t(t) * per); };
  for (int t = 0; t < kThreads; ++t) incl[t] = rbk::scan_run(v.data(), lo(t), lo(t + 1), &last[t]);
  for (int o = 1; o < 32; o <<= 1) {
    const std::vector<double> was(incl);
    for (int t = 0; t < kThreads; ++t)
      if ((t & 31) >= o) incl[t] += was[t - o];
  }
  std::vector<double> sums(32);
  for (int w = 0; w < 32; ++w) sums[w] = incl[32 * w + 31];
  for (int o = 1; o < 32; o <<= 1) {
    const std::vector<double> was(sums);
    for (int w = o; w < 32; ++w) sums[w] += was[w - o];
  }
  for (int t = 0; t < kThreads; ++t) end[t] = last[t] > lo(t) ? (t >= 32 ? sums[t / 32 - 1] + incl[t] : incl[t]) : 0.0;
  for (int o = 1; o < 32; o <<= 1) {
    const std::vector<double> was(end);
    for (int t = 0; t < kThreads; ++t)
      if ((t & 31) >= o) end[t] = rbk::scan_later(was[t - o], end[t]);
  }
  const std::vector<double> of_warp(end);
  for (int t = 0; t < kThreads; ++t) {
    double prev = 0.0;
    for (int w = 0; w < t / 32; ++w) prev = rbk::scan_later(prev, of_warp[32 * w + 31]);
    const double before = (t & 31) ? rbk::scan_later(prev, of_warp[t - 1]) : prev;
    rbk::scan_write(v.data(), lo(t), lo(t + 1), last[t], before, rbk::scan_later(prev, of_warp[t]));
  }
}

int main()
{
  std::mt19937_64 rng(3);
  std::uniform_real_distribution<double> u(0, 1);
  int decreasing = 0, moved = 0, lost = 0;
  for (int bits : {0, 1, 5, 10, 11, 12, 14, 16})
    for (double share : {1.0, 0.3, 0.05, 0.001})
      for (int run = 0; run < 20; ++run) {
        std::vector<double> sums(size_t(1) << bits);
        double total = 0;
        for (double& x : sums) total += x = u(rng) < share ? std::pow(10.0, -20.0 * u(rng) * u(rng)) : 0.0;
        std::vector<double> v(sums);
        scan(v);
        for (size_t i = 0; i < v.size(); ++i) {
          const double prev = i ? v[i - 1] : 0.0;
          decreasing += v[i] < prev;
          moved += sums[i] == 0.0 && v[i] != prev;
        }
        lost += !(std::abs(v.back() - total) <= 1e-13 * total);
      }
  // A NaN or an infinity reaches the total.
  for (double bad : {double(NAN), double(INFINITY)})
    for (size_t at : {size_t(0), size_t(100), size_t(4095)}) {
      std::vector<double> v(4096, 0.25);
      v[at] = bad;
      scan(v);
      lost += std::isfinite(v.back());
    }
  std::printf("decreasing steps %d, steps at a zero sum %d, wrong totals %d\n", decreasing, moved, lost);
  if (decreasing || moved || lost) { std::printf("FAILED\n"); return 1; }
  std::printf("ALL OK\n");
  return 0;
}
