// rbk::simplify_queue on random queues of every gate form: the state it gives
// equals the original's, gates that are not plain unitaries included.
#include <cmath>
#include <complex>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "rbk_plan.h"

using cd = std::complex<double>;

static cd at(const double* m, int k) { return {m[2 * k], m[2 * k + 1]}; }

static void apply(std::vector<cd>& a, const rbk::hgate& g)
{
  for (uint32_t i = 0; i < a.size(); ++i) {
    if (g.kind == rbk::HK_SWAP) {
      const uint32_t x = 1u << g.target, y = 1u << g.target2;
      if ((i & x) && !(i & y)) std::swap(a[i], a[i ^ x ^ y]);
      continue;
    }
    if ((i & g.cmask) != g.cmask) continue;
    if (g.kind == rbk::OPK_NEG) { a[i] = -a[i]; continue; }
    const uint32_t t = 1u << g.target;
    if (g.kind == rbk::OPK_DIAG) {
      if (i & t) a[i] *= at(g.m, 1);
      else if (!g.diag_one) a[i] *= at(g.m, 0);
      continue;
    }
    if (i & t) continue;
    const cd x = a[i], y = a[i | t];
    if (g.kind == rbk::OPK_X) { a[i] = y; a[i | t] = x; }
    else if (g.kind == rbk::OPK_Y) { a[i] = cd{y.imag(), -y.real()}; a[i | t] = cd{-x.imag(), x.real()}; }
    else { a[i] = at(g.m, 0) * x + at(g.m, 1) * y; a[i | t] = at(g.m, 2) * x + at(g.m, 3) * y; }
  }
}

int main()
{
  std::mt19937_64 rng(11);
  std::uniform_real_distribution<double> u(-3.2, 3.2);
  double worst = 0;
  size_t before = 0, after = 0;
  for (int run = 0; run < 400; ++run) {
    const int n = 1 + int(rng() % 6);
    std::vector<rbk::hgate> q;
    for (int k = 0; k < 60; ++k) {
      rbk::hgate g{};
      g.target = int8_t(rng() % n);
      g.target2 = -1;
      const int controls = n > 1 ? int(rng() % 5) - 2 : 0;
      for (int c = 0; c < controls; ++c) {
        const int b = int(rng() % n);
        if (b != g.target) g.cmask |= 1ull << b;
      }
      const double th = rng() % 9 == 0 ? 3.14159265358979312 * int(rng() % 3) / 2 : u(rng), p = u(rng), l = u(rng);
      const cd e1 = std::polar(1.0, p), e2 = std::polar(1.0, l);
      auto put = [&](cd a, cd b, cd c, cd d) {
        const cd v[4] = {a, b, c, d};
        for (int e = 0; e < 4; ++e) { g.m[2 * e] = v[e].real(); g.m[2 * e + 1] = v[e].imag(); }
      };
      switch (rng() % 9) {
        case 0: g.kind = rbk::OPK_X; break;
        case 1: g.kind = rbk::OPK_Y; break;
        case 2: g.kind = rbk::OPK_NEG; g.cmask |= 1ull << g.target; g.target = -1; break;
        case 3:
          g.kind = rbk::OPK_DIAG;
          g.diag_one = rng() % 2;
          g.m[0] = g.diag_one ? 1.0 : e1.real(); g.m[1] = g.diag_one ? 0.0 : e1.imag();
          g.m[2] = e2.real(); g.m[3] = e2.imag();
          break;
        case 4: g.kind = rbk::OPK_MAT; put(std::cos(th), std::sin(th), -std::sin(th), std::cos(th)); break;   // real
        case 5:
          if (rng() % 8 == 0) {  // not unitary
            g.kind = rbk::OPK_MAT;
            put({0.3, 0.1}, {0.2, -0.4}, {1.1, 0.2}, {-0.5, 0.6});
            break;
          }
          if (n > 1 && rng() % 2) { g.kind = rbk::HK_SWAP; g.cmask = 0; g.target2 = int8_t((g.target + 1 + rng() % (n - 1)) % n); break; }
          [[fallthrough]];
        default:
          g.kind = rbk::OPK_MAT;
          put(std::cos(th / 2), -std::sin(th / 2) * e2, std::sin(th / 2) * e1, std::cos(th / 2) * e1 * e2);
      }
      q.push_back(g);
    }
    const auto s = rbk::simplify_queue(n, q);
    before += q.size();
    after += s.size();
    std::vector<cd> a(1u << n), b;
    for (auto& x : a) x = cd{u(rng), u(rng)};
    b = a;
    for (const auto& g : q) apply(a, g);
    for (const auto& g : s) apply(b, g);
    double norm = 0, err = 0;
    for (size_t i = 0; i < a.size(); ++i) { norm = std::max(norm, std::abs(a[i])); err = std::max(err, std::abs(a[i] - b[i])); }
    worst = std::max(worst, err / norm);
  }
  std::printf("gates %zu -> %zu, worst relative error %.3g\n", before, after, worst);
  // 60 gates of some 1e-16 each; a non-unitary gate may shrink the state against its rounding by 1e2
  if (!(worst < 1e-12) || after >= before) { std::printf("FAILED\n"); return 1; }
  std::printf("ALL OK\n");
  return 0;
}
