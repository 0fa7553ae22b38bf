// rbk::simplify_queue on random queues of every gate form: the state it gives
// equals the original's, gates that are not plain unitaries included; and the
// matrices it makes of rotations close to pi are as exact as those it is given.
#include <cmath>
#include <complex>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "rbk_plan.h"

using cd = std::complex<double>;

template <typename C>
static void apply(std::vector<C>& a, const rbk::hgate& g)
{
  auto at = [](const double* m, int k) { return C(m[2 * k], m[2 * k + 1]); };
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
    const C x = a[i], y = a[i | t];
    if (g.kind == rbk::OPK_X) { a[i] = y; a[i | t] = x; }
    else if (g.kind == rbk::OPK_Y) { a[i] = C{y.imag(), -y.real()}; a[i | t] = C{-x.imag(), x.real()}; }
    else { a[i] = at(g.m, 0) * x + at(g.m, 1) * y; a[i | t] = at(g.m, 2) * x + at(g.m, 3) * y; }
  }
}

// Chains of U3, CZ, U3, CNOT on 2 qubits with |cos(theta / 2)| from 1e-3 to 1, whose
// matrices take phases and X rotations from one another.  Every simplified matrix is a
// product of at most 4 of some 4 roundings each: 16 * 1.1e-16 in each entry, twice
// that in its unitarity.  The states are evaluated in long double, so that their
// distance is the matrices' rounding alone, which adds up over 24 gates like a random
// walk: 5 * 16 * 1.1e-16.
static bool precise_near_pi()
{
  using cl = std::complex<long double>;
  std::mt19937_64 rng(5);
  std::uniform_real_distribution<double> u(-3.2, 3.2), e(-3.0, 0.0);
  double defect = 0;
  long double distance = 0;
  for (int run = 0; run < 20000; ++run) {
    std::vector<rbk::hgate> q;
    for (int k = 0; k < 12; ++k) {
      for (int b = 0; b < 2; ++b) {
        rbk::hgate g{};
        g.kind = rbk::OPK_MAT;
        g.target = int8_t(b);
        g.target2 = -1;
        const double c = std::pow(10.0, e(rng)), s = std::sqrt((1.0 - c) * (1.0 + c)), p = u(rng), l = u(rng);
        const cd v[4] = {c, -s * std::polar(1.0, l), s * std::polar(1.0, p), c * std::polar(1.0, p + l)};
        for (int i = 0; i < 4; ++i) { g.m[2 * i] = v[i].real(); g.m[2 * i + 1] = v[i].imag(); }
        q.push_back(g);
      }
      rbk::hgate g{};
      g.target2 = -1;
      const bool cz = rng() % 2;
      g.kind = cz ? rbk::OPK_NEG : rbk::OPK_X;
      g.target = cz ? int8_t(-1) : int8_t(rng() % 2);
      g.cmask = cz ? 3ull : 1ull << (1 - g.target);
      q.push_back(g);
    }
    const auto s = rbk::simplify_queue(2, q);
    for (const auto& g : s) {
      if (g.kind != rbk::OPK_MAT) continue;
      const cl a(g.m[0], g.m[1]), b(g.m[2], g.m[3]), c(g.m[4], g.m[5]), d(g.m[6], g.m[7]);
      defect = std::max({defect, double(std::abs(std::norm(a) + std::norm(b) - 1)), double(std::abs(std::norm(c) + std::norm(d) - 1)),
                         double(std::abs(a * std::conj(c) + b * std::conj(d)))});
    }
    std::vector<cl> x(4), y;
    for (auto& v : x) v = cl{u(rng), u(rng)};
    y = x;
    long double norm = 0, err = 0;
    for (const auto& v : x) norm += std::norm(v);
    for (const auto& g : q) apply(x, g);
    for (const auto& g : s) apply(y, g);
    for (size_t i = 0; i < x.size(); ++i) err += std::norm(x[i] - y[i]);
    distance = std::max(distance, std::sqrt(err / norm));
  }
  std::printf("rotations close to pi: unitarity defect %.3g, distance %.3Lg\n", defect, distance);
  return defect <= 32 * 1.1e-16 && distance <= 80 * 1.1e-16L;
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
  if (!precise_near_pi()) { std::printf("FAILED\n"); return 1; }
  std::printf("ALL OK\n");
  return 0;
}
