// CPU model of small_circuit_kernel over the programs of rbk::plan_small: every
// phase through the kernel's index arithmetic (swizzled slots, register and base
// masks), against the gates applied one by one to a logical state.  Then the time
// that planning a long queue takes where a qubit is never a target.
#include <complex>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <ctime>
#include <random>
#include <set>
#include <vector>

#include "rbk_plan.h"

using cd = std::complex<double>;

static uint32_t slot(uint32_t u) { return u ^ (((u >> 3) ^ (u >> 6) ^ (u >> 9) ^ (u >> 12)) & 7u); }
static uint32_t insert_zero(uint32_t v, int q) { return ((v & ~((1u << q) - 1)) << 1) | (v & ((1u << q) - 1)); }
static cd at(const double* m, int k) { return {m[2 * k], m[2 * k + 1]}; }

static void apply_direct(std::vector<cd>& a, const rbk::hgate& g)
{
  for (uint32_t i = 0; i < a.size(); ++i) {
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

static void fail(const char* what) { std::printf("FAILED: %s\n", what); std::exit(1); }

static void run_program(std::vector<cd>& phys, int n, const rbk::small_program& p)
{
  constexpr int R = rbk::kSmallRegBits, NR = 1 << R;
  const uint32_t size = 1u << n, padded = size < NR ? NR : size;
  if (p.ops.empty() || p.ops.size() > size_t(rbk::kSmallGates) || p.phases.size() > p.ops.size()) fail("program size");
  std::vector<cd> s(padded);
  for (uint32_t i = 0; i < padded; ++i) s.at(slot(i)) = i < size ? phys[i] : cd{};
  size_t next = 0;
  for (const auto& ph : p.phases) {
    if (ph.begin != next || ph.end <= ph.begin || ph.end > p.ops.size()) fail("phase range");
    next = ph.end;
    if (!(ph.reg[0] < ph.reg[1] && ph.reg[1] < ph.reg[2]) || (1u << ph.reg[2]) >= padded) fail("phase registers");
    std::set<uint32_t> seen;
    for (uint32_t t = 0; t < padded / NR; ++t) {
      uint32_t base = t;
      for (int k = 0; k < R; ++k) base = insert_zero(base, ph.reg[k]);
      uint32_t idx[NR];
      cd a[NR];
      for (int i = 0; i < NR; ++i) {
        uint32_t x = slot(base);
        for (int k = 0; k < R; ++k) if ((i >> k) & 1) x ^= slot(1u << ph.reg[k]);
        idx[i] = x;
        if (!seen.insert(x).second) fail("two threads on one slot");
        a[i] = s.at(x);
      }
      for (uint32_t g = ph.begin; g < ph.end; ++g) {
        const auto& o = p.ops[g];
        const int family = o.kind == rbk::OPK_X ? rbk::SMALL_X : o.kind == rbk::OPK_Y ? rbk::SMALL_Y
                           : o.code >= rbk::SMALL_REAL ? rbk::SMALL_REAL : rbk::SMALL_MAT;
        const bool diag = o.kind == rbk::OPK_DIAG || o.kind == rbk::OPK_NEG;
        if (diag ? (o.kind == rbk::OPK_NEG ? o.code != rbk::SMALL_NEG : o.code != rbk::SMALL_DIAG && o.code != rbk::SMALL_DIAG1)
                 : o.code != family + o.treg)
          fail("dispatch code");
        for (int i = 0; i < NR; ++i)
          if (((o.act >> i) & 1) != ((i & o.creg) == o.creg) || ((o.hi >> i) & 1) != ((i & o.dreg) != 0)) fail("slot masks");
        if ((base & o.cbase) != o.cbase) continue;
        for (int i = 0; i < NR; ++i) {
          if (!((o.act >> i) & 1)) continue;
          if (o.kind == rbk::OPK_NEG) a[i] = -a[i];
          else if (o.kind == rbk::OPK_DIAG) {
            if ((base & o.dbase) || ((o.hi >> i) & 1)) a[i] *= at(o.m, 1);
            else if (o.code == rbk::SMALL_DIAG) a[i] *= at(o.m, 0);
          } else {
            if (o.treg >= R) fail("target register");
            if ((i >> o.treg) & 1) continue;
            cd &x = a[i], &y = a[i | (1 << o.treg)];
            const cd u = x, v = y;
            if (o.kind == rbk::OPK_X) { x = v; y = u; }
            else if (o.kind == rbk::OPK_Y) { x = cd{v.imag(), -v.real()}; y = cd{-u.imag(), u.real()}; }
            else if (family == rbk::SMALL_REAL) { x = o.m[0] * u + o.m[2] * v; y = o.m[4] * u + o.m[6] * v; }
            else { x = at(o.m, 0) * u + at(o.m, 1) * v; y = at(o.m, 2) * u + at(o.m, 3) * v; }
          }
        }
      }
      for (int i = 0; i < NR; ++i) s.at(idx[i]) = a[i];
    }
  }
  if (next != p.ops.size()) fail("ops outside the phases");
  for (uint32_t i = 0; i < size; ++i) phys[i] = s.at(slot(i));
}

int main()
{
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> u(-1, 1);
  double worst = 0;
  for (int n = 1; n <= rbk::kSmallBits; ++n)
    for (int count : {1, 40, n <= 8 ? 900 : 120}) {
      std::vector<rbk::hgate> q;
      for (int k = 0; k < count; ++k) {
        rbk::hgate g{};
        g.target2 = -1;
        g.target = int8_t(rng() % n);
        for (int b = 0; b < n; ++b)
          if (b != g.target && rng() % 4 == 0 && rng() % 2) g.cmask |= 1ull << b;
        const double th = u(rng), ph = u(rng);
        switch (rng() % 8) {
          case 0: g.kind = rbk::OPK_X; break;
          case 1: g.kind = rbk::OPK_Y; break;
          case 2: g.kind = rbk::OPK_NEG; g.cmask |= 1ull << g.target; g.target = -1; break;
          case 3: case 4: {
            g.kind = rbk::OPK_DIAG;
            const cd d0 = rng() % 2 ? cd{1, 0} : std::polar(1.0, th), d1 = std::polar(1.0, ph);
            g.diag_one = d0 == cd{1, 0};
            g.m[0] = d0.real(); g.m[1] = d0.imag(); g.m[2] = d1.real(); g.m[3] = d1.imag();
            break;
          }
          case 5: {  // real rotation
            g.kind = rbk::OPK_MAT;
            g.m[0] = g.m[6] = std::cos(th); g.m[2] = std::sin(th); g.m[4] = -std::sin(th);
            break;
          }
          case 6: {
            if (n > 1 && rng() % 3 == 0) {
              g.kind = rbk::HK_SWAP; g.cmask = 0; g.target2 = int8_t((g.target + 1 + rng() % (n - 1)) % n);
              break;
            }
          }  // fall through: a general unitary
          default: {
            g.kind = rbk::OPK_MAT;
            const cd m[4] = {std::cos(th), -std::polar(std::sin(th), ph), std::polar(std::sin(th), u(rng)), 0};
            const cd m3 = std::cos(th) * (m[2] / -std::conj(m[1]) * 1.0);
            const cd v[4] = {m[0], m[1], m[2], std::sin(th) == 0 ? cd{1, 0} : m3};
            for (int e = 0; e < 4; ++e) { g.m[2 * e] = v[e].real(); g.m[2 * e + 1] = v[e].imag(); }
          }
        }
        q.push_back(g);
      }
      std::vector<cd> want(1u << n), phys(1u << n);
      std::vector<int> perm(n), inv(n);
      for (int b = 0; b < n; ++b) perm[b] = b;
      for (int b = n - 1; b > 0; --b) std::swap(perm[b], perm[rng() % (b + 1)]);
      for (int b = 0; b < n; ++b) inv[perm[b]] = b;
      auto to_phys = [&](uint32_t i) { uint32_t p = 0; for (int b = 0; b < n; ++b) p |= ((i >> b) & 1u) << perm[b]; return p; };
      for (uint32_t i = 0; i < want.size(); ++i) { want[i] = cd{u(rng), u(rng)}; phys[to_phys(i)] = want[i]; }
      for (const auto& g : q) {
        if (g.kind == rbk::HK_SWAP) {
          std::vector<cd> t(want);
          for (uint32_t i = 0; i < want.size(); ++i) {
            const uint32_t a = (i >> g.target) & 1, b = (i >> g.target2) & 1;
            t[(i & ~((1u << g.target) | (1u << g.target2))) | (b << g.target) | (a << g.target2)] = want[i];
          }
          want = t;
        } else {
          apply_direct(want, g);
        }
      }
      std::vector<rbk::small_program> progs;
      rbk::plan_small(n, q, perm, inv, progs);
      for (const auto& p : progs) run_program(phys, n, p);
      double norm = 0, err = 0;
      for (uint32_t i = 0; i < want.size(); ++i) {
        norm = std::max(norm, std::abs(want[i]));
        err = std::max(err, std::abs(want[i] - phys[to_phys(i)]));
      }
      worst = std::max(worst, err / norm);
    }
  std::printf("worst relative error %.3g\n", worst);
  if (!(worst < 1e-12)) fail("error");
  // 200,000 gates on 11 of 12 qubits, the twelfth idle or only a control: 0.1 s here
  // where a phase looks ahead a bounded way, 60 s where it scans the whole queue.
  for (const bool control : {false, true}) {
    constexpr int n = 12, count = 200000;
    std::vector<rbk::hgate> q;
    for (int k = 0; k < count; ++k) {
      rbk::hgate g{};
      g.target2 = -1;
      g.target = int8_t(rng() % (n - 1));
      if (rng() % 2) {
        g.kind = rbk::OPK_X;
        g.cmask = 1ull << (control && rng() % 3 == 0 ? n - 1 : (g.target + 1 + rng() % (n - 2)) % (n - 1));
      } else {
        g.kind = rbk::OPK_MAT;
        g.m[0] = g.m[6] = 0.6; g.m[2] = 0.8; g.m[4] = -0.8;
      }
      q.push_back(g);
    }
    std::vector<int> perm(n), inv(n);
    for (int b = 0; b < n; ++b) perm[b] = inv[b] = b;
    std::vector<rbk::small_program> progs;
    const std::clock_t t0 = std::clock();
    rbk::plan_small(n, q, perm, inv, progs);
    const double seconds = double(std::clock() - t0) / CLOCKS_PER_SEC;
    size_t ops = 0;
    for (const auto& p : progs) ops += p.ops.size();
    std::printf("%d gates planned in %.3f s\n", count, seconds);
    if (ops != count) fail("gates lost");
    if (seconds > 5.0) fail("planning time");
  }
  std::printf("ALL OK\n");
  return 0;
}
