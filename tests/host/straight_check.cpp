// Straight passes (dev_pass::straight) on the host: the pass programs run by the
// kernel model of plan_check.cpp equal the gates one by one, and each phase's
// layer tables give what the phase's gates give.
#define main plan_check_main
#include "plan_check.cpp"
#undef main

// The kernel's straight layer on one thread's registers.
static void run_layer(const plan_params& p, const dev_pass::straight_layer& L, std::vector<cplx>& a)
{
  auto value = [&](const double* t, int i) { return p.vbits == 0 ? t[i] : double(reinterpret_cast<const float*>(t)[i]); };
  auto factor = [&](const double* t, int i) { return cplx{value(t, 2 * i), value(t, 2 * i + 1)}; };
  const int NR = 1 << p.R;
  if (L.bits == 0) return;
  if (L.bits & kStraightPre) for (int i = 1; i < NR; ++i) a[i] *= factor(L.pre, i);
  for (int b = 0; b < p.R; ++b) {
    if (!((L.bits >> b) & 1)) continue;
    for (int i = 0; i < NR; ++i) {
      if ((i >> b) & 1) continue;
      const cplx a0 = a[i], a1 = a[i | (1 << b)];
      a[i] = a0 + value(L.t, 2 * b) * a1;
      a[i | (1 << b)] = value(L.t, 2 * b + 1) * a0 + a1;
    }
  }
  for (int i = 0; i < NR; ++i) a[i] *= factor(L.post, i);
}

static double layer_error(const plan_params& p, const dev_pass& P, std::mt19937_64& rng)
{
  std::normal_distribution<double> nd;
  double err = 0;
  for (int ph = 0; ph < P.num_phases; ++ph) {
    std::vector<cplx> a(size_t(1) << p.R), want;
    for (auto& x : a) x = cplx{nd(rng), nd(rng)};
    want = a;
    run_layer(p, P.straight_layers[ph], a);
    if (P.straight_layers[ph].run >= 0 && (!P.straight_runs || P.ops[P.straight_layers[ph].run].kind != OPK_PHASES)) return 1.0;
    for (int o = P.phases[ph].op_begin; o < P.phases[ph].op_end; ++o) {
      const dev_op& g = P.ops[o];
      if (g.kind == OPK_PHASES) {  // one run, the last records of the phase (run_pass checks its members)
        if (P.straight_layers[ph].run != o || o + 1 + int(g.run) != P.phases[ph].op_end) return 1.0;
        break;
      }
      if (g.kind != OPK_MAT || g.creg || g.cthr || g.cout) return 1.0;  // nothing else may be left in a straight pass
      hgate h{};
      h.kind = OPK_MAT;
      h.target = g.treg;
      h.target2 = -1;
      std::memcpy(h.m, g.m, sizeof(h.m));
      apply_direct(want, h);
    }
    for (size_t i = 0; i < a.size(); ++i) err = std::max(err, std::abs(a[i] - want[i]));
  }
  return err;
}

// U3 and Hadamard gates among X and CNOT gates; now and then a gate that no straight pass takes.
static std::vector<hgate> cnot_gates(std::mt19937_64& rng, int n, int count, bool others)
{
  std::vector<hgate> out;
  for (int k = 0; k < count; ++k) {
    hgate g{};
    g.target2 = -1;
    g.target = static_cast<int>(rng() % n);
    const int c = static_cast<int>(rng() % n);
    switch (rng() % (others ? 8 : 6)) {
      case 0: case 1: g.kind = OPK_MAT; unitary_u3(rng, g.m); break;
      case 2: g.kind = OPK_MAT; g.m[0] = g.m[2] = g.m[4] = std::sqrt(0.5); g.m[6] = -g.m[0]; break;
      case 3: g.kind = OPK_X; break;
      case 6: g = random_gate(rng, n); break;
      case 7:  // two controls
        g.kind = OPK_X;
        g.cmask = ((1ull << c) | (1ull << ((c + 1) % n))) & ~(1ull << g.target);
        break;
      default: g.kind = OPK_X; if (c != g.target) g.cmask = 1ull << c; break;
    }
    out.push_back(g);
  }
  return out;
}

int main()
{
  int failures = 0, most_phases = 0, most_folds = 0, with_runs = 0;
  for (int prec = 0; prec < 2; ++prec)
  for (int seed = 0; seed < 24; ++seed) {
    std::mt19937_64 rng(7000 * prec + seed);
    plan_params p{};
    shape_bits(prec, 2, &p.K, &p.R);
    p.vbits = prec;
    p.LOW = prec == 0 ? 5 : 6;
    p.n = p.K + seed % 4;
    p.dense_budget = seed % 8 == 7 ? 30 : 1 + static_cast<int>(rng() % 20);
    p.straight = true;
    const bool others = seed % 4 == 3;
    const auto gates = seed % 8 == 1 ? ansatz_gates(rng, p.n, 6) : seed % 2 ? cnot_gates(rng, p.n, 200, others) : brick_gates(rng, p.n, 6);
    std::vector<cplx> st(1ull << p.n), want;
    std::normal_distribution<double> nd;
    for (auto& x : st) x = cplx{nd(rng), nd(rng)};
    want = st;
    for (const auto& g : gates) apply_direct(want, g);
    std::vector<int> perm(p.n), inv(p.n);
    for (int i = 0; i < p.n; ++i) perm[i] = inv[i] = i;
    std::vector<dev_pass> passes;
    plan_passes(p, gates, perm, inv, passes);
    plan_canonicalize(p, perm, inv, passes);
    int straight = 0;
    double layers = 0;
    for (const auto& P : passes) {
      run_pass(st, p, P);
      if (!P.straight) continue;
      ++straight;
      with_runs += P.straight_runs != 0;
      if (P.straight != P.num_phases || P.straight > unsigned(kMaxStraight)) ++failures;
      layers = std::max(layers, layer_error(p, P, rng));
      most_phases = std::max<int>(most_phases, P.num_phases);
      for (int ph = 0; ph < P.num_phases; ++ph) most_folds = std::max<int>(most_folds, P.phases[ph].num_folds);
    }
    // random_gate's matrices are not unitary: relative to the largest amplitude
    double err = 0, scale = 1;
    for (const auto& x : want) scale = std::max(scale, std::abs(x));
    for (size_t i = 0; i < st.size(); ++i) err = std::max(err, std::abs(st[i] - want[i]) / scale);
    std::printf("prec=%d seed=%d n=%d budget=%d passes=%zu straight=%d err=%.2e layers=%.2e\n", prec, seed, p.n, p.dense_budget,
                passes.size(), straight, err, layers);
    // rounding 1e-16 a gate; complex<float> tables (of layers, also in general passes) are
    // rounded to 6e-8, a few times over in a layer of 5 gates
    if (!(err < (prec == 0 ? 1e-12 : 1e-5)) || !(layers < (prec == 0 ? 1e-13 : 3e-6))) ++failures;
    if (seed % 2 == 0 && straight == 0) ++failures;  // brick circuits
  }
  std::printf("phases up to %d, conditional folds up to %d, passes with phase runs %d\n", most_phases, most_folds, with_runs);
  if (most_phases != kMaxStraight || most_folds == 0 || with_runs == 0) ++failures;
  std::printf(failures ? "FAILED %d\n" : "ALL OK\n", failures);
  return failures ? 1 : 0;
}
