// Host check of the two-float range rule (ff_pair_range in csrc/gbhf_ff.cuh): the
// generated ERI and gradient code on primitive quartets whose pairs sit at the rule's
// upper edge, exponents from 1e-8 to 1e8, against long double.  Prints per class how
// many gave a value that is not finite and, for the ERIs of pairs that the rule also
// lets grow (largest quartet of the molecule: 1), the worst difference over
// 2^-38 of the largest component plus 2^-45.  Compile as ff_check.cpp.
#define main ff_check_main
#include "ff_check.cpp"
#undef main

// A quartet of momenta l[4]: K of both pairs as large as the rule allows.
static bool grows;   // both pairs of the last quartet are within FF_MAX_GROW
static Quartet edge(const int* l, int kind) {
  grows = true;
  double X[4][3], e[4];
  for (double& v : e) v = std::exp(U(std::log(1e-8), std::log(1e8)));
  if (kind % 3 == 0) e[1] = e[2] = e[3] = e[0];
  if (kind % 3 == 1) e[1] = e[0], e[3] = e[2];
  const double far = 1 / std::sqrt(std::min(std::min(e[0], e[1]), std::min(e[2], e[3])));
  for (int k = 0; k < 4; ++k)
    for (int x = 0; x < 3; ++x) X[k][x] = kind & 1 && k ? X[0][x] : U(-1, 1) * std::min(far, 1e4);
  Quartet q;
  auto pair = [&](int i, int j, ld* r, ff* f) {
    const ld a = e[i], b = e[j], p = a + b;
    double big = 0;
    r[0] = p, r[1] = 1 / p;
    for (int x = 0; x < 3; ++x) {
      const ld d = (ld)X[i][x] - (ld)X[j][x];
      r[5 + x] = -b / p * d;
      r[8 + x] = a / p * d;
      r[2 + x] = (ld)X[i][x] - (ld)X[0][x] + r[5 + x];
      big = std::max(big, (double)std::max(std::fabs(r[5 + x]), std::fabs(r[8 + x])));
    }
    float size, grow;
    gbhf::ff_pair_range((double)p, 1.0, big, l[i] + l[j], size, grow);
    r[11] = std::ldexp(1.0L, (int)std::floor(gbhf::FF_MAX_SIZE - size));
    grows &= grow <= gbhf::FF_MAX_GROW;
    r[12] = a;
    for (int k = 0; k < 13; ++k) f[k] = split(r[k]);
  };
  pair(0, 1, q.sb, q.fb);
  pair(2, 3, q.kt, q.fk);
  for (int x = 0; x < 3; ++x) {   // P and Q relative to A, as the kernels hold them
    q.fk[2 + x] = split(q.kt[2 + x]);
    q.fb[2 + x] = q.fb[5 + x];
  }
  return q;
}
template <typename F1, typename F2> static void range(const char* name, int nout, F1 run_ld, F2 run_ff) {
  const char* c = name + (std::strncmp(name, "grad_", 5) ? 0 : 5);
  int l[4], bad = 0, n = 0;
  for (int k = 0; k < 4; ++k) l[k] = c[k] == 's' ? 0 : c[k] == 'p' ? 1 : 2;
  ld worst = 0;
  for (int rep = 0; rep < 3000; ++rep) {
    const Quartet q = edge(l, rep);
    Acc<ld> a;
    Acc<ff> b;
    run_ld(q, a);
    run_ff(q, b);
    ld mx = 0, d = 0;
    bool finite = true;
    for (int i = 0; i < nout; ++i) {
      finite &= std::isfinite(b.v[i].h) && std::isfinite(b.v[i].l);
      mx = std::max(mx, std::fabs(a.v[i]));
      d = std::max(d, std::fabs(a.v[i] - value(b.v[i])));
    }
    bad += !finite;
    if (finite && grows && c == name) worst = std::max(worst, d / (std::ldexp(mx, -38) + std::ldexp(1.0L, -45))), ++n;
  }
  std::printf("%s %d %d %.3Lf\n", name, bad, n, worst);
}
#undef ERI
#undef GRAD
#define ERI(cls, n) range(#cls, n, \
  [](const Quartet& q, Acc<ld>& a) { const ld* k = q.kt; eri_ketprim_##cls<ld, Acc<ld>>(q.sb, 1, BRA_SB, k[0], k[1], k[2], k[3], k[4], k[5], k[6], k[7], k[8], k[9], k[10], k[11], nullptr, a); }, \
  [](const Quartet& q, Acc<ff>& a) { const ff* k = q.fk; eri_ketprim_##cls<ff, Acc<ff>>(q.fb, 1, BRA_SB, k[0], k[1], k[2], k[3], k[4], k[5], k[6], k[7], k[8], k[9], k[10], k[11], (const ff*)table.data(), a); })
#define GRAD(cls, n) range("grad_" #cls, 6, \
  [](const Quartet& q, Acc<ld>& a) { const ld* k = q.kt; ld g[n]; for (ld& x : g) x = 4; \
    Gam<ld> gm{g}; TkA<ld> tk; grad_ket_##cls<ld>(k[1], k[5], k[6], k[7], k[8], k[9], k[10], gm, tk); grad_ketprim_##cls<ld>(q.sb, 1, BRA_SB, k[0], k[2], k[3], k[4], k[11], nullptr, tk, a.v); }, \
  [](const Quartet& q, Acc<ff>& a) { const ff* k = q.fk; ff g[n]; for (ff& x : g) x = ff(4); \
    Gam<ff> gm{g}; TkA<ff> tk; grad_ket_##cls<ff>(k[1], k[5], k[6], k[7], k[8], k[9], k[10], gm, tk); grad_ketprim_##cls<ff>(q.fb, 1, BRA_SB, k[0], k[2], k[3], k[4], k[11], (const ff*)table.data(), tk, a.v); })

int main() {
  build_table();
  ERI(ssss, 1); ERI(psss, 3); ERI(psps, 9); ERI(sspp, 9); ERI(pspp, 27); ERI(pppp, 81);
  ERI(dsss, 6); ERI(dsps, 18); ERI(dspp, 54); ERI(dsds, 36); ERI(dpss, 18); ERI(dpps, 54); ERI(ddss, 36);
  GRAD(ssss, 1); GRAD(ssps, 3); GRAD(sspp, 9); GRAD(psss, 3); GRAD(psps, 9); GRAD(pspp, 27); GRAD(ppss, 9); GRAD(ppps, 27);
  GRAD(pppp, 81); GRAD(ssds, 6); GRAD(ssdp, 18); GRAD(psds, 18); GRAD(dsss, 6); GRAD(dsps, 18);
  // the rule's verdict on primitives that overflow: p functions on one centre, a contraction weight each
  for (const double ex : {1e4, 1e5, 1e6, 1e7})
    for (const double w : {1.0, 0.01}) {
      const double c = w * 2 * std::sqrt(ex) * std::pow(2 * ex / M_PI, 0.75);
      Quartet q;
      std::memset((void*)&q, 0, sizeof q);
      const ld r[13] = {2 * ex, 0.5 / ex, 0, 0, 0, 0, 0, 0, 0, 0, 0, std::sqrt(34.98683665524972) * c * c / (2 * ex), ex};
      for (int k = 0; k < 13; ++k) q.fb[k] = q.fk[k] = split(r[k]), q.sb[k] = q.kt[k] = r[k];
      float size, grow;
      gbhf::ff_pair_range(2 * ex, (double)r[11], 0.0, 2, size, grow);
      Acc<ff> a, g;
      const ff* k = q.fk;
      eri_ketprim_pppp<ff, Acc<ff>>(q.fb, 1, BRA_SB, k[0], k[1], k[2], k[3], k[4], k[5], k[6], k[7], k[8], k[9], k[10], k[11], (const ff*)table.data(), a);
      ff gg[81];
      for (ff& x : gg) x = ff(1);
      Gam<ff> gm{gg};
      TkA<ff> tk;
      grad_ket_pppp<ff>(k[1], k[5], k[6], k[7], k[8], k[9], k[10], gm, tk);
      grad_ketprim_pppp<ff>(q.fb, 1, BRA_SB, k[0], k[2], k[3], k[4], k[11], (const ff*)table.data(), tk, g.v);
      bool fin = true;
      for (int i = 0; i < 81; ++i) fin &= std::isfinite(a.v[i].h + a.v[i].l);
      for (int i = 0; i < 6; ++i) fin &= std::isfinite(g.v[i].h + g.v[i].l);
      std::printf("steep %d %d %d\n", (int)std::lround(std::log10(ex)), fin, size <= gbhf::FF_MAX_SIZE);
    }
  return 0;
}
