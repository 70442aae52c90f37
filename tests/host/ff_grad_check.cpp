// Host check of the two-float gradient code by kind of quartet (no shared centre, a
// one-centre bra, the ket's first centre on it, one centre), against long double.
// Prints per class and kind the worst and the rms difference relative to the largest
// component.  The derivative of a one-centre (ps| bra is the difference 2a (ds| - (ss|,
// whose parts may exceed it by 2^11: there relative to K_ab K_cd / sqrt(p + q), their
// size, where that is larger.  A one-centre quartet whose derivatives vanish is left out.
// Compile as ff_check.cpp.
#define main ff_check_main
#include "ff_check.cpp"
#undef main

template <typename F1, typename F2> static void kinds(const char* name, F1 run_ld, F2 run_ff) {
  for (int kind = 0; kind < 4; ++kind) {
    ld worst = 0, sum = 0;
    int n = 0;
    for (int rep = 0; rep < 3000; ++rep) {
      const Quartet q = make(kind);
      Acc<ld> a;
      Acc<ff> b;
      run_ld(q, a);
      run_ff(q, b);
      ld mx = 0, d = 0;
      for (int i = 0; i < 6; ++i) {
        mx = std::max(mx, std::fabs(a.v[i]));
        d = std::max(d, std::fabs(a.v[i] - value(b.v[i])));
      }
      if (mx < 1e-20L) continue;
      if (kind >= 1 && name[0] == 'p' && name[1] == 's') mx = std::max(mx, q.sb[11] * q.kt[11] / std::sqrt(q.sb[0] + q.kt[0]));
      worst = std::max(worst, d / mx);
      sum += d / mx * d / mx;
      ++n;
    }
    if (n) std::printf("%s %d %.3Le %.3Le\n", name, kind, worst, std::sqrt(sum / n));
  }
}
#undef GRAD
#define GRAD(cls, n) kinds(#cls, \
  [](const Quartet& q, Acc<ld>& a) { const ld* k = q.kt; ld g[n]; for (int i = 0; i < n; ++i) g[i] = 0.3L + 0.1L * (i % 7) - 0.05L * (i % 3); \
    Gam<ld> gm{g}; TkA<ld> tk; grad_ket_##cls<ld>(k[1], k[5], k[6], k[7], k[8], k[9], k[10], gm, tk); grad_ketprim_##cls<ld>(q.sb, 1, BRA_SB, k[0], k[2], k[3], k[4], k[11], nullptr, tk, a.v); }, \
  [](const Quartet& q, Acc<ff>& a) { const ff* k = q.fk; ff g[n]; for (int i = 0; i < n; ++i) g[i] = split(0.3L + 0.1L * (i % 7) - 0.05L * (i % 3)); \
    Gam<ff> gm{g}; TkA<ff> tk; grad_ket_##cls<ff>(k[1], k[5], k[6], k[7], k[8], k[9], k[10], gm, tk); grad_ketprim_##cls<ff>(q.fb, 1, BRA_SB, k[0], k[2], k[3], k[4], k[11], (const ff*)table.data(), tk, a.v); })

int main() {
  build_table();
  GRAD(ssss, 1); GRAD(ssps, 3); GRAD(sspp, 9); GRAD(psss, 3); GRAD(psps, 9); GRAD(pspp, 27); GRAD(ppss, 9); GRAD(ppps, 27);
  GRAD(pppp, 81); GRAD(ssds, 6); GRAD(ssdp, 18); GRAD(psds, 18); GRAD(dsss, 6); GRAD(dsps, 18);
  return 0;
}
