// Host check of the two-float arithmetic (csrc/gbhf_ff.cuh) in the generated
// ERI and gradient code: random primitive quartets over steep, ordinary and
// diffuse exponents, shared and distinct centres and Boys arguments on both
// sides of the table's end, each class in two floats and in long double (an
// exact Boys series).  Prints per class the largest difference relative to the
// largest component of the quartet, and of 1/sqrt and the Boys function alone.
// Compile with -ffp-contract=off (the error terms need the operations as written).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#define __device__
#define __host__
#define __forceinline__ inline
#define __restrict__
#define __align__(n) alignas(n)
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline int __float_as_int(float x) { int i; std::memcpy(&i, &x, 4); return i; }
struct alignas(16) float4 { float x, y, z, w; };
inline float4 __ldg(const float4* p) { return *p; }
// an estimate with the hardware's error, 2^-22.9, of either sign
inline float rsqrt_est(float x) { return (float)(1.0 / std::sqrt((double)x) * (1.0 + (__float_as_int(x) & 1 ? 1.2e-7 : -1.2e-7))); }
namespace gbhf { using ::rsqrt_est; }
#include "gbhf_ff.cuh"
using gbhf::ff;
using ld = long double;
enum { BRA_P = 0, BRA_INVP, BRA_PX, BRA_PY, BRA_PZ, BRA_PAX, BRA_PAY, BRA_PAZ, BRA_PBX, BRA_PBY, BRA_PBZ, BRA_K, BRA_AEXP };
#define BRA_SB 16
template <typename T> struct BraPrim { T p, invp, Px, Py, Pz, PAx, PAy, PAz, PBx, PBy, PBz, K, a; };
template <typename T> void load_bra_prim(const T* r, BraPrim<T>& b) {
  b.p = r[0]; b.invp = r[1]; b.Px = r[2]; b.Py = r[3]; b.Pz = r[4]; b.PAx = r[5]; b.PAy = r[6]; b.PAz = r[7];
  b.PBx = r[8]; b.PBy = r[9]; b.PBz = r[10]; b.K = r[11]; b.a = r[12];
}
template <typename T> T rsqrt_t(T x) { return 1 / std::sqrt(x); }
template <> ff rsqrt_t<ff>(ff x) { return gbhf::rsqrt_ff(gbhf::nrm(x)); }
template <typename T> T fma_t(T a, T b, T c) { return a * b + c; }
template <> ff fma_t<ff>(ff a, ff b, ff c) { return gbhf::fma_ff(a, b, c); }

static ld boys_exact(int m, ld t) {
  if (t > 60) {
    ld f = std::sqrt(M_PIl / t) / 2;
    for (int k = 1; k <= m; ++k) f *= (2 * k - 1) / (2 * t);
    return f;
  }
  ld term = 1.0L / (2 * m + 1), s = term;
  for (int k = 1; k < 2000; ++k) {
    term *= 2 * t / (2 * m + 2 * k + 1);
    s += term;
    if (term < 1e-24L * s) break;
  }
  return std::exp(-t) * s;
}
static std::vector<float> table;
static void build_table() {   // the layout of BOYSFF_*
  table.assign((size_t)(BOYSH_LMAX + 1) * BOYSFF_NROW * BOYSFF_STRIDE + 4, 0.0f);
  for (int L = 0; L <= BOYSH_LMAX; ++L)
    for (int j = 0; j < BOYSFF_NROW; ++j) {
      float* row = table.data() + ((size_t)L * BOYSFF_NROW + j) * BOYSFF_STRIDE;
      const ld tj = (ld)j * BOYSFF_H;
      ld fact = 1;
      for (int k = 0; k < 6; ++k) {
        if (k) fact *= k;
        const double v = (double)(boys_exact(L + k, tj) / fact);
        if (k < 4) { row[2 * k] = (float)v; row[2 * k + 1] = (float)(v - (double)row[2 * k]); }
        else row[4 + k] = (float)v;
      }
      const double e = (double)std::exp(-tj);
      row[10] = (float)e;
      row[11] = (float)(e - (double)row[10]);
    }
}
template <typename T, int L> void boys_eval(T t, const T*, T* F) {
  for (int m = 0; m <= L; ++m) F[m] = boys_exact(m, t);
}
template <> void boys_eval<ff, 0>(ff t, const ff* tab, ff* F) { gbhf::boys_eval_ff<0>(t, tab, F); }
#define BOYS(L) template <> void boys_eval<ff, L>(ff t, const ff* tab, ff* F) { gbhf::boys_eval_ff<L>(t, tab, F); }
BOYS(1) BOYS(2) BOYS(3) BOYS(4) BOYS(5) BOYS(6)
template <typename T> struct Acc { T v[1296]; Acc() { for (T& x : v) x = T(0); } T& operator[](int i) { return v[i]; } };
template <typename T> struct Gam { const T* v; T get(int i) const { return v[i]; } };
template <typename T> struct TkA { T v[1296]; T get(int i) const { return v[i]; } void set(int i, T x) { v[i] = x; } };
#include "eri_gen.cuh"
#include "grad_gen.cuh"

static std::mt19937_64 rng(7);
static double U(double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); }
static ff split(ld x) { const float h = (float)x; return ff(h, (float)(x - (ld)h)); }
static ld value(ff x) { return (ld)x.h + (ld)x.l; }

struct Quartet {
  ld sb[16], kt[16];   // long double fields (P relative to A for both pairs)
  ff fb[16], fk[16];
};
static Quartet make(int kind) {
  double X[4][3], e[4];
  for (int k = 0; k < 4; ++k) {
    for (int x = 0; x < 3; ++x) X[k][x] = U(-3, 3);
    const double r = U(0, 1);
    e[k] = kind == 0 ? std::exp(U(std::log(0.1), std::log(5.0))) : r < 0.3 ? std::exp(U(std::log(5.0), std::log(6000.0))) : std::exp(U(std::log(0.05), std::log(5.0)));
  }
  if (kind >= 1) for (int x = 0; x < 3; ++x) X[1][x] = X[0][x];            // one-centre bra
  if (kind >= 2) for (int x = 0; x < 3; ++x) X[2][x] = X[0][x];            // the ket's C on it
  if (kind >= 3) for (int x = 0; x < 3; ++x) X[3][x] = X[0][x];            // all on one centre
  Quartet q;
  auto pair = [&](int i, int j, ld* r, ff* f) {
    const ld a = e[i], b = e[j], p = a + b;
    ld ab2 = 0;
    r[0] = p; r[1] = 1 / p;
    for (int x = 0; x < 3; ++x) {
      const ld d = (ld)X[i][x] - (ld)X[j][x];
      ab2 += d * d;
      r[5 + x] = -b / p * d;
      r[8 + x] = a / p * d;
      r[2 + x] = (ld)X[i][x] - (ld)X[0][x] + r[5 + x];   // relative to A
    }
    r[11] = std::exp(-a * b / p * ab2) / p;
    r[12] = a;
    for (int k = 0; k < 13; ++k) f[k] = split(r[k]);
  };
  pair(0, 1, q.sb, q.fb);
  pair(2, 3, q.kt, q.fk);
  // as the kernels: Q - A = (Q - C) - (A - C) in two floats, A - C from three FP32 parts
  for (int x = 0; x < 3; ++x) {
    float c[2][3];
    for (int k = 0; k < 2; ++k) {
      double r = X[k ? 2 : 0][x];
      for (int i = 0; i < 3; ++i) { c[k][i] = (float)r; r -= (double)c[k][i]; }
    }
    const ff AC = gbhf::diff3(c[0][0], c[0][1], c[0][2], c[1][0], c[1][1], c[1][2]);
    q.fk[2 + x] = gbhf::nrm(q.fk[5 + x] - AC);
    q.fb[2 + x] = q.fb[5 + x];
  }
  return q;
}
template <typename F1, typename F2> static void eri(const char* name, int nout, F1 run_ld, F2 run_ff) {
  ld worst = 0, sum = 0;
  int n = 0;
  for (int rep = 0; rep < 4000; ++rep) {
    const Quartet q = make(rep % 4);
    Acc<ld> a;
    Acc<ff> b;
    run_ld(q, a);
    run_ff(q, b);
    ld mx = 0, d = 0;
    for (int i = 0; i < nout; ++i) { mx = std::max(mx, std::fabs(a.v[i])); d = std::max(d, std::fabs(a.v[i] - value(b.v[i]))); }
    if (mx > 1e-20L) { worst = std::max(worst, d / mx); sum += d / mx * d / mx; ++n; }
  }
  std::printf("%s %.3Le %.3Le\n", name, worst, std::sqrt(sum / n));
}
#define ERI(cls, n) eri(#cls, n, \
  [](const Quartet& q, Acc<ld>& a) { const ld* k = q.kt; eri_ketprim_##cls<ld, Acc<ld>>(q.sb, 1, BRA_SB, k[0], k[1], k[2], k[3], k[4], k[5], k[6], k[7], k[8], k[9], k[10], k[11], nullptr, a); }, \
  [](const Quartet& q, Acc<ff>& a) { const ff* k = q.fk; eri_ketprim_##cls<ff, Acc<ff>>(q.fb, 1, BRA_SB, k[0], k[1], k[2], k[3], k[4], k[5], k[6], k[7], k[8], k[9], k[10], k[11], (const ff*)table.data(), a); })
#define GRAD(cls, n) eri("grad_" #cls, 6, \
  [](const Quartet& q, Acc<ld>& a) { const ld* k = q.kt; ld g[n]; for (int i = 0; i < n; ++i) g[i] = 0.3L + 0.1L * (i % 7) - 0.05L * (i % 3); \
    Gam<ld> gm{g}; TkA<ld> tk; grad_ket_##cls<ld>(k[1], k[5], k[6], k[7], k[8], k[9], k[10], gm, tk); grad_ketprim_##cls<ld>(q.sb, 1, BRA_SB, k[0], k[2], k[3], k[4], k[11], nullptr, tk, a.v); }, \
  [](const Quartet& q, Acc<ff>& a) { const ff* k = q.fk; ff g[n]; for (int i = 0; i < n; ++i) g[i] = split(0.3L + 0.1L * (i % 7) - 0.05L * (i % 3)); \
    Gam<ff> gm{g}; TkA<ff> tk; grad_ket_##cls<ff>(k[1], k[5], k[6], k[7], k[8], k[9], k[10], gm, tk); grad_ketprim_##cls<ff>(q.fb, 1, BRA_SB, k[0], k[2], k[3], k[4], k[11], (const ff*)table.data(), tk, a.v); })

int main() {
  build_table();
  ld worst = 0;
  for (int i = 0; i < 200000; ++i) {
    const ff x = split(std::exp(U(-10, 12)));
    worst = std::max(worst, std::fabs(value(gbhf::rsqrt_ff(x)) * std::sqrt(value(x)) - 1));
  }
  std::printf("rsqrt %.3Le %.3Le\n", worst, worst);
  worst = 0;
  for (int i = 0; i < 20000; ++i) {
    const ff t = split(i % 3 ? U(0, 80) : std::exp(U(-30, 4)));
    ff F[10];
    gbhf::boys_eval_ff<9>(t, (const ff*)table.data(), F);
    for (int m = 0; m < 10; ++m) {
      const ld r = boys_exact(m, value(t));
      worst = std::max(worst, std::fabs(value(F[m]) - r) / r);
    }
    gbhf::boys_eval_ff<0>(t, (const ff*)table.data(), F);
    worst = std::max(worst, std::fabs(value(F[0]) / boys_exact(0, value(t)) - 1));
  }
  std::printf("boys %.3Le %.3Le\n", worst, worst);
  ERI(ssss, 1); ERI(psss, 3); ERI(psps, 9); ERI(sspp, 9); ERI(pspp, 27); ERI(pppp, 81);
  ERI(dsss, 6); ERI(dsps, 18); ERI(dspp, 54); ERI(dsds, 36); ERI(dpss, 18); ERI(dpps, 54); ERI(ddss, 36);
  GRAD(ssss, 1); GRAD(ssps, 3); GRAD(sspp, 9); GRAD(psss, 3); GRAD(psps, 9); GRAD(pspp, 27); GRAD(ppss, 9); GRAD(ppps, 27);
  GRAD(pppp, 81); GRAD(ssds, 6); GRAD(ssdp, 18); GRAD(psds, 18); GRAD(dsss, 6); GRAD(dsps, 18);
  return 0;
}
