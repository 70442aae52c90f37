// Two-float arithmetic for the direct builds: a value is the unevaluated sum
// h + l of two FP32 numbers (about 2^-46 relative error per operation).
//
// Why: this GPU runs FP64 at 1/64 of its FP32 rate (2 against 128 lanes per SM
// and cycle), so one FP64 fused multiply-add costs the issue slots of 64 FP32
// instructions; the two-float one takes 12.  The kernels use it for the
// quartets whose Schwarz bound makes its absolute error smaller than the error
// that the build has anyway (ff_limits in setup.cu says which).
//
// Rules of the representation: a sum keeps the exact rounding error of the
// heads (Knuth's two-sum, D. E. Knuth, TAOCP vol. 2, 4.2.2) and a product that
// of the heads' product (one FMA, Dekker 1971); l is not renormalised by either,
// so it may grow to a few ulp of h along a chain.  Products drop l * l.  nrm()
// restores |l| <= ulp(h) / 2 where a value is multiplied on many times.
// __fadd_rn and __fmul_rn keep the compiler from contracting the error terms away.
#pragma once
#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif

#define BOYSH_LMAX 9   // (dd|dd) gradient: L = 9
// Two-float Boys table: spacing 1/64 up to 60, so that a node is an
// exact FP32 number and |dx| <= 1/128 (6 terms: remainder 3e-16); orders 0-3 of
// the expansion hold two floats, 4 and 5 (below 2e-10 of the sum) one.
#define BOYSFF_H 0.015625f
#define BOYSFF_TMAX 60.0f
#define BOYSFF_NROW 3842
#define BOYSFF_STRIDE 12   // floats: G0..G3 (two each), G4, G5, exp(-T_j) (two): three 16-byte loads

// Nearest integer j of x (0 <= x < 2^22), returned as j and as its exact FP32
// value: adding 1.5 * 2^23 leaves j in the low mantissa bits of the sum, with no
// float<->int conversion instruction.
__device__ __forceinline__ float round_node(float x, int& j) {
  const float r = x + 12582912.0f;
  j = __float_as_int(r) - 0x4B400000;
  return r - 12582912.0f;
}

namespace gbhf {

struct __align__(8) ff {
  float h, l;
  ff() = default;
  __host__ __device__ constexpr ff(float a, float b) : h(a), l(b) {}
  __host__ __device__ constexpr ff(float a) : h(a), l(0.0f) {}
  __host__ __device__ constexpr ff(int a) : h((float)a), l(0.0f) {}
  __host__ __device__ constexpr ff(double a) : h((float)a), l((float)(a - (double)(float)a)) {}
};

// |b| <= |a| (or a = 0): three operations
__device__ __forceinline__ ff quick_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return ff(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ ff two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return ff(s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb)));
}
__device__ __forceinline__ ff nrm(ff a) { return quick_sum(a.h, a.l); }
__device__ __forceinline__ double nrm(double a) { return a; }
__device__ __forceinline__ float nrm(float a) { return a; }

__device__ __forceinline__ ff operator-(ff a) { return ff(-a.h, -a.l); }
__device__ __forceinline__ ff operator+(ff a, ff b) {
  ff s = two_sum(a.h, b.h);
  s.l = __fadd_rn(s.l, __fadd_rn(a.l, b.l));
  return s;
}
__device__ __forceinline__ ff operator-(ff a, ff b) { return a + (-b); }
__device__ __forceinline__ ff operator*(ff a, ff b) {
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  return ff(p, __fmaf_rn(a.l, b.h, e));
}
// by a number that FP32 holds exactly
__device__ __forceinline__ ff operator*(float a, ff b) {
  const float p = __fmul_rn(a, b.h);
  return ff(p, __fmaf_rn(a, b.l, __fmaf_rn(a, b.h, -p)));
}
__device__ __forceinline__ ff operator*(ff a, float b) { return b * a; }
__device__ __forceinline__ ff& operator+=(ff& a, ff b) { return a = a + b; }
__device__ __forceinline__ ff& operator*=(ff& a, ff b) { return a = nrm(a * b); }
__device__ __forceinline__ ff fma_ff(ff a, ff b, ff c) { return c + a * b; }

// a - b of coordinates held as three FP32 parts each (every bit of the double)
__device__ __forceinline__ ff diff3(float a0, float a1, float a2, float b0, float b1, float b2) {
  const ff s = two_sum(a0, -b0), t = two_sum(a1, -b1);
  const ff u = two_sum(s.l, t.h), v = two_sum(s.h, u.h);
  return quick_sum(v.h, v.l + (u.l + t.l + (a2 - b2)));
}

#ifdef __CUDACC__
__device__ __forceinline__ float rsqrt_est(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
#endif
// 1/sqrt(x): the hardware estimate, one FP32 Newton step, then the residual
// 1 - x y^2 formed exactly from y^2 and both parts of x; relative error 2^-47.
__device__ __forceinline__ ff rsqrt_ff(ff x) {
  float y = rsqrt_est(x.h);
  y = __fmaf_rn(0.5f * y, __fmaf_rn(-x.h * y, y, 1.0f), y);
  const float s = __fmul_rn(y, y), se = __fmaf_rn(y, y, -s);
  float e = __fmaf_rn(-x.h, s, 1.0f);
  e = __fmaf_rn(-x.h, se, e);
  e = __fmaf_rn(-x.l, s, e);
  return ff(y, y * (e * __fmaf_rn(0.375f, e, 0.5f)));
}

// F_0..F_L(t) from the two-float table.  Each Horner step of the leading four
// terms adds a product that is below 1/128 of the head (quick_sum); exp(-t) is
// exp(-T_j) times the series of exp(dx).
template <int L>
__device__ __forceinline__ void boys_eval_ff(ff tin, const ff* __restrict__ tab, ff* F) {
  static_assert(L <= BOYSH_LMAX, "the Boys tables hold orders up to BOYSH_LMAX");
  const ff t = nrm(tin);
  if (t.h < BOYSFF_TMAX) {
    int j;
    const float node = round_node(t.h * 64.0f, j) * BOYSFF_H;
    const float4* row = reinterpret_cast<const float4*>(tab) + ((size_t)L * BOYSFF_NROW + j) * (BOYSFF_STRIDE / 4);
    const float4 c0 = __ldg(row), c1 = __ldg(row + 1), c2 = __ldg(row + 2);
    const ff dx = two_sum(__fsub_rn(node, t.h), -t.l);   // node - t.h is exact
    auto horner = [&](float gh, float gl, ff s) {
      const ff p = dx * s;
      ff r = quick_sum(gh, p.h);
      r.l = __fadd_rn(r.l, __fadd_rn(gl, p.l));
      return r;
    };
    const float tail = dx.h * __fmaf_rn(dx.h, c2.y, c2.x);
    ff s = quick_sum(c1.z, tail);
    s.l = __fadd_rn(s.l, c1.w);
    s = horner(c1.x, c1.y, s);
    s = horner(c0.z, c0.w, s);
    s = horner(c0.x, c0.y, s);
    F[L] = nrm(s);
    if constexpr (L >= 1) {
      constexpr ff sixth(1.0 / 6.0);
      ff e = quick_sum(sixth.h, dx.h * __fmaf_rn(dx.h, float(1.0 / 120), float(1.0 / 24)));
      e.l = __fadd_rn(e.l, sixth.l);
      e = horner(0.5f, 0.0f, e);
      e = horner(1.0f, 0.0f, e);
      e = horner(1.0f, 0.0f, e) * ff(c2.z, c2.w);
      const ff t2(t.h + t.h, t.l + t.l);
#pragma unroll
      for (int m = L - 1; m >= 0; --m) {
        ff f = e + t2 * F[m + 1];
        if (m > 0) f = f * ff(1.0 / (2 * m + 1));
        F[m] = nrm(f);
      }
    }
  } else {
    const ff r = rsqrt_ff(t);
    F[0] = nrm(ff(0.88622692545275801365) * r);
    const ff h = nrm(r * r);
#pragma unroll
    for (int m = 1; m <= L; ++m) F[m] = nrm(F[m - 1] * (float(m - 0.5) * h));
  }
}

// Range of a primitive pair in two floats, as exponents of two.  The class code
// forms pref (-2 alpha)^n F_n times expansion coefficients, pref = K_ab K_cd /
// sqrt(p + q), alpha = p q / (p + q) <= min(p, q), n <= L_ab + L_cd + 1 (one order
// more in the gradient, whose coefficients also take a factor 2a <= 2p).  A
// coefficient is a polynomial of degree <= L + 1 in P - A, P - B (r: the largest of
// their components) and 1 / (2p); the powers of P - Q fall off with F_n.  Split over
// the two pairs, `grow` bounds the factors on K but those of r (where r is large, K
// is small) and `size` all of them times |K|.
__host__ __device__ inline void ff_pair_range(double p, double K, double r, int L, float& size, float& grow) {
  const float lp = log2f((float)p), lh = fmaxf(0.0f, -lp - 1.0f);
  grow = ((float)L + 1.5f) * fmaxf(0.0f, lp + 1.0f) + fmaxf(0.0f, -0.25f * lp) + ((float)L + 1.0f) * lh;
  size = grow + ((float)L + 1.0f) * fmaxf(0.0f, log2f((float)r) - lh) + log2f((float)(K < 0 ? -K : K));
}
// Largest values for which every quartet of such pairs may run in two floats.  FP32
// ends at 2^128: 2^20 are left to the sums over components, density blocks and
// primitives.  An operation loses at most 2^-149 to underflow; the factors that
// follow make that 2^-45 of the molecule's largest quartet qmax^2 by this estimate,
// 2^-58 without the second 2a that it counts for a steep shell.
// (6-31G* stays within 43 and 50 up to neon.)
constexpr float FF_MAX_SIZE = 54.0f, FF_MAX_GROW = 52.0f;   // the latter plus log2(qmax)

// The type of an exactly representable constant in generated code, and of the
// screening magnitudes: FP32 beside two-float values.
template <typename T> struct ConstOf { using type = T; };
template <> struct ConstOf<ff> { using type = float; };
template <typename T> using const_t = typename ConstOf<T>::type;

}  // namespace gbhf
