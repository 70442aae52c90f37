// Analytic RHF nuclear gradient (the backward call).
//
// dE/dR_K = sum_ab D_ab dH_ab/dR_K + 1/2 sum_abcd Gamma_abcd d(ab|cd)/dR_K
//           - sum_ab W_ab dS_ab/dR_K + dV_nn/dR_K
// with D = 2 C_occ C_occ^T, W = 2 sum_i eps_i C_i C_i^T and
// Gamma_abcd = D_ab D_cd - (D_ac D_bd + D_ad D_bc)/4.  This is the gradient
// the reference's (uncompiled) energyGradient (HartreeFock/Derivatives.hs:40-48)
// intends, including the Hellmann-Feynman operator term that it zeroes
// (Derivatives.hs:144).  Derivatives of primitive Gaussians follow
// d/dA_x [x_A^i exp(-a r_A^2)] = 2a x_A^(i+1) exp(..) - i x_A^(i-1) exp(..)
// (as calcDervCGF, Derivatives.hs:246-257), applied to the Hermite expansion
// coefficients: dE^(ij)_t/dA_x = 2a E^(i+1,j)_t - i E^(i-1,j)_t.
// Translational invariance gives the fourth centre of an ERI and the
// operator centre of a nuclear-attraction integral.
//
// Open shell (UHF): with D = D_a + D_b, D_s = D_a - D_b and
// W = sum_s C_s,occ eps_s C_s,occ^T, the two-electron density is
// Gamma = D_ab D_cd - (D_a,ac D_a,bd + D_b,ac D_b,bd + D_a,ad D_a,bc + D_b,ad D_b,bc)/2
//       = Gamma_RHF(D) - (D_s,ac D_s,bd + D_s,ad D_s,bc)/4,
// so the kernels run twice: on D as above, and on D_s with the Coulomb
// weight jcoef = 0 (gradient_uhf_dev).
#include <algorithm>
#include <cmath>
#include <vector>

#include "gbhf_internal.h"
#include "gbhf_md.cuh"
#include "grad_kern.cuh"

namespace gbhf {

// Gradient combinations with a d pair evaluated by the generated lane-per-ket
// code; the others go to the warp-per-quartet kernels of gradd.cu.
bool grad_gen_combo(int k) {
  return k < NGCOMBO_SP || k == 9 || k == 10 || k == 12 || k == 18 || k == 19;
}

// Two-electron gradient of D (n x n, device) into d_grad (accumulated).  With
// profiling events the launches run in order on the context stream, each timed
// into prof.gcls_ms; otherwise round-robin on the side streams.
gbhf_status grad_2e(gbhf_ctx* c, const double* d_D, double schwarz, double mixed_cutoff, int precision,
                           double* d_grad) {
  GBHF_TRY(build_grad_tasks(c, d_D, schwarz, mixed_cutoff, precision));
  TaskLists& gt = c->gtasks;
  gt.thr_exact = schwarz;   // per-quartet Gamma test in the kernels
  int nts[NCOMBO_MAX][NTIER];
  for (int k = 0; k < NCOMBO_MAX; ++k)
    for (int t = 0; t < NTIER; ++t)
      nts[k][t] = gt.hranges[2 * (NTIER * k + t) + 1] - gt.hranges[2 * (NTIER * k + t)];
  const bool ev = c->prof.events;
  int ne = 0, ev_combo[NTIER * NCOMBO_MAX], ev_prec[NTIER * NCOMBO_MAX];
  SideFork side(c->stream, c->fork_ev, c->side, c->join_ev, gbhf_ctx::NSIDE_GRAD);
  if (ev) GBHF_CUDA(c, cudaEventRecord(c->evg[0], c->stream));
  else GBHF_CUDA(c, side.fork());
  int nl = 0;
  // heaviest first: the d combinations, then the s/p ones
  static const int order[NCOMBO_MAX] = {35, 34, 29, 33, 28, 23, 32, 27, 22, 17, 31, 26, 21, 16, 11, 30, 25, 20,
                                        15, 14, 10, 24, 19, 13, 9, 18, 12, 8, 7, 5, 6, 4, 2, 3, 1, 0};
  static const int tiers[NTIER] = {TIER_64, TIER_FF, TIER_32};
  for (const int tier : tiers) {
    for (int oi = 0; oi < NCOMBO_MAX; ++oi) {
      const int k = order[oi];
      const int nt = nts[k][tier];
      if (nt <= 0) continue;
      cudaStream_t strm = ev ? c->stream : c->side[nl++ % gbhf_ctx::NSIDE_GRAD];
      if (!grad_gen_combo(k)) GBHF_TRY(launch_grad_dclass(c, strm, k, tier, d_D, d_grad, nt));
      else if (tier == TIER_64) GBHF_TRY(launch_grad_combo<double>(c, strm, k, tier, d_D, d_grad, nt));
      else if (tier == TIER_32) GBHF_TRY(launch_grad_combo<float>(c, strm, k, tier, c->dfloat.p, d_grad, nt));
      else GBHF_TRY(launch_grad_ff(c, strm, k, d_grad, nt));
      if (ev) {
        ev_combo[ne] = k;
        ev_prec[ne] = tier == TIER_32 ? 1 : 0;   // two-float work counts as FP64 in the profile
        ++ne;
        GBHF_CUDA(c, cudaEventRecord(c->evg[ne], c->stream));
      }
    }
  }
  if (!ev) {
    GBHF_CUDA(c, side.join());
    return GBHF_OK;
  }
  GBHF_CUDA(c, cudaEventSynchronize(c->evg[ne]));
  for (int e = 0; e < ne; ++e) {
    float ms = 0;
    GBHF_CUDA(c, cudaEventElapsedTime(&ms, c->evg[e], c->evg[e + 1]));
    c->prof.gcls_ms[ev_combo[e]][ev_prec[e]] += ms;
  }
  return GBHF_OK;
}

// ---------------------------------------------------------- one-electron ----
// Eight lanes per function pair (a <= b), primitive pairs shared out among them:
// D-weighted derivatives of T and W-weighted derivatives of S (translational
// invariance gives d/dB = -d/dA).  Primitive pairs whose weighted prefactor is
// below 1e-17 are skipped.  The nuclear attraction follows in k_grad_vne.  A thread
// per pair walked up to 36 primitive pairs alone: 0.46 ms for one water and for eight
// alike.
constexpr int G1_THREADS = 64, G1_LANES = 8;

// Molecule-aware: row i (global function) pairs with the functions j >= i of
// its molecule; D and W are the stacked n_m x n_m blocks; the operator centres
// are the molecule's atoms.
struct Grad1eArgs {
  const double* xyz;
  const double* Z;
  const int* fn;            // per global CGF: atom (global), lx, ly, lz, np, off
  const double* coef;
  const double* expo;
  const double* tab;
  const int* fmol;          // per global CGF: molecule
  const int* mfo;           // per molecule: first function (nmol+1)
  const int* mao;           // per molecule: first atom (nmol+1)
  const long long* moff;    // per molecule: block offset in D, W
  const double* D;
  const double* W;
  double* grad;             // 3 * total atoms
};

__global__ void __launch_bounds__(G1_THREADS) k_grad_1e(Grad1eArgs g) {
  const int i = blockIdx.y;
  const int mol = g.fmol[i];
  const int f0m = g.mfo[mol], nm = g.mfo[mol + 1] - f0m;
  const int il = i - f0m;
  const int jl = (blockIdx.x * blockDim.x + threadIdx.x) / G1_LANES;   // local column
  const int sub = threadIdx.x % G1_LANES;
  double gA[3] = {0, 0, 0};   // d/dA of (D T - W S); d/dB = -d/dA
  int atA = 0, atB = 0;
  const double* __restrict__ xyz = g.xyz;
  const double* __restrict__ coef = g.coef;
  const double* __restrict__ expo = g.expo;
  double* __restrict__ grad = g.grad;
  if (jl < nm && jl >= il) {
    const int j = f0m + jl;
    const DevFn f = load_fn(g.fn, i), gfn = load_fn(g.fn, j);
    const double *A = xyz + 3 * f.atom, *B = xyz + 3 * gfn.atom;
    const double mult = (i == j) ? 1.0 : 2.0;
    const double dab = mult * g.D[g.moff[mol] + (long)il * nm + jl], wab = mult * g.W[g.moff[mol] + (long)il * nm + jl];
    double ab2 = 0;
    for (int x = 0; x < 3; ++x) ab2 += (A[x] - B[x]) * (A[x] - B[x]);
    atA = f.atom;
    atB = gfn.atom;
    for (int r = sub; r < f.np * gfn.np; r += G1_LANES) {
        const int p1 = r / gfn.np, p2 = r - p1 * gfn.np;
        const double c1 = coef[f.off + p1], a = expo[f.off + p1];
        const double c2 = coef[gfn.off + p2], b = expo[gfn.off + p2];
        const double p = a + b, mu = a * b / p;
        const double kab = c1 * c2 * exp(-mu * ab2);
        if (fabs(kab) * (1.0 + p) * (fabs(dab) * (1.0 + p) + fabs(wab)) * (GBHF_PI / p) * sqrt(GBHF_PI / p) < 1e-17)
          continue;
        const double cte = sqrt(GBHF_PI / p);
        double P[3], s[3][4][5];   // up to l_a + 1 <= 3 on A, l_b + 2 <= 4 on B
        for (int x = 0; x < 3; ++x) {
          P[x] = (a * A[x] + b * B[x]) / p;
          const double abx = A[x] - B[x];
          // table up to i+1 on A and j+2 on B (kinetic)
          const double s00 = exp(-mu * abx * abx) * cte;
          const double c = 1.0 / (2.0 * p);
          const double pax = P[x] - A[x], pbx = P[x] - B[x];
          for (int m = 0; m <= f.l[x] + 1; ++m)
            for (int nn = 0; nn <= gfn.l[x] + 2; ++nn) {
              double v;
              if (m == 0 && nn == 0) v = s00;
              else if (m == 0) v = pbx * s[x][0][nn - 1] + (nn >= 2 ? c * (nn - 1) * s[x][0][nn - 2] : 0.0);
              else if (nn == 0) v = pax * s[x][m - 1][0] + (m >= 2 ? c * (m - 1) * s[x][m - 2][0] : 0.0);
              else v = pax * s[x][m - 1][nn] + c * ((m >= 2 ? (m - 1) * s[x][m - 2][nn] : 0.0) + nn * s[x][m - 1][nn - 1]);
              s[x][m][nn] = v;
            }
        }
        auto S1 = [&](int x, int m, int nn) { return (m < 0 || nn < 0) ? 0.0 : s[x][m][nn]; };
        auto T1 = [&](int x, int m, int nn) {   // kinetic 1-D term
          if (m < 0) return 0.0;
          return -2.0 * b * b * S1(x, m, nn + 2) + b * (2 * nn + 1) * S1(x, m, nn) -
                 (nn >= 2 ? 0.5 * nn * (nn - 1) * S1(x, m, nn - 2) : 0.0);
        };
        double sx[3], tx[3], dsx[3], dtx[3];
        for (int x = 0; x < 3; ++x) {
          const int li = f.l[x], lj = gfn.l[x];
          sx[x] = S1(x, li, lj);
          tx[x] = T1(x, li, lj);
          dsx[x] = 2 * a * S1(x, li + 1, lj) - li * S1(x, li - 1, lj);
          dtx[x] = 2 * a * T1(x, li + 1, lj) - li * T1(x, li - 1, lj);
        }
        for (int dir = 0; dir < 3; ++dir) {
          // d/dA_dir of S and T: the axis-dir factor becomes 2a f(i+1) - i f(i-1)
          double dS = 1.0, dT = 0;
          for (int x = 0; x < 3; ++x) dS *= (x == dir) ? dsx[x] : sx[x];
          for (int k = 0; k < 3; ++k) {
            double term = 1.0;
            for (int x = 0; x < 3; ++x) {
              if (x == k) term *= (x == dir) ? dtx[x] : tx[x];
              else term *= (x == dir) ? dsx[x] : sx[x];
            }
            dT += term;
          }
          gA[dir] += c1 * c2 * (dab * dT - wab * dS);
        }
    }
  }
#pragma unroll
  for (int x = 0; x < 3; ++x) {
#pragma unroll
    for (int o = G1_LANES / 2; o > 0; o >>= 1) gA[x] += __shfl_xor_sync(0xffffffffu, gA[x], o);
    if (sub == 0 && jl < nm && jl >= il) {
      atomicAdd(&grad[3 * atA + x], gA[x]);
      atomicAdd(&grad[3 * atB + x], -gA[x]);
    }
  }
}

// Nuclear-attraction terms: warp per shell pair of class (LA, LB), lanes over the
// molecule's nuclei; generated per-primitive-pair code (grad_gen.cuh).  The pair
// covers (a, b) and (b, a) when A != B (weight 2).  Bra-centre sums are reduced
// over the warp; each lane adds the operator-centre term -(dA + dB) of its nucleus.
template <int LA, int LB>
struct VneFn;
template <>
struct VneFn<0, 0> {
  static __device__ __forceinline__ void run(const BraPrim<double>& bp, double x, double y, double z, double zp,
                                             const double* dw, const double* boys, double* g) {
    vne_grad_ss<double>(bp, x, y, z, zp, dw, boys, g);
  }
};
template <>
struct VneFn<1, 0> {
  static __device__ __forceinline__ void run(const BraPrim<double>& bp, double x, double y, double z, double zp,
                                             const double* dw, const double* boys, double* g) {
    vne_grad_ps<double>(bp, x, y, z, zp, dw, boys, g);
  }
};
template <>
struct VneFn<1, 1> {
  static __device__ __forceinline__ void run(const BraPrim<double>& bp, double x, double y, double z, double zp,
                                             const double* dw, const double* boys, double* g) {
    vne_grad_pp<double>(bp, x, y, z, zp, dw, boys, g);
  }
};
template <>
struct VneFn<2, 0> {
  static __device__ __forceinline__ void run(const BraPrim<double>& bp, double x, double y, double z, double zp,
                                             const double* dw, const double* boys, double* g) {
    vne_grad_ds<double>(bp, x, y, z, zp, dw, boys, g);
  }
};
template <>
struct VneFn<2, 1> {
  static __device__ __forceinline__ void run(const BraPrim<double>& bp, double x, double y, double z, double zp,
                                             const double* dw, const double* boys, double* g) {
    vne_grad_dp<double>(bp, x, y, z, zp, dw, boys, g);
  }
};
template <>
struct VneFn<2, 2> {
  static __device__ __forceinline__ void run(const BraPrim<double>& bp, double x, double y, double z, double zp,
                                             const double* dw, const double* boys, double* g) {
    vne_grad_dd<double>(bp, x, y, z, zp, dw, boys, g);
  }
};

struct VneArgs {
  int p0, p1;               // pairs of this class
  const int *pA, *pB, *pK, *poff, *pmol;
  const double* bra;        // pair-contiguous primitive-pair fields
  long long npp;
  const int* shell_f0;      // within the molecule
  const int* shell_atom;
  const double* sscale;     // per shell 6 component scales (d shells)
  const int* mn;
  const long long* moff;
  const int* mao;           // first atom of each molecule (nmol + 1)
  const double* xyz;
  const double* Z;
  const double* D;          // stacked
  const double* boys;       // FP64 Horner tables
  double kvf;               // 2 pi / sqrt(2 pi^2.5): K' of the pair data -> 2 pi/p c c exp(-mu AB^2)
  double* grad;
};

template <int LA, int LB>
__global__ void __launch_bounds__(128) k_grad_vne(VneArgs a) {
  constexpr int NA = ncart_c(LA), NB = ncart_c(LB);
  const int lane = threadIdx.x & 31;
  const int pr = a.p0 + blockIdx.x * 4 + (threadIdx.x >> 5);
  if (pr >= a.p1) return;
  const int A = a.pA[pr], B = a.pB[pr], mol = a.pmol[pr], n = a.mn[mol];
  const double* Dm = a.D + a.moff[mol];
  const int fa = a.shell_f0[A], fb = a.shell_f0[B];
  const double mult = A == B ? 1.0 : 2.0;
  double dw[NA * NB];
  double dmax = 0;
#pragma unroll
  for (int ia = 0; ia < NA; ++ia)
#pragma unroll
    for (int ib = 0; ib < NB; ++ib) {
      dw[ia * NB + ib] = mult * Dm[(long)(fa + ia) * n + fb + ib] * a.sscale[6 * A + ia] * a.sscale[6 * B + ib];
      dmax = fmax(dmax, fabs(dw[ia * NB + ib]));
    }
  double gAB[6] = {0, 0, 0, 0, 0, 0};
  const int K = a.pK[pr];
  const long long po = a.poff[pr];
  const int c0 = a.mao[mol], c1 = a.mao[mol + 1];
  // nuclei on the low lanes; with few of them the rest of the warp shares the primitives
  // (lane per nucleus: one water's 36 primitive pairs were walked by three lanes)
  const int lgc = c1 - c0 >= 17 ? 5 : 32 - __clz(max(c1 - c0, 1) - 1);
  const int slice = lane >> lgc, nslice = 32 >> lgc;
  for (int cb = c0; cb < c1; cb += 32) {
    const int cn = cb + (lane & ((1 << lgc) - 1));
    if (cn < c1) {
      const double Cx = a.xyz[3 * cn], Cy = a.xyz[3 * cn + 1], Cz = a.xyz[3 * cn + 2], Zc = a.Z[cn];
      double gC[3] = {0, 0, 0};
      for (int k = slice; k < K; k += nslice) {
        BraPrim<double> bp;
        const long long idx = po + k;
        bp.p = a.bra[BRA_P * a.npp + idx];
        bp.invp = a.bra[BRA_INVP * a.npp + idx];
        bp.Px = a.bra[BRA_PX * a.npp + idx];
        bp.Py = a.bra[BRA_PY * a.npp + idx];
        bp.Pz = a.bra[BRA_PZ * a.npp + idx];
        bp.PAx = a.bra[BRA_PAX * a.npp + idx];
        bp.PAy = a.bra[BRA_PAY * a.npp + idx];
        bp.PAz = a.bra[BRA_PAZ * a.npp + idx];
        bp.PBx = a.bra[BRA_PBX * a.npp + idx];
        bp.PBy = a.bra[BRA_PBY * a.npp + idx];
        bp.PBz = a.bra[BRA_PBZ * a.npp + idx];
        bp.K = a.bra[BRA_K * a.npp + idx];
        bp.a = a.bra[BRA_AEXP * a.npp + idx];
        const double zpref = -Zc * bp.K * a.kvf;
        if (fabs(zpref) * dmax * (1.0 + bp.p) < 1e-17) continue;
        double g6[6] = {0, 0, 0, 0, 0, 0};
        VneFn<LA, LB>::run(bp, Cx, Cy, Cz, zpref, dw, a.boys, g6);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          gAB[x] += g6[x];
          gAB[3 + x] += g6[3 + x];
          gC[x] -= g6[x] + g6[3 + x];
        }
      }
#pragma unroll
      for (int x = 0; x < 3; ++x)
        if (gC[x] != 0.0) atomicAdd(&a.grad[3 * cn + x], gC[x]);
    }
  }
#pragma unroll
  for (int x = 0; x < 6; ++x) {
    const double v = warp_sum_d(gAB[x]);
    if (lane == 0 && v != 0.0) atomicAdd(&a.grad[3 * a.shell_atom[x < 3 ? A : B] + x % 3], v);
  }
}

template <int LA, int LB>
static gbhf_status launch_vne(gbhf_ctx* c, cudaStream_t strm, int cls, const double* d_D, double* d_grad) {
  PairData& P = c->pairs;
  VneArgs a;
  a.p0 = P.cls_start[cls];
  a.p1 = P.cls_start[cls + 1];
  if (a.p1 <= a.p0) return GBHF_OK;
  a.pA = P.A.p;
  a.pB = P.B.p;
  a.pK = P.K.p;
  a.poff = P.poff.p;
  a.pmol = P.mol.p;
  a.bra = P.bra64.p;
  a.npp = (long long)P.nprim_pairs;
  a.shell_f0 = c->tasks.f0.p;
  a.shell_atom = c->tasks.atom.p;
  a.sscale = c->tasks.sscale.p;
  a.mn = c->tasks.mn.p;
  a.moff = c->tasks.moff.p;
  a.mao = c->tasks.mao.p;
  a.xyz = c->d_xyz.p;
  a.Z = c->d_Z.p;
  a.D = d_D;
  a.boys = c->boysh64.p;
  a.kvf = 2.0 * GBHF_PI / std::sqrt(TWO_PI_2P5);
  a.grad = d_grad;
  k_grad_vne<LA, LB><<<(a.p1 - a.p0 + 3) / 4, 128, 0, strm>>>(a);
  count_launch(c);
  GBHF_CUDA(c, cudaGetLastError());
  return GBHF_OK;
}

// Nuclear repulsion gradient, one thread per atom: -sum_L Z_K Z_L (R_K - R_L) / R_KL^3
// over the atoms L of the same molecule.
__global__ void k_grad_nuc(int natoms, const int* __restrict__ amol, const int* __restrict__ mao,
                           const double* __restrict__ xyz, const double* __restrict__ Z, double* __restrict__ grad) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= natoms) return;
  const int m = amol[k];
  double g[3] = {0, 0, 0};
  for (int l = mao[m]; l < mao[m + 1]; ++l) {
    if (l == k) continue;
    double d[3], r2 = 0;
    for (int x = 0; x < 3; ++x) {
      d[x] = xyz[3 * k + x] - xyz[3 * l + x];
      r2 += d[x] * d[x];
    }
    const double f = Z[k] * Z[l] / (r2 * sqrt(r2));
    for (int x = 0; x < 3; ++x) g[x] -= f * d[x];
  }
  for (int x = 0; x < 3; ++x) grad[3 * k + x] += g[x];
}

// Host driver: D and W square (device), gradient into d_grad (3*natoms, device).
gbhf_status gradient_dev(gbhf_ctx* c, const double* d_D, const double* d_W, double schwarz, double mixed_cutoff,
                         int precision, double* d_grad) {
  const Basis& b = c->basis;
  if (!b.shells_ok || b.maxL > 2)
    return fail(c, GBHF_ERR_UNSUPPORTED, "gradient kernels need complete s, p and d shells");
  GBHF_TRY(ensure_boys_tables(c));
  GBHF_TRY(ensure_pairs(c));
  const int n = b.nbf, na = b.natoms;
  GBHF_TRY(ensure_shell_arrays(c));
  GBHF_CUDA(c, cudaMemsetAsync(d_grad, 0, 3 * na * sizeof(double), c->stream));
  k_grad_nuc<<<(na + 127) / 128, 128, 0, c->stream>>>(na, c->tasks.amol.p, c->tasks.mao.p, c->d_xyz.p, c->d_Z.p,
                                                      d_grad);
  int max_fn = 0;
  for (int m = 0; m < b.nmol; ++m) max_fn = std::max(max_fn, b.mol_fn_off[m + 1] - b.mol_fn_off[m]);
  Grad1eArgs g1;
  g1.xyz = c->d_xyz.p;
  g1.Z = c->d_Z.p;
  g1.fn = c->d_fn.p;
  g1.coef = c->d_coef.p;
  g1.expo = c->d_exp.p;
  g1.tab = c->boys64.p;
  g1.fmol = c->tasks.fmol.p;
  g1.mfo = c->tasks.mfo.p;
  g1.mao = c->tasks.mao.p;
  g1.moff = c->tasks.moff.p;
  g1.D = d_D;
  g1.W = d_W;
  g1.grad = d_grad;
  // The one-electron terms are short launches of few warps: they run beside the
  // two-electron task lists and kernels, on the side streams that those leave free
  // (one after another before them: (H2O)8 FP64 gradient 7.3 ms, beside them and with the
  // primitives shared out 6.1; (H2O)5/6-31G* mixed 10.8 and 8.5; one water's energy and
  // gradient 6.5 and 5.6).
  // With profiling events everything stays in order on the context's stream.
  constexpr int S0 = gbhf_ctx::NSIDE_GRAD, NS = gbhf_ctx::NSIDE - S0;
  static_assert(NS >= 1, "side streams for the one-electron terms");
  const bool beside = !c->prof.events;
  auto strm = [&](int k) { return beside ? c->side[S0 + k % NS] : c->stream; };
  SideFork side(c->stream, c->fork_ev, c->side + S0, c->join_ev + S0, NS);
  if (beside) GBHF_CUDA(c, side.fork());
  constexpr int PB = G1_THREADS / G1_LANES;
  k_grad_1e<<<dim3((max_fn + PB - 1) / PB, n), G1_THREADS, 0, strm(0)>>>(g1);
  count_launch(c, 2);
  GBHF_CUDA(c, cudaGetLastError());
  GBHF_TRY((launch_vne<2, 2>(c, strm(1), 5, d_D, d_grad)));
  GBHF_TRY((launch_vne<1, 1>(c, strm(2), 2, d_D, d_grad)));
  GBHF_TRY((launch_vne<1, 0>(c, strm(3), 1, d_D, d_grad)));
  GBHF_TRY((launch_vne<2, 1>(c, strm(2), 4, d_D, d_grad)));
  GBHF_TRY((launch_vne<2, 0>(c, strm(3), 3, d_D, d_grad)));
  GBHF_TRY((launch_vne<0, 0>(c, strm(0), 0, d_D, d_grad)));
  GBHF_TRY(grad_2e(c, d_D, schwarz, mixed_cutoff, precision, d_grad));
  if (beside) GBHF_CUDA(c, side.join());
  GBHF_CUDA(c, cudaStreamSynchronize(c->stream));
  return GBHF_OK;
}

// W = 2 sum_{i < nocc} eps_i C_i C_i^T  (energy-weighted density)
__global__ void k_scale_occ(int n, int nocc, const double* __restrict__ C, const double* __restrict__ eps,
                            double* __restrict__ out) {
  const int i = blockIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nocc) return;
  out[(long)i * nocc + j] = C[(long)i * n + j] * eps[j];
}

// UHF gradient: D_a, D_b and W square (device), gradient into d_grad.
gbhf_status gradient_uhf_dev(gbhf_ctx* c, const double* d_Da, const double* d_Db, const double* d_W, double schwarz,
                             double mixed_cutoff, int precision, double* d_grad) {
  const size_t nn = (size_t)c->basis.nbf * c->basis.nbf;
  DBuf<double> DT, DS;
  GBHF_CUDA(c, DT.alloc(nn));
  GBHF_CUDA(c, DS.alloc(nn));
  GBHF_TRY(axpby(c, nn, 1.0, d_Da, 1.0, d_Db, DT.p));
  GBHF_TRY(axpby(c, nn, 1.0, d_Da, -1.0, d_Db, DS.p));
  GBHF_TRY(gradient_dev(c, DT.p, d_W, schwarz, mixed_cutoff, precision, d_grad));
  c->grad_jcoef = 0.0;
  const gbhf_status st = grad_2e(c, DS.p, schwarz, mixed_cutoff, precision, d_grad);
  c->grad_jcoef = 1.0;
  GBHF_TRY(st);
  GBHF_CUDA(c, cudaStreamSynchronize(c->stream));
  return GBHF_OK;
}

gbhf_status energy_weighted_density(gbhf_ctx* c, int n, int nocc, const double* d_C, const double* d_eps,
                                    double* d_W) {
  if (nocc <= 0) {
    GBHF_CUDA(c, cudaMemsetAsync(d_W, 0, (size_t)n * n * sizeof(double), c->stream));
    return GBHF_OK;
  }
  GBHF_WS(c, T, 23, (size_t)n * nocc);
  k_scale_occ<<<dim3((nocc + 127) / 128, n), 128, 0, c->stream>>>(n, nocc, d_C, d_eps, T);
  count_launch(c);
  // W = 2 (C eps)_occ C_occ^T with C_occ the first nocc columns of C (ldb = n)
  GBHF_TRY(gemm(c, false, true, n, n, nocc, 2.0, T, nocc, d_C, n, 0.0, d_W, n));
  GBHF_CUDA(c, cudaStreamSynchronize(c->stream));
  return GBHF_OK;
}

}  // namespace gbhf
