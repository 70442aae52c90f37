// The lane-per-ket two-electron gradient kernel and its launches.  Included by
// grad.cu (FP64, FP32) and grad_ff.cu (two-float), which compile side by side.
#pragma once
#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>

#include "gbhf_internal.h"
#include "screen.cuh"
#include "grad_gen.cuh"

namespace gbhf {

// ----------------------------------------------------------- two-electron ----
// Warp per task (bra shell pair, up to 32 kets of one segment, a range of bra
// primitives), as the J/K kernels: the bra primitive pairs are staged in
// shared memory, each lane runs the generated bra-derivative code for its ket
// pair against them, and the warp reduces the six bra-centre components before
// one set of atomics.  Summed over every ordered pair of shell pairs with
// weights (2 - delta_AB)(2 - delta_CD), the bra-centre derivatives give the
// whole two-electron gradient (the ket-centre terms of (P|Q) are the
// bra-centre terms of (Q|P)).

constexpr int GR_THREADS = 128;
constexpr int GR_WARPS = GR_THREADS / 32;

template <typename T, int N>
struct GamReg {
  T v[N];
  __device__ __forceinline__ T get(int i) const { return v[i]; }
  __device__ __forceinline__ void set(int i, T x) { v[i] = x; }
};
template <typename T, int N, int TH>
struct GamSmem {   // per-thread column of a [N][TH] shared array
  T* p;
  // volatile: a read stays where the code places it (the bra loop reads T_ab
  // block by block; hoisted out of the loop, all of T would be live at once)
  __device__ __forceinline__ T get(int i) const {
    if constexpr (std::is_same<T, ff>::value) {
      const unsigned long long b = *(volatile const unsigned long long*)(p + i * TH);
      return ff(__uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
    } else {
      return *(volatile const T*)(p + i * TH);
    }
  }
  __device__ __forceinline__ void set(int i, T x) { p[i * TH] = x; }
};

template <int LA, int LB, int LC, int LD>
struct GradFn;
#define GBHF_GRAD_FN(la, lb, lc, ld, name)                                                                      \
  template <>                                                                                                  \
  struct GradFn<la, lb, lc, ld> {                                                                              \
    template <typename T, typename G, typename TK>                                                             \
    static __device__ __forceinline__ void ket(T invq, T QCx, T QCy, T QCz, T QDx, T QDy, T QDz, const G& gam, \
                                               TK& tk) {                                                       \
      grad_ket_##name<T, G, TK>(invq, QCx, QCy, QCz, QDx, QDy, QDz, gam, tk);                                  \
    }                                                                                                          \
    template <typename T, typename TK>                                                                         \
    static __device__ __forceinline__ void run(const T* sb, int nbra, int bstep, T q, T Qx, T Qy, T Qz, T Kcd, \
                                               const T* boys, const TK& tk, T* g) {                            \
      grad_ketprim_##name<T, TK>(sb, nbra, bstep, q, Qx, Qy, Qz, Kcd, boys, tk, g);                            \
    }                                                                                                          \
  };
GBHF_GRAD_FN(0, 0, 2, 0, ssds)
GBHF_GRAD_FN(0, 0, 2, 1, ssdp)
GBHF_GRAD_FN(1, 0, 2, 0, psds)
GBHF_GRAD_FN(2, 0, 0, 0, dsss)
GBHF_GRAD_FN(2, 0, 1, 0, dsps)
GBHF_GRAD_FN(0, 0, 0, 0, ssss)
GBHF_GRAD_FN(0, 0, 1, 0, ssps)
GBHF_GRAD_FN(0, 0, 1, 1, sspp)
GBHF_GRAD_FN(1, 0, 0, 0, psss)
GBHF_GRAD_FN(1, 0, 1, 0, psps)
GBHF_GRAD_FN(1, 0, 1, 1, pspp)
GBHF_GRAD_FN(1, 1, 0, 0, ppss)
GBHF_GRAD_FN(1, 1, 1, 0, ppps)
GBHF_GRAD_FN(1, 1, 1, 1, pppp)

template <typename T>
struct GradArgs {
  const int4* tasks;
  const int* range;          // start, end of this class and precision
  int* counter;
  const int *poff, *kseg;
  const int4* seg;
  const T* bra;
  const T* ket;
  long long npp;
  const int* shell_atom;     // global atom of each shell (grad index)
  const int* pmol;
  const int* mn;
  const long long* moff;
  const T* D;                // stacked n_m x n_m densities, this precision
  const T* boys;
  double* grad;              // 3 * natoms
  const double* sscale;      // per shell 6 component scales (d shells)
  QuartetScreen scr;         // block maxima of D: a quartet whose bound of |Gamma| is too small is not queued
  const double* Q;           // Schwarz bound of each pair (scr.Qf: in FP32)
  double thr;                // drop a quartet when Q_ab Q_cd max|Gamma_abcd| is below
  float jabs;                // |jcoef|
  T jcoef;                   // weight of the Coulomb term D_ab D_cd in Gamma (0: exchange only)
  const float4* cen;         // two-float kernels: shell centres and the density's scale exponent (as k_jk)
  const int* dexp;
};

// The screening threshold of two-float kernels, whose Gamma is 2^-dex times the
// density's, rounded down by more than the FP32 magnitudes beside it are.
__device__ __forceinline__ float grad_threshold(double thr, int dex) {
  return __double2float_rd(scalbn(thr * (1.0 - 3e-7), -dex));
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One batch: the quartets of bra pair ib with the kets jk of the active lanes,
// kets on the low lg bits of the lane; lanes beyond them split the primitive
// quartets (as in k_jk) and the closing warp sum adds the slices.  STEP: every
// primitive quartet is one tick of the block (k_grad_jk_step), in warp-uniform loops.
template <int LA, int LB, int LC, int LD, typename T, typename GamT, typename TkT, bool STEP = false>
__device__ __forceinline__ void grad_batch(const GradArgs<T>& a, GamT& gam, TkT& tk, const T* sbra, const T* sDab, int ib,
                                           int4 pab, int jk, int4 pcd, bool active, int lg, int lane, int Kb, int4 sg,
                                           int n, const T* __restrict__ Dm, float thrs, int dex) {
  constexpr int NA = ncart_c(LA), NB = ncart_c(LB), NC = ncart_c(LC), ND = ncart_c(LD);
  constexpr bool FF = std::is_same<T, ff>::value;
  using S = const_t<T>;
  const long long npp = a.npp;
  const int A = pab.x, B = pab.y, a0 = pab.z, b0 = pab.w, C = pcd.x, Dd = pcd.y, c0 = pcd.z, d0 = pcd.w;
  const int K = sg.z, len = sg.y - sg.x;
  const int nsl = 32 >> lg, slice = lane >> lg;
  constexpr int KETC = sizeof(T) == 4 ? 1 : 0;   // per-ket-primitive work, as in k_jk
  int lb = 0;
  for (int l = 0, best = 1 << 30; (1 << l) <= nsl; ++l) {
    const int cost = (((Kb + (1 << l) - 1) >> l) + KETC) * ((K + (nsl >> l) - 1) / (nsl >> l));
    if (KETC ? cost < best : cost <= best) {
      best = cost;
      lb = l;
    }
  }
  const int nsb = 1 << lb, nsk = nsl >> lb;
  const int sb = slice & (nsb - 1), sk = slice >> lb;
  T g[6] = {0, 0, 0, 0, 0, 0};
  S wgt = 0;
  bool keep = false;
  ff AC[3];
  if (active) {
    S gmax = S(0);
    // Gamma_abcd = jcoef D_ab D_cd - (D_ac D_bd + D_ad D_bc) / 4
#pragma unroll
    for (int ia = 0; ia < NA; ++ia)
#pragma unroll
      for (int ibb = 0; ibb < NB; ++ibb)
#pragma unroll
        for (int ic = 0; ic < NC; ++ic)
#pragma unroll
          for (int id = 0; id < ND; ++id) {
            const T dab = sDab[ia * NB + ibb];
            const T dcd = Dm[(long long)(c0 + ic) * n + d0 + id];
            const T dac = Dm[(long long)(a0 + ia) * n + c0 + ic];
            const T dbd = Dm[(long long)(b0 + ibb) * n + d0 + id];
            const T dad = Dm[(long long)(a0 + ia) * n + d0 + id];
            const T dbc = Dm[(long long)(b0 + ibb) * n + c0 + ic];
            T gv = a.jcoef * dab * dcd - S(0.25) * (dac * dbd + dad * dbc);
            if constexpr (LA == 2 || LB == 2 || LC == 2 || LD == 2) {   // d components: scaled functions
              if (LA == 2) gv *= T(a.sscale[6 * A + ia]);
              if (LB == 2) gv *= T(a.sscale[6 * B + ibb]);
              if (LC == 2) gv *= T(a.sscale[6 * C + ic]);
              if (LD == 2) gv *= T(a.sscale[6 * Dd + id]);
            }
            gam.set(((ia * NB + ibb) * NC + ic) * ND + id, gv);
            gmax = fmax_t(gmax, mag(gv));
          }
    // exact screening of this quartet by its own Gamma (the task lists bound it
    // by the pairs' density weights)
    if constexpr (sizeof(T) == 4 || FF) keep = a.scr.Qf[ib] * a.scr.Qf[jk] * gmax >= thrs;
    else keep = a.Q[ib] * a.Q[jk] * gmax >= a.thr;
    if constexpr (FF) {
      const float4 a0v = a.cen[3 * A], a1v = a.cen[3 * A + 1], a2v = a.cen[3 * A + 2];
      const float4 c0v = a.cen[3 * C], c1v = a.cen[3 * C + 1], c2v = a.cen[3 * C + 2];
      AC[0] = diff3(a0v.x, a1v.x, a2v.x, c0v.x, c1v.x, c2v.x);
      AC[1] = diff3(a0v.y, a1v.y, a2v.y, c0v.y, c1v.y, c2v.y);
      AC[2] = diff3(a0v.z, a1v.z, a2v.z, c0v.z, c1v.z, c2v.z);
    }
    wgt = (A == B ? S(1) : S(2)) * (C == Dd ? S(1) : S(2));
  }
  const long long base = (long long)sg.w + (jk - sg.x);
  const int nbl = sb < Kb && keep ? (Kb - sb + nsb - 1) / nsb : 0;
  T q = 0, Qx = 0, Qy = 0, Qz = 0, Kcd = 0;
  auto ket_prim = [&](int kc) {
    const long long idx = base + (long long)kc * len;
    q = a.ket[BRA_P * npp + idx];
    const T invq = a.ket[BRA_INVP * npp + idx];
    T QCx = 0, QCy = 0, QCz = 0, QDx = 0, QDy = 0, QDz = 0;
    if (LC >= 1 || FF) {
      QCx = a.ket[BRA_PAX * npp + idx];
      QCy = a.ket[BRA_PAY * npp + idx];
      QCz = a.ket[BRA_PAZ * npp + idx];
    }
    if (LD >= 1) {
      QDx = a.ket[BRA_PBX * npp + idx];
      QDy = a.ket[BRA_PBY * npp + idx];
      QDz = a.ket[BRA_PBZ * npp + idx];
    }
    if constexpr (FF) {   // the bra's P is P - A: Q - A here
      Qx = nrm(QCx - AC[0]);
      Qy = nrm(QCy - AC[1]);
      Qz = nrm(QCz - AC[2]);
    } else {
      Qx = a.ket[BRA_PX * npp + idx];
      Qy = a.ket[BRA_PY * npp + idx];
      Qz = a.ket[BRA_PZ * npp + idx];
    }
    Kcd = a.ket[BRA_K * npp + idx];
    GradFn<LA, LB, LC, LD>::ket(invq, QCx, QCy, QCz, QDx, QDy, QDz, gam, tk);
  };
  if constexpr (STEP) {
    const int nbu = __any_sync(0xffffffffu, keep) ? (Kb + nsb - 1) / nsb : 0;   // the longest lane's
    for (int k0 = 0; nbu > 0 && k0 < K; k0 += nsk) {
      const bool mine = keep && k0 + sk < K;
      if (mine) ket_prim(k0 + sk);
      for (int kb = 0; kb < nbu; ++kb) {
        block_tick(true);
        if (mine && kb < nbl)
          GradFn<LA, LB, LC, LD>::run(sbra + (sb + kb * nsb) * BRA_SB, 1, BRA_SB, q, Qx, Qy, Qz, Kcd, a.boys, tk, g);
      }
    }
  } else {
    for (int kc = sk; keep && kc < K; kc += nsk) {
      ket_prim(kc);
      GradFn<LA, LB, LC, LD>::run(sbra + sb * BRA_SB, nbl, nsb * BRA_SB, q, Qx, Qy, Qz, Kcd, a.boys, tk, g);
    }
  }
#pragma unroll
  for (int x = 0; x < 6; ++x) {
    T v = wgt * g[x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += shfl_xor_t(v, o);
    if (lane == 0) atomicAdd(&a.grad[3 * a.shell_atom[x < 3 ? A : B] + x % 3], widen(v, dex));
  }
}

template <int LA, int LB, int LC, int LD, typename T, bool SG, bool QUEUE>
__global__ void __launch_bounds__(GR_THREADS) k_grad_jk(GradArgs<T> a) {
  constexpr int NA = ncart_c(LA), NB = ncart_c(LB), NC = ncart_c(LC), ND = ncart_c(LD);
  constexpr int NAB = NA * NB, NOUT = NAB * NC * ND;
  __shared__ __align__(16) T sbra[GR_WARPS][KMAX_PRIM_PAIRS * BRA_SB];
  __shared__ T sDab[GR_WARPS][NAB];
  __shared__ int sq[QUEUE ? GR_WARPS : 1][QUEUE_SLOTS];
  extern __shared__ double gsm_dyn[];
  constexpr int NT = NAB * nherm_c(LC + LD);
  using GamT = typename std::conditional<SG, GamSmem<T, NOUT, GR_THREADS>, GamReg<T, NOUT>>::type;
  using TkT = typename std::conditional<SG, GamSmem<T, NT, GR_THREADS>, GamReg<T, NT>>::type;
  GamT gam;
  TkT tk;
  if constexpr (SG) {
    gam.p = reinterpret_cast<T*>(gsm_dyn) + threadIdx.x;
    tk.p = reinterpret_cast<T*>(gsm_dyn) + NOUT * GR_THREADS + threadIdx.x;
  }
  constexpr bool FF = std::is_same<T, ff>::value;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int dex = 0;          // two-float: Gamma is 2^-dex times the density's
  float thrs = (float)a.thr;
  if constexpr (FF) {
    dex = 2 * *a.dexp;
    thrs = grad_threshold(a.thr, dex);
  }
  const int start = a.range[0];
  const int ntask = a.range[1] - start;
  const long long npp = a.npp;
  while (true) {
    int t = 0;
    if (lane == 0) t = atomicAdd(a.counter, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= ntask) break;
    const int4 task = a.tasks[start + t];
    const int ib = task.x;
    const int mol = a.pmol[ib];
    const int n = a.mn[mol];
    const T* __restrict__ Dm = a.D + a.moff[mol];
    const int kb0 = task.w & 0xffff, Kb = (task.w >> 16) - kb0, pb0 = a.poff[ib] + kb0;
    const int4 sg = a.seg[a.kseg[task.y]];
    const unsigned rkb = (65536u + Kb - 1) / Kb;   // idx / Kb = (idx * rkb) >> 16 for idx < 16 * 36
    for (int idx = lane; idx < BRA_NFIELD * Kb; idx += 32) {
      const int f = (int)(((unsigned)idx * rkb) >> 16), k = idx - f * Kb;
      sbra[warp][k * BRA_SB + f] = a.bra[(long long)f * npp + pb0 + k];
    }
    const int4 pab = a.scr.pinfo[ib];
    for (int i = lane; i < NAB; i += 32) sDab[warp][i] = Dm[(long long)(pab.z + i / NB) * n + pab.w + i % NB];
    __syncwarp();
    // the screened kets in full batches, as in k_jk ((H2O)8 FP64 gradient 11.3 -> 10.0 ms)
    if constexpr (QUEUE) {
      const BraScreen bs(a.scr, ib, pab, mol);
      const OneCentre one(a.shell_atom, pab);
      int queued = 0, scanned = 0;
      while (true) {
        while (queued < 32 && scanned < task.z) {
          const int o = scanned + lane;
          const int jk = task.y + o;
          const bool pass = o < task.z && bs.gamma_pass(a.scr, jk, a.jabs, one, a.shell_atom);
          queue_push(sq[warp], queued, jk, pass, lane);
          scanned += 32;
        }
        if (queued == 0) break;
        const int nk = min(queued, 32);
        const int lg = 32 - __clz(nk - 1);
        bool active, bad;
        const int jk = queue_ket(sq[warp], nk, lg, lane, task.y, task.z, active, bad);
        if (bad) a.grad[0] = nan("");
        grad_batch<LA, LB, LC, LD, T, GamT, TkT>(a, gam, tk, sbra[warp], sDab[warp], ib, pab, jk, a.scr.pinfo[jk], active,
                                                 lg, lane, Kb, sg, n, Dm, thrs, dex);
        queue_pop(sq[warp], queued, nk, lane);
      }
    } else {
      const int nk = task.z;
      const int lg = 32 - __clz(max(nk, 1) - 1);
      const bool active = (lane & ((1 << lg) - 1)) < nk;
      const int jk = active ? task.y + (lane & ((1 << lg) - 1)) : task.y;
      const int4 pcd = a.scr.pinfo[jk];
      const bool own = active && !OneCentre(a.shell_atom, pab).holds(a.shell_atom, pcd);
      grad_batch<LA, LB, LC, LD, T, GamT, TkT>(a, gam, tk, sbra[warp], sDab[warp], ib, pab, jk, pcd, own, lg, lane, Kb, sg,
                                               n, Dm, thrs, dex);
      __syncwarp();
    }
  }
}

// The queue form with the block's warps in step.  The two-float code of a (pp|ps)
// primitive quartet is some 7,000 instructions in one run; warps that go through it
// at places of their own fetch it eight times over, and waiting for instructions
// took 80% of their time (0.43 instructions per cycle and SM, 2.9 in (ss|ps)).  Here a
// primitive quartet is one tick: the warps of the block, each with its own batch,
// meet at a barrier before every one and go through the code together.  (H2O)8 FP64
// gradient, (pp|ps) 2.19 -> 1.12 ms, (ps|pp) 0.90 -> 0.42, (pp|ss) 1.64 -> 1.07, (pp|pp)
// 1.26 -> 1.01, the gradient 10.0 -> 7.7; a barrier per batch instead of per tick left
// (pp|ps) at 1.47, its batches being uneven.  Still bound by instruction fetch and by
// waiting at the ticks.  256 threads where registers and shared memory allow, so that
// one block fills the SM.
template <int LA, int LB, int LC, int LD, typename T, bool SG, int TH>
__global__ void __launch_bounds__(TH) k_grad_jk_step(GradArgs<T> a) {
  constexpr int NA = ncart_c(LA), NB = ncart_c(LB), NC = ncart_c(LC), ND = ncart_c(LD);
  constexpr int NAB = NA * NB, NOUT = NAB * NC * ND, W = TH / 32;
  __shared__ __align__(16) T sbra[W][KMAX_PRIM_PAIRS * BRA_SB];
  __shared__ T sDab[W][NAB];
  __shared__ int sq[W][QUEUE_SLOTS];
  extern __shared__ double gsm_dyn[];
  constexpr int NT = NAB * nherm_c(LC + LD);
  using GamT = typename std::conditional<SG, GamSmem<T, NOUT, TH>, GamReg<T, NOUT>>::type;
  using TkT = typename std::conditional<SG, GamSmem<T, NT, TH>, GamReg<T, NT>>::type;
  GamT gam;
  TkT tk;
  if constexpr (SG) {
    gam.p = reinterpret_cast<T*>(gsm_dyn) + threadIdx.x;
    tk.p = reinterpret_cast<T*>(gsm_dyn) + NOUT * TH + threadIdx.x;
  }
  constexpr bool FF = std::is_same<T, ff>::value;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int dex = 0;          // as in k_grad_jk
  float thrs = (float)a.thr;
  if constexpr (FF) {
    dex = 2 * *a.dexp;
    thrs = grad_threshold(a.thr, dex);
  }
  const int start = a.range[0];
  const int ntask = a.range[1] - start;
  int4 task = make_int4(0, 0, 0, 0);
  int queued = 0, scanned = 0;
  bool more = true;   // tasks left
  while (true) {
    // the warp's next batch: survivors of its task, or of the next ones
    while (true) {
      if (scanned < task.z) {
        const int ib = task.x;
        const BraScreen bs(a.scr, ib, a.scr.pinfo[ib], a.pmol[ib]);
        const OneCentre one(a.shell_atom, a.scr.pinfo[ib]);
        while (queued < 32 && scanned < task.z) {
          const int o = scanned + lane;
          const int jk = task.y + o;
          const bool pass = o < task.z && bs.gamma_pass(a.scr, jk, a.jabs, one, a.shell_atom);
          queue_push(sq[warp], queued, jk, pass, lane);
          scanned += 32;
        }
      }
      if (queued > 0 || !more) break;
      int t = 0;
      if (lane == 0) t = atomicAdd(a.counter, 1);
      t = __shfl_sync(0xffffffffu, t, 0);
      more = t < ntask;
      if (!more) {
        task.z = 0;
        break;
      }
      task = a.tasks[start + t];
      scanned = 0;
      const int ib = task.x, mol = a.pmol[ib], n = a.mn[mol];
      const T* __restrict__ Dm = a.D + a.moff[mol];
      const int kb0 = task.w & 0xffff, Kb = (task.w >> 16) - kb0, pb0 = a.poff[ib] + kb0;
      const unsigned rkb = (65536u + Kb - 1) / Kb;
      for (int idx = lane; idx < BRA_NFIELD * Kb; idx += 32) {
        const int f = (int)(((unsigned)idx * rkb) >> 16), k = idx - f * Kb;
        sbra[warp][k * BRA_SB + f] = a.bra[(long long)f * a.npp + pb0 + k];
      }
      const int4 pab = a.scr.pinfo[ib];
      for (int i = lane; i < NAB; i += 32) sDab[warp][i] = Dm[(long long)(pab.z + i / NB) * n + pab.w + i % NB];
      __syncwarp();
    }
    if (queued == 0) break;   // out of work
    {
      const int ib = task.x, mol = a.pmol[ib];
      const int nk = min(queued, 32);
      const int lg = 32 - __clz(nk - 1);
      bool active, bad;
      const int jk = queue_ket(sq[warp], nk, lg, lane, task.y, task.z, active, bad);
      if (bad) a.grad[0] = nan("");
      grad_batch<LA, LB, LC, LD, T, GamT, TkT, true>(a, gam, tk, sbra[warp], sDab[warp], ib, a.scr.pinfo[ib], jk,
                                                     a.scr.pinfo[jk], active, lg, lane,
                                                     (task.w >> 16) - (task.w & 0xffff), a.seg[a.kseg[task.y]],
                                                     a.mn[mol], a.D + a.moff[mol], thrs, dex);
      queue_pop(sq[warp], queued, nk, lane);
    }
  }
  while (block_tick(false)) {   // keeps ticking until the block's other warps are done as well
  }
}

// Code that fits runs better alone: (ps|ps) 0.81 ms, 0.83 in step; (ss|pp) 0.18 and 0.21.
template <int LA, int LB, int LC, int LD, typename T>
constexpr bool grad_in_step() {
  return std::is_same<T, ff>::value && LA < 2 && LB < 2 && LC < 2 && LD < 2 && LA == 1 && (LB == 1 || LD == 1);
}

template <int LA, int LB, int LC, int LD, typename T>
static gbhf_status launch_grad_class(gbhf_ctx* c, cudaStream_t strm, int combo, int prec, const T* D, double* grad,
                                     int ntask) {
  if (ntask <= 0) return GBHF_OK;
  constexpr int NOUT = ncart_c(LA) * ncart_c(LB) * ncart_c(LC) * ncart_c(LD);
  constexpr int NT = ncart_c(LA) * ncart_c(LB) * nherm_c(LC + LD);
  constexpr bool SG = sizeof(T) == 8 ? NOUT > 9 : NOUT > 27;   // Gamma and T in shared memory
  constexpr bool STEP = grad_in_step<LA, LB, LC, LD, T>();
  constexpr int TH = STEP && (NOUT + NT) * 256 * sizeof(T) <= 160 * 1024 ? 256 : GR_THREADS;
  const size_t smem = SG ? (size_t)(NOUT + NT) * TH * sizeof(T) : 0;
  void (*kern)(GradArgs<T>);
  if constexpr (STEP) kern = k_grad_jk_step<LA, LB, LC, LD, T, SG, TH>;
  else kern = k_grad_jk<LA, LB, LC, LD, T, SG, (LA < 2 && LB < 2 && LC < 2 && LD < 2)>;
  static bool attr_set = false;
  if (SG && !attr_set) {
    GBHF_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set = true;
  }
  int per_sm = 0;
  GBHF_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TH, smem));
  per_sm = std::max(per_sm, 1);
  const int grid = std::min(c->nsm * per_sm, (ntask + TH / 32 - 1) / (TH / 32));
  PairData& P = c->pairs;
  TaskLists& gt = c->gtasks;
  GradArgs<T> a;
  a.tasks = gt.tasks[prec].p;
  a.range = gt.ranges.p + 2 * (NTIER * combo + prec);
  a.counter = gt.counters.p + NTIER * combo + prec;
  a.poff = P.poff.p;
  a.kseg = P.kseg.p;
  a.seg = P.seg_info.p;
  a.bra = pair_bra<T>(P);
  a.ket = pair_ket<T>(P);
  a.npp = (long long)P.nprim_pairs;
  a.shell_atom = c->tasks.atom.p;
  a.pmol = P.mol.p;
  a.mn = c->tasks.mn.p;
  a.moff = c->tasks.moff.p;
  a.D = D;
  a.boys = boys_table<T>(c);
  a.cen = c->tasks.cen.p;
  a.dexp = c->dff_exp.p;
  a.grad = grad;
  a.sscale = c->tasks.sscale.p;
  a.Q = P.Q.p;
  a.thr = gt.thr_exact;
  a.scr = quartet_screen(c, gt.thr_exact);
  a.jabs = (float)std::fabs(c->grad_jcoef);
  a.jcoef = T(c->grad_jcoef);
  kern<<<grid, TH, smem, strm>>>(a);
  count_launch(c);
  GBHF_CUDA(c, cudaGetLastError());
  return GBHF_OK;
}

template <typename T>
static gbhf_status launch_grad_combo(gbhf_ctx* c, cudaStream_t strm, int k, int prec, const T* D, double* grad, int nt) {
  switch (k) {   // (bra class, ket class) = (k / 3, k % 3); class 0 = ss, 1 = ps, 2 = pp
    case 0: return launch_grad_class<0, 0, 0, 0, T>(c, strm, k, prec, D, grad, nt);
    case 1: return launch_grad_class<0, 0, 1, 0, T>(c, strm, k, prec, D, grad, nt);
    case 2: return launch_grad_class<0, 0, 1, 1, T>(c, strm, k, prec, D, grad, nt);
    case 3: return launch_grad_class<1, 0, 0, 0, T>(c, strm, k, prec, D, grad, nt);
    case 4: return launch_grad_class<1, 0, 1, 0, T>(c, strm, k, prec, D, grad, nt);
    case 5: return launch_grad_class<1, 0, 1, 1, T>(c, strm, k, prec, D, grad, nt);
    case 6: return launch_grad_class<1, 1, 0, 0, T>(c, strm, k, prec, D, grad, nt);
    case 7: return launch_grad_class<1, 1, 1, 0, T>(c, strm, k, prec, D, grad, nt);
    case 8: return launch_grad_class<1, 1, 1, 1, T>(c, strm, k, prec, D, grad, nt);
    // combinations with a d pair on generated code (GRAD_COMBO_BRA / GRAD_COMBO_KET)
    case 9: return launch_grad_class<0, 0, 2, 0, T>(c, strm, k, prec, D, grad, nt);
    case 10: return launch_grad_class<0, 0, 2, 1, T>(c, strm, k, prec, D, grad, nt);
    case 12: return launch_grad_class<1, 0, 2, 0, T>(c, strm, k, prec, D, grad, nt);
    case 18: return launch_grad_class<2, 0, 0, 0, T>(c, strm, k, prec, D, grad, nt);
    case 19: return launch_grad_class<2, 0, 1, 0, T>(c, strm, k, prec, D, grad, nt);
    default: return fail(c, GBHF_ERR_UNSUPPORTED, "no generated gradient kernel for combo " + std::to_string(k));
  }
}

}  // namespace gbhf
