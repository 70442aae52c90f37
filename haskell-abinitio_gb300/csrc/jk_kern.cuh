// The lane-per-ket J/K kernel and its launches (see jk.cu for the task lists).
// Included by jk.cu (FP64, FP32) and jk_ff.cu (two-float), which compile side by side.
#pragma once
#include <algorithm>
#include <string>
#include <type_traits>

#include "gbhf_internal.h"
#include "screen.cuh"

namespace gbhf {


template <typename T, int N>
struct RegAcc {
  T v[N];
  __device__ __forceinline__ T& operator[](int i) { return v[i]; }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = T(0);
  }
  __device__ __forceinline__ T get(int i) const { return v[i]; }
};

template <typename T, int N, int TH>
struct SmemAcc {
  T* p;   // this thread's column, stride blockDim (TH)
  __device__ __forceinline__ T& operator[](int i) { return p[i * TH]; }
  __device__ __forceinline__ void zero() {
#pragma unroll 4
    for (int i = 0; i < N; ++i) p[i * TH] = T(0);
  }
  __device__ __forceinline__ T get(int i) const { return p[i * TH]; }
};

// Bra primitives of a lane and of the warp's longest lane (k_jk_step).
struct StepCount {
  int own, all;
};
__device__ __forceinline__ int nb_end(StepCount n) { return n.all; }
__device__ __forceinline__ bool nb_skip(StepCount n, int kb) {
  block_tick(true);
  return kb >= n.own;
}

}  // namespace gbhf

#include "eri_gen.cuh"

namespace gbhf {

template <typename T>
struct JKArgs {
  const int4* tasks;
  const int* range;    // [start, end)
  int* counter;
  const int* poff;
  const int* kseg;
  const int4* seg;
  const T* bra;
  const T* ket;
  long long npp;
  const int* pmol;             // molecule of each pair
  const int* mn;               // functions per molecule
  const long long* moff;       // offset of each molecule's block in D and G
  const T* D;                  // stacked n_m x n_m densities
  double* G;                   // stacked n_m x n_m Fock accumulators
  const T* boys;
  unsigned long long* stats;   // [shell quartets, fn quartets, prim quartets]
  const double* sscale;        // per shell 6 component scales (d shells)
  int with_j;                  // 0: exchange only (the open-shell spin-density build)
  QuartetScreen scr;           // drop a quartet when Q_ab Q_cd max|D| over its six density blocks is below scr.thr
  const float4* cen;           // two-float kernels: three FP32 parts of each shell's centre
  const int* dexp;             // and the exponent e of the scale 2^-e of D
};

template <int LA, int LB, int LC, int LD>
struct ClassFn;

#define GBHF_CLASS_FN(la, lb, lc, ld, name)                                                              \
  template <>                                                                                            \
  struct ClassFn<la, lb, lc, ld> {                                                                       \
    template <typename T, typename Acc, typename NB>                                                     \
    static __device__ __forceinline__ void run(const T* sb, NB nbra, int bstep, T q, T invq, T Qx, T Qy, T Qz,  \
                                               T QCx, T QCy, T QCz, T QDx, T QDy, T QDz, T Kcd,           \
                                               const T* boys, Acc& acc) {                                 \
      eri_ketprim_##name<T, Acc, NB>(sb, nbra, bstep, q, invq, Qx, Qy, Qz, QCx, QCy, QCz, QDx, QDy, QDz, Kcd, boys, \
                                 acc);                                                                   \
    }                                                                                                    \
  };
GBHF_CLASS_FN(0, 0, 0, 0, ssss)
GBHF_CLASS_FN(1, 0, 0, 0, psss)
GBHF_CLASS_FN(1, 0, 1, 0, psps)
GBHF_CLASS_FN(0, 0, 1, 1, sspp)
GBHF_CLASS_FN(1, 0, 1, 1, pspp)
GBHF_CLASS_FN(1, 1, 1, 1, pppp)
GBHF_CLASS_FN(2, 0, 0, 0, dsss)
GBHF_CLASS_FN(2, 0, 1, 0, dsps)
GBHF_CLASS_FN(2, 0, 1, 1, dspp)
GBHF_CLASS_FN(2, 0, 2, 0, dsds)
GBHF_CLASS_FN(2, 1, 0, 0, dpss)
GBHF_CLASS_FN(2, 1, 1, 0, dpps)
GBHF_CLASS_FN(2, 2, 0, 0, ddss)

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ ff warp_sum(ff v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += shfl_xor_t(v, o);
  return v;
}

constexpr int JK_THREADS = 128;
constexpr int JK_WARPS = JK_THREADS / 32;

// One batch: the quartets of bra pair ib with the kets jk of the lanes that
// `keep` one, kets on the low lg bits of the lane.  STEP: every primitive quartet is
// one tick of the block (k_jk_step), in warp-uniform loops.
template <int LA, int LB, int LC, int LD, typename T, typename AccT, bool STEP = false>
__device__ __forceinline__ void jk_batch(const JKArgs<T>& a, AccT& acc, const T* sbra, const T* sDab, int ib, int4 pab,
                                         int jk, int4 pcd, bool keep, int lg, int lane, int kb0, int Kb, int4 sg, int n,
                                         const T* __restrict__ Dm, double* __restrict__ Gm, int dex,
                                         unsigned long long& cnt_q, unsigned long long& cnt_p) {
  constexpr int NA = ncart_c(LA), NB = ncart_c(LB), NC = ncart_c(LC), ND = ncart_c(LD);
  constexpr int NAB = NA * NB, NCD = NC * ND, NOUT = NAB * NCD;
  constexpr bool FF = std::is_same<T, ff>::value;
  using S = const_t<T>;
  const long long npp = a.npp;
  const int K = sg.z, len = sg.y - sg.x;   // ket primitive pairs, kets of the segment
  // lanes beyond the batch's kets split the primitive quartets: kets sit on the
  // low lg bits of the lane (nk <= 2^lg), the rest of the lane is the slice;
  // the nsl slices form an nsb x (nsl / nsb) grid over bra and ket primitives
  const int nsl = 32 >> lg;
  const int slice = lane >> lg;
  // the classes whose per-lane pair has the higher momentum transform it once
  // per call (ket primitive and bra-primitive range): about one primitive
  // quartet of extra work per call
  constexpr int CALLC = (LA + LB < LC + LD) ? 1 : 0;
  // per ket primitive a lane also loads the ket pair's fields and enters the
  // bra loop: about one FP32 primitive quartet of issue slots, next to nothing
  // beside the FP64 arithmetic of an FP64 primitive quartet
  constexpr int KETC = sizeof(T) == 4 ? 1 : 0;
  int lb = 0;
  for (int l = 0, best = 1 << 30; (1 << l) <= nsl; ++l) {   // least work for the busiest lane
    const int cost = (((Kb + (1 << l) - 1) >> l) + CALLC + KETC) * ((K + (nsl >> l) - 1) / (nsl >> l));
    if (KETC ? cost < best : cost <= best) {
      best = cost;
      lb = l;
    }
  }
  const int nsb = 1 << lb, nsk = nsl >> lb;
  const int sb = slice & (nsb - 1), sk = slice >> lb;
  const bool lead_k = keep && slice == 0;               // scatters
  const int A = pab.x, B = pab.y, a0 = pab.z, b0 = pab.w;
  const int C = pcd.x, Dd = pcd.y, c0 = pcd.z, d0 = pcd.w;
  acc.zero();
  if (!STEP && keep) {
    const long long base = (long long)sg.w + (jk - sg.x);
    const int nbl = sb < Kb ? (Kb - sb + nsb - 1) / nsb : 0;   // this lane's bra primitives
    ff AC[3];
    if constexpr (FF) {
      const float4 a0v = a.cen[3 * A], a1v = a.cen[3 * A + 1], a2v = a.cen[3 * A + 2];
      const float4 c0v = a.cen[3 * C], c1v = a.cen[3 * C + 1], c2v = a.cen[3 * C + 2];
      AC[0] = diff3(a0v.x, a1v.x, a2v.x, c0v.x, c1v.x, c2v.x);
      AC[1] = diff3(a0v.y, a1v.y, a2v.y, c0v.y, c1v.y, c2v.y);
      AC[2] = diff3(a0v.z, a1v.z, a2v.z, c0v.z, c1v.z, c2v.z);
    }
    for (int kc = sk; kc < K; kc += nsk) {
      const long long idx = base + (long long)kc * len;
      const T q = a.ket[BRA_P * npp + idx];
      const T invq = a.ket[BRA_INVP * npp + idx];
      T Qx, Qy, Qz;
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
      const T Kcd = a.ket[BRA_K * npp + idx];
      ClassFn<LA, LB, LC, LD>::template run<T, AccT>(sbra + sb * BRA_SB, nbl, nsb * BRA_SB, q, invq,
                                                     Qx, Qy, Qz, QCx, QCy, QCz, QDx, QDy, QDz, Kcd, a.boys, acc);
    }
    cnt_q += lead_k && kb0 == 0;
    cnt_p += (unsigned long long)nbl * (sk < K ? (K - sk + nsk - 1) / nsk : 0);
  }
  if constexpr (STEP) {   // the same, warp-uniform: lanes without a primitive quartet come along for the ticks
    static_assert(FF, "two-float kernels");
    const long long base = (long long)sg.w + (jk - sg.x);
    const int nbl = keep && sb < Kb ? (Kb - sb + nsb - 1) / nsb : 0;   // this lane's bra primitives
    ff AC[3];
    if (keep) {
      const float4 a0v = a.cen[3 * A], a1v = a.cen[3 * A + 1], a2v = a.cen[3 * A + 2];
      const float4 c0v = a.cen[3 * C], c1v = a.cen[3 * C + 1], c2v = a.cen[3 * C + 2];
      AC[0] = diff3(a0v.x, a1v.x, a2v.x, c0v.x, c1v.x, c2v.x);
      AC[1] = diff3(a0v.y, a1v.y, a2v.y, c0v.y, c1v.y, c2v.y);
      AC[2] = diff3(a0v.z, a1v.z, a2v.z, c0v.z, c1v.z, c2v.z);
    }
    const int all = __any_sync(0xffffffffu, keep) ? (Kb + nsb - 1) / nsb : 0;
    for (int k0 = 0; all > 0 && k0 < K; k0 += nsk) {
      const bool mine = keep && k0 + sk < K;
      T q = 0, invq = 0, Qx = 0, Qy = 0, Qz = 0, Kcd = 0;
      T QCx = 0, QCy = 0, QCz = 0, QDx = 0, QDy = 0, QDz = 0;
      if (mine) {
        const long long idx = base + (long long)(k0 + sk) * len;
        q = a.ket[BRA_P * npp + idx];
        invq = a.ket[BRA_INVP * npp + idx];
        QCx = a.ket[BRA_PAX * npp + idx];
        QCy = a.ket[BRA_PAY * npp + idx];
        QCz = a.ket[BRA_PAZ * npp + idx];
        if (LD >= 1) {
          QDx = a.ket[BRA_PBX * npp + idx];
          QDy = a.ket[BRA_PBY * npp + idx];
          QDz = a.ket[BRA_PBZ * npp + idx];
        }
        Qx = nrm(QCx - AC[0]);
        Qy = nrm(QCy - AC[1]);
        Qz = nrm(QCz - AC[2]);
        Kcd = a.ket[BRA_K * npp + idx];
      }
      ClassFn<LA, LB, LC, LD>::template run<T, AccT>(sbra + sb * BRA_SB, StepCount{mine ? nbl : 0, all}, nsb * BRA_SB, q,
                                                     invq, Qx, Qy, Qz, QCx, QCy, QCz, QDx, QDy, QDz, Kcd, a.boys, acc);
    }
    if (keep) {
      cnt_q += lead_k && kb0 == 0;
      cnt_p += (unsigned long long)nbl * (sk < K ? (K - sk + nsk - 1) / nsk : 0);
    }
  }
  // warp-uniform: sum the slices (every lane ends with the total of its ket)
  for (int o = 1 << lg; o < 32; o <<= 1) {
#pragma unroll
    for (int i = 0; i < NOUT; ++i) acc[i] += shfl_xor_t(acc.get(i), o);
  }
  if constexpr (LA == 2 || LB == 2 || LC == 2 || LD == 2) {
    // d shells: the generated code used the first component's coefficients
    if (keep) {
#pragma unroll
      for (int e = 0; e < NOUT; ++e) {
        const int ab = e / NCD, cd = e - ab * NCD;
        T f = T(1);
        if (LA == 2) f *= T(a.sscale[6 * A + ab / NB]);
        if (LB == 2) f *= T(a.sscale[6 * B + ab % NB]);
        if (LC == 2) f *= T(a.sscale[6 * C + cd / ND]);
        if (LD == 2) f *= T(a.sscale[6 * Dd + cd % ND]);
        acc[e] = acc.get(e) * f;
      }
    }
  }
  // ---- scatter into G'' (FP64 atomics)
  const S s = (A == B ? S(0.5) : S(1)) * (C == Dd ? S(0.5) : S(1)) * (ib == jk ? S(0.5) : S(1));
  T dcd[NCD];
#pragma unroll
  for (int ic = 0; ic < NC; ++ic)
#pragma unroll
    for (int id = 0; id < ND; ++id) dcd[ic * ND + id] = lead_k ? Dm[(long long)(c0 + ic) * n + d0 + id] : T(0);
  // J_ab (warp reduce over kets)
  if (a.with_j) {
#pragma unroll
    for (int ab = 0; ab < NAB; ++ab) {
      T v = 0;
#pragma unroll
      for (int cd = 0; cd < NCD; ++cd) v = fma_t(acc.get(ab * NCD + cd), dcd[cd], v);
      v = warp_sum(S(2) * s * v);   // s depends on the lane's ket: apply before the reduction
      if (lane == 0) atomicAdd(&Gm[(long long)(a0 + ab / NB) * n + b0 + ab % NB], widen(v, dex));
    }
  }
  if (lead_k) {
    // J_cd
    if (a.with_j) {
#pragma unroll
      for (int cd = 0; cd < NCD; ++cd) {
        T v = 0;
#pragma unroll
        for (int ab = 0; ab < NAB; ++ab) v = fma_t(acc.get(ab * NCD + cd), sDab[ab], v);
        atomicAdd(&Gm[(long long)(c0 + cd / ND) * n + d0 + cd % ND], widen(S(2) * s * v, dex));
      }
    }
    const S ks = S(-0.5) * s;
    // K_ac -= sum_bd v D_bd ; K_ad -= sum_bc v D_bc
#pragma unroll
    for (int ia = 0; ia < NA; ++ia) {
#pragma unroll
      for (int ic = 0; ic < NC; ++ic) {
        T v = 0;
#pragma unroll
        for (int ibb = 0; ibb < NB; ++ibb)
#pragma unroll
          for (int id = 0; id < ND; ++id)
            v = fma_t(acc.get((ia * NB + ibb) * NCD + ic * ND + id), Dm[(long long)(b0 + ibb) * n + d0 + id], v);
        atomicAdd(&Gm[(long long)(a0 + ia) * n + c0 + ic], widen(ks * v, dex));
      }
#pragma unroll
      for (int id = 0; id < ND; ++id) {
        T v = 0;
#pragma unroll
        for (int ibb = 0; ibb < NB; ++ibb)
#pragma unroll
          for (int ic = 0; ic < NC; ++ic)
            v = fma_t(acc.get((ia * NB + ibb) * NCD + ic * ND + id), Dm[(long long)(b0 + ibb) * n + c0 + ic], v);
        atomicAdd(&Gm[(long long)(a0 + ia) * n + d0 + id], widen(ks * v, dex));
      }
    }
    // K_bc -= sum_ad v D_ad ; K_bd -= sum_ac v D_ac
#pragma unroll
    for (int ibb = 0; ibb < NB; ++ibb) {
#pragma unroll
      for (int ic = 0; ic < NC; ++ic) {
        T v = 0;
#pragma unroll
        for (int ia = 0; ia < NA; ++ia)
#pragma unroll
          for (int id = 0; id < ND; ++id)
            v = fma_t(acc.get((ia * NB + ibb) * NCD + ic * ND + id), Dm[(long long)(a0 + ia) * n + d0 + id], v);
        atomicAdd(&Gm[(long long)(b0 + ibb) * n + c0 + ic], widen(ks * v, dex));
      }
#pragma unroll
      for (int id = 0; id < ND; ++id) {
        T v = 0;
#pragma unroll
        for (int ia = 0; ia < NA; ++ia)
#pragma unroll
          for (int ic = 0; ic < NC; ++ic)
            v = fma_t(acc.get((ia * NB + ibb) * NCD + ic * ND + id), Dm[(long long)(a0 + ia) * n + c0 + ic], v);
        atomicAdd(&Gm[(long long)(b0 + ibb) * n + d0 + id], widen(ks * v, dex));
      }
    }
  }
}

template <int LA, int LB, int LC, int LD, typename T, bool SACC, bool QUEUE>
__global__ void __launch_bounds__(JK_THREADS) k_jk(JKArgs<T> a) {
  constexpr int NA = ncart_c(LA), NB = ncart_c(LB), NC = ncart_c(LC), ND = ncart_c(LD);
  constexpr int NAB = NA * NB, NOUT = NAB * NC * ND;
  __shared__ __align__(16) T sbra[JK_WARPS][KMAX_PRIM_PAIRS * BRA_SB];
  __shared__ T sDab[JK_WARPS][NAB > 1 ? NAB : 1];
  __shared__ int sq[QUEUE ? JK_WARPS : 1][QUEUE_SLOTS];   // kets that passed the screening
  constexpr bool FF = std::is_same<T, ff>::value;
  extern __shared__ double sacc_dyn[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int dex = FF ? *a.dexp : 0;   // two-float: D is 2^-dex times the density
  const int start = a.range[0];
  const int ntask = a.range[1] - start;
  unsigned long long cnt_q = 0, cnt_p = 0;
  using AccT = typename std::conditional<SACC, SmemAcc<T, NOUT, JK_THREADS>, RegAcc<T, NOUT>>::type;
  AccT acc;
  if constexpr (SACC) acc.p = reinterpret_cast<T*>(sacc_dyn) + threadIdx.x;
  const long long npp = a.npp;
  while (true) {
    int t = 0;
    if (lane == 0) t = atomicAdd(a.counter, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= ntask) break;
    const int4 task = a.tasks[start + t];
    const int ib = task.x;
    const int kb0 = task.w & 0xffff, Kb = (task.w >> 16) - kb0, pb0 = a.poff[ib] + kb0;
    const int4 sg = a.seg[a.kseg[task.y]];   // the task's kets share their segment
    // the molecule's density and Fock blocks (stacked matrices)
    const int mol = a.pmol[ib];
    const int n = a.mn[mol];
    const T* __restrict__ Dm = a.D + a.moff[mol];
    double* __restrict__ Gm = a.G + a.moff[mol];
    // bra primitives [kb0, kb1) of pair ib
    const unsigned rkb = (65536u + Kb - 1) / Kb;   // idx / Kb = (idx * rkb) >> 16 for idx < 16 * 36
    for (int idx = lane; idx < BRA_NJK * Kb; idx += 32) {
      const int f = (int)(((unsigned)idx * rkb) >> 16), k = idx - f * Kb;
      sbra[warp][k * BRA_SB + f] = a.bra[(long long)f * npp + pb0 + k];
    }
    const int4 pab = a.scr.pinfo[ib];
    for (int i = lane; i < NAB; i += 32) sDab[warp][i] = Dm[(long long)(pab.z + i / NB) * n + pab.w + i % NB];
    __syncwarp();
    const BraScreen bs(a.scr, ib, pab, mol);
    if constexpr (QUEUE) {
      int queued = 0, scanned = 0;
      while (true) {
        // full batches of 32 surviving kets, then the rest
        while (queued < 32 && scanned < task.z) {
          const int o = scanned + lane;
          const int jk = task.y + o;
          const bool pass = o < task.z && bs.jk_pass(a.scr, jk);
          queue_push(sq[warp], queued, jk, pass, lane);
          scanned += 32;
        }
        if (queued == 0) break;
        const int nk = min(queued, 32);
        const int lg = 32 - __clz(nk - 1);   // ceil(log2(nk)), 0 for one ket
        bool keep, bad;
        const int jk = queue_ket(sq[warp], nk, lg, lane, task.y, task.z, keep, bad);
        if (bad) Gm[0] = nan("");
        jk_batch<LA, LB, LC, LD, T, AccT>(a, acc, sbra[warp], sDab[warp], ib, pab, jk, a.scr.pinfo[jk], keep, lg, lane,
                                          kb0, Kb, sg, n, Dm, Gm, dex, cnt_q, cnt_p);
        queue_pop(sq[warp], queued, nk, lane);
      }
    } else {   // a task holds at most 32 kets: one batch, screened in place
      const int nk = task.z;
      const int lg = 32 - __clz(max(nk, 1) - 1);
      const bool active = (lane & ((1 << lg) - 1)) < nk;
      const int jk = active ? task.y + (lane & ((1 << lg) - 1)) : task.y;
      const bool keep = active && bs.jk_pass(a.scr, jk);
      jk_batch<LA, LB, LC, LD, T, AccT>(a, acc, sbra[warp], sDab[warp], ib, pab, jk, a.scr.pinfo[jk], keep, lg, lane, kb0,
                                        Kb, sg, n, Dm, Gm, dex, cnt_q, cnt_p);
      __syncwarp();
    }
  }
  // statistics (one atomic per warp and counter)
  cnt_q = (unsigned long long)warp_sum((double)cnt_q);
  cnt_p = (unsigned long long)warp_sum((double)cnt_p);
  if (lane == 0 && a.stats) {
    atomicAdd(&a.stats[0], cnt_q);
    atomicAdd(&a.stats[1], cnt_q * (unsigned long long)(NOUT));
    atomicAdd(&a.stats[2], cnt_p);
  }
}

// The queue form with the block's warps in step, as k_grad_jk_step and for the same
// reason (the two-float code of these two classes was waiting for instructions most of
// the time): (H2O)16 FP64, (ps|pp) 1.76 -> 1.30 ms, (pp|pp) 1.10 -> 0.90, the build 6.7
// -> 5.9; (H2O)64 mixed build 55.7 -> 51.8.  Eight warps a block: with four the builds
// took 6.4 and 53.9 ms.  The other classes' code fits the caches.
template <int LA, int LB, int LC, int LD, typename T, bool SACC, int TH>
__global__ void __launch_bounds__(TH) k_jk_step(JKArgs<T> a) {
  constexpr int NA = ncart_c(LA), NB = ncart_c(LB), NC = ncart_c(LC), ND = ncart_c(LD);
  constexpr int NAB = NA * NB, NOUT = NAB * NC * ND, W = TH / 32;
  __shared__ __align__(16) T sbra[W][KMAX_PRIM_PAIRS * BRA_SB];
  __shared__ T sDab[W][NAB > 1 ? NAB : 1];
  __shared__ int sq[W][QUEUE_SLOTS];
  constexpr bool FF = std::is_same<T, ff>::value;
  extern __shared__ double sacc_dyn[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int dex = FF ? *a.dexp : 0;
  const int start = a.range[0];
  const int ntask = a.range[1] - start;
  unsigned long long cnt_q = 0, cnt_p = 0;
  using AccT = typename std::conditional<SACC, SmemAcc<T, NOUT, TH>, RegAcc<T, NOUT>>::type;
  AccT acc;
  if constexpr (SACC) acc.p = reinterpret_cast<T*>(sacc_dyn) + threadIdx.x;
  int4 task = make_int4(0, 0, 0, 0);
  int queued = 0, scanned = 0;
  bool more = true;   // tasks left
  while (true) {
    // the warp's next batch: survivors of its task, or of the next ones
    while (true) {
      if (scanned < task.z) {
        const int ib = task.x;
        const BraScreen bs(a.scr, ib, a.scr.pinfo[ib], a.pmol[ib]);
        while (queued < 32 && scanned < task.z) {
          const int o = scanned + lane;
          const int jk = task.y + o;
          const bool pass = o < task.z && bs.jk_pass(a.scr, jk);
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
      for (int idx = lane; idx < BRA_NJK * Kb; idx += 32) {
        const int f = (int)(((unsigned)idx * rkb) >> 16), k = idx - f * Kb;
        sbra[warp][k * BRA_SB + f] = a.bra[(long long)f * a.npp + pb0 + k];
      }
      const int4 pab = a.scr.pinfo[ib];
      for (int i = lane; i < NAB; i += 32) sDab[warp][i] = Dm[(long long)(pab.z + i / NB) * n + pab.w + i % NB];
      __syncwarp();
    }
    if (queued == 0) break;   // out of work
    const int ib = task.x, mol = a.pmol[ib], kb0 = task.w & 0xffff;
    const int nk = min(queued, 32);
    const int lg = 32 - __clz(nk - 1);
    bool keep, bad;
    const int jk = queue_ket(sq[warp], nk, lg, lane, task.y, task.z, keep, bad);
    if (bad) a.G[a.moff[mol]] = nan("");
    jk_batch<LA, LB, LC, LD, T, AccT, true>(a, acc, sbra[warp], sDab[warp], ib, a.scr.pinfo[ib], jk, a.scr.pinfo[jk],
                                            keep, lg, lane, kb0, (task.w >> 16) - kb0, a.seg[a.kseg[task.y]], a.mn[mol],
                                            a.D + a.moff[mol], a.G + a.moff[mol], dex, cnt_q, cnt_p);
    queue_pop(sq[warp], queued, nk, lane);
  }
  while (block_tick(false)) {   // keeps ticking until the block's other warps are done as well
  }
  cnt_q = (unsigned long long)warp_sum((double)cnt_q);
  cnt_p = (unsigned long long)warp_sum((double)cnt_p);
  if (lane == 0 && a.stats) {
    atomicAdd(&a.stats[0], cnt_q);
    atomicAdd(&a.stats[1], cnt_q * (unsigned long long)(NOUT));
    atomicAdd(&a.stats[2], cnt_p);
  }
}

template <int LA, int LB, int LC, int LD, typename T>
constexpr bool jk_in_step() {
  return std::is_same<T, ff>::value && LA == 1 && LC == 1 && LD == 1 && LB < 2;
}

template <int LA, int LB, int LC, int LD, typename T, bool SACC>
static gbhf_status launch_class(gbhf_ctx* c, cudaStream_t strm, int combo, int prec, const T* D, double* G, int ntask,
                                int with_j) {
  if (ntask <= 0) return GBHF_OK;
  constexpr int NOUT = ncart_c(LA) * ncart_c(LB) * ncart_c(LC) * ncart_c(LD);
  constexpr bool STEP = jk_in_step<LA, LB, LC, LD, T>();
  constexpr int TH = STEP ? 256 : JK_THREADS;
  const size_t smem = SACC ? (size_t)NOUT * TH * sizeof(T) : 0;
  // The queue packs the survivors of a task's kets into full batches (s/p classes;
  // a d task is one batch of at most 32 kets): (ps|ss) FP32 of (H2O)64 17.5 ->
  // 11.9 ms, (ss|ss) 10.7 -> 7.1, the whole mixed build 84.6 -> 61 ms.  The d classes
  // keep the plain form: the (dd|ss) instance of the queue form read out of bounds on
  // the device.  Its cause was not found: the queue holds every ket once and in range
  // (host test), the staging, the density block of 36 entries, the accumulator's shared
  // memory (36.9 KB beside 20.6 KB static, opted in) and every index of the batch are in
  // bounds by reading, and the instance's registers and stack frame (8 bytes, (dp|ps) 80)
  // do not set it apart.
  void (*kern)(JKArgs<T>);
  if constexpr (STEP) kern = k_jk_step<LA, LB, LC, LD, T, SACC, TH>;
  else kern = k_jk<LA, LB, LC, LD, T, SACC, (LA < 2 && LB < 2 && LC < 2 && LD < 2)>;
  static bool attr_set = false;
  if (SACC && !attr_set) {
    GBHF_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set = true;
  }
  int per_sm = 0;
  GBHF_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TH, smem));
  per_sm = std::max(per_sm, 1);
  int grid = std::min(c->nsm * per_sm, (ntask + TH / 32 - 1) / (TH / 32));
  PairData& P = c->pairs;
  JKArgs<T> a;
  a.tasks = c->tasks.tasks[prec].p;
  a.range = c->tasks.ranges.p + 2 * (NTIER * combo + prec);
  a.counter = c->tasks.counters.p + NTIER * combo + prec;
  a.poff = P.poff.p;
  a.kseg = P.kseg.p;
  a.seg = P.seg_info.p;
  a.bra = pair_bra<T>(P);
  a.ket = pair_ket<T>(P);
  a.npp = (long long)P.nprim_pairs;
  a.pmol = P.mol.p;
  a.mn = c->tasks.mn.p;
  a.moff = c->tasks.moff.p;
  a.D = D;
  a.G = G;
  a.boys = boys_table<T>(c);
  a.stats = c->tasks.stats.p + 3 * (NTIER * combo + prec);
  a.sscale = c->tasks.sscale.p;
  a.with_j = with_j;
  a.scr = quartet_screen(c, c->tasks.thr_exact);
  a.cen = c->tasks.cen.p;
  a.dexp = c->dff_exp.p;
  kern<<<grid, TH, smem, strm>>>(a);
  count_launch(c);
  GBHF_CUDA(c, cudaGetLastError());
  return GBHF_OK;
}


// The generated lane-per-ket kernels.  FP64 and two-float values take two
// registers each: their larger classes accumulate in shared memory.
template <typename T>
static gbhf_status launch_combo(gbhf_ctx* c, cudaStream_t strm, int k, int prec, const T* D, double* G, int nt, int wj) {
  constexpr bool W = sizeof(T) == 8;
  switch (k) {
    case 0: return launch_class<0, 0, 0, 0, T, false>(c, strm, k, prec, D, G, nt, wj);
    case 1: return launch_class<1, 0, 0, 0, T, false>(c, strm, k, prec, D, G, nt, wj);
    case 2: return launch_class<1, 0, 1, 0, T, false>(c, strm, k, prec, D, G, nt, wj);
    case 3: return launch_class<0, 0, 1, 1, T, false>(c, strm, k, prec, D, G, nt, wj);
    case 4: return launch_class<1, 0, 1, 1, T, false>(c, strm, k, prec, D, G, nt, wj);
    case 5: return launch_class<1, 1, 1, 1, T, W>(c, strm, k, prec, D, G, nt, wj);
    case 6: return launch_class<2, 0, 0, 0, T, false>(c, strm, k, prec, D, G, nt, wj);
    case 7: return launch_class<2, 0, 1, 0, T, false>(c, strm, k, prec, D, G, nt, wj);
    case 8: return launch_class<2, 0, 1, 1, T, W>(c, strm, k, prec, D, G, nt, wj);
    case 9: return launch_class<2, 0, 2, 0, T, W>(c, strm, k, prec, D, G, nt, wj);
    case 10: return launch_class<2, 1, 0, 0, T, false>(c, strm, k, prec, D, G, nt, wj);
    case 11: return launch_class<2, 1, 1, 0, T, W>(c, strm, k, prec, D, G, nt, wj);
    case 15: return launch_class<2, 2, 0, 0, T, W>(c, strm, k, prec, D, G, nt, wj);
    default: return fail(c, GBHF_ERR_UNSUPPORTED, "no generated J/K kernel for class " + std::to_string(k));
  }
}

}  // namespace gbhf
