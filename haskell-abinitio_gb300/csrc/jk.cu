// Direct J/K Fock build: screened task lists and per-class ERI+scatter kernels.
//
// Unique shell quartets (AB|CD): bra pair of class X, ket pair of class Y
// with X >= Y, and within one class ket index <= bra index, which visits
// each quartet of the 8-fold permutation orbit once.  With the degeneracy
// weight s = (A==B ? 1/2 : 1)(C==D ? 1/2 : 1)(AB==CD ? 1/2 : 1) every
// component integral v = (ab|cd) adds, to a non-symmetric accumulator G'',
//   G''_ab += 2 s v D_cd,  G''_cd += 2 s v D_ab,
//   G''_ac -= s v D_bd/2,  G''_bc -= s v D_ad/2,  G''_ad -= s v D_bc/2,  G''_bd -= s v D_ac/2,
// and G = G'' + G''^T equals J - K/2 of the reference's calcGmatrix
// (HartreeFock/HartreeFock.hs:225-241): G_ab = sum_kl D_lk [(ab|kl) - (al|kb)/2].
//
// Work decomposition: a task is (bra pair, consecutive kets of one ket segment,
// a range of bra primitives); one warp runs one task.  An s/p task holds up to
// 32, 128 or 256 kets: the warp screens them by the density and evaluates the
// survivors 32 at a time, lane = ket (screen.cuh); a d task holds at most 32, or
// one where a warp evaluates one quartet (jkd.cu).  Kets inside a segment share
// the primitive-pair count, so lanes do equal work; the segment is sorted by
// Schwarz bound, so the kets that pass Q_bra Q_ket w >= cutoff form a prefix
// found by binary search, and the split between the precision tiers (FP64,
// two-float, FP32 in mixed precision) is two more prefix boundaries.  Two-float
// tier (gbhf_ff.cuh): full FP64 build of (H2O)16/6-31G 26.1 -> 8.0 ms, mixed one
// of (H2O)64 144 -> 88 ms (FP64 launches 75 ms, FP64 + two-float 21 ms).  Warps
// pull tasks from a per-kernel atomic counter; only the blocks of the two in-step
// kernels wait, for their own warps (block_tick).
#include <algorithm>
#include <cstring>
#include <functional>

#include "gbhf_internal.h"
#include "jk_kern.cuh"

namespace gbhf {

// ------------------------------------------------------- Schwarz bounds ----
// Q_AB = sqrt(max_ab (ab|ab)) for the pairs of one class (bra = ket = pair),
// with the generated FP64 class code; one warp per pair, its primitive pairs
// staged in the warp's slice of shared memory, lanes over (bra primitive,
// slice of the ket primitives) so that pairs with few primitives still fill
// the warp.
constexpr int SCHWARZ_WARPS = 4;   // 4 x 4608 B of staged primitives per block

template <int LA, int LB>
__global__ void __launch_bounds__(SCHWARZ_WARPS * 32) k_schwarz_cls(int p0, int p1, const int* __restrict__ pK,
                                                                     const int* __restrict__ poff,
                                                                     const double* __restrict__ bra, long long npp,
                                                                     const double* __restrict__ boys,
                                                                     double* __restrict__ Q) {
  constexpr int NA = ncart_c(LA), NB = ncart_c(LB), NAB = NA * NB;
  __shared__ __align__(16) double sb[SCHWARZ_WARPS][KMAX_PRIM_PAIRS * BRA_SB];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = p0 + blockIdx.x * SCHWARZ_WARPS + warp;
  if (t >= p1) return;   // whole warps
  const int K = pK[t];
  const long long o = poff[t];
  double* s = sb[warp];
  for (int idx = lane; idx < BRA_NFIELD * K; idx += 32) {
    const int f = idx / K, k = idx - f * K;
    s[k * BRA_SB + f] = bra[f * npp + o + k];
  }
  __syncwarp();
  const int nch = max(1, min(K, 32 / max(K, 1)));
  const int cs = (K + nch - 1) / nch;
  RegAcc<double, NAB * NAB> acc;
  acc.zero();
  for (int it = lane; it < K * nch; it += 32) {
    const int k = it / nch, ch = it - k * nch;
    const int k0 = ch * cs, nk = min(K, k0 + cs) - k0;
    if (nk <= 0) continue;
    auto g = [&](int f) { return s[k * BRA_SB + f]; };
    ClassFn<LA, LB, LA, LB>::template run<double, RegAcc<double, NAB * NAB>>(
        s + k0 * BRA_SB, nk, BRA_SB, g(BRA_P), g(BRA_INVP), g(BRA_PX), g(BRA_PY), g(BRA_PZ), g(BRA_PAX), g(BRA_PAY),
        g(BRA_PAZ), g(BRA_PBX), g(BRA_PBY), g(BRA_PBZ), g(BRA_K), boys, acc);
  }
  double mx = 0;
#pragma unroll
  for (int ab = 0; ab < NAB; ++ab) mx = fmax(mx, fabs(warp_sum(acc.get(ab * NAB + ab))));
  if (lane == 0) Q[t] = sqrt(mx);
}

gbhf_status schwarz_classes_dev(gbhf_ctx* c, const int* cls_start, const int* d_K, const int* d_poff,
                                const double* d_bra, long long npp, double* d_Q) {
  for (int cl = 0; cl < 3; ++cl) {   // s/p classes; jkd.cu has the d classes
    const int p0 = cls_start[cl], p1 = cls_start[cl + 1];
    if (p1 <= p0) continue;
    const int blocks = (p1 - p0 + SCHWARZ_WARPS - 1) / SCHWARZ_WARPS, thr = SCHWARZ_WARPS * 32;
    if (cl == 0)
      k_schwarz_cls<0, 0><<<blocks, thr, 0, c->stream>>>(p0, p1, d_K, d_poff, d_bra, npp, c->boysh64.p, d_Q);
    else if (cl == 1)
      k_schwarz_cls<1, 0><<<blocks, thr, 0, c->stream>>>(p0, p1, d_K, d_poff, d_bra, npp, c->boysh64.p, d_Q);
    else
      k_schwarz_cls<1, 1><<<blocks, thr, 0, c->stream>>>(p0, p1, d_K, d_poff, d_bra, npp, c->boysh64.p, d_Q);
    count_launch(c);
    GBHF_CUDA(c, cudaGetLastError());
  }
  return GBHF_OK;
}

// ------------------------------------------------------------ task lists ----

struct TaskGenArgs {
  int nitems;
  int ncombo;                    // quartet classes (bra pair class, ket pair class)
  int cbra[NCOMBO_MAX], cket[NCOMBO_MAX];
  int all_pairs;                 // every ordered (bra, ket) pair, else each unordered pair once in one class
  int ket_ge[NCOMBO_MAX];        // one class: 1 = (i | j >= i), the bra with more primitives; 0 = (i | j <= i)
  int lane_prims[NCOMBO_MAX];    // per combo: primitive quartets per lane and task (bra split)
  int task_kets[NCOMBO_MAX];     // per combo: kets per task (32: a lane per ket; fewer: a warp per quartet)
  int square_w;                  // bound uses the squared density weight (gradient)
  const int* item_combo_start;   // ncombo+1 item offsets
  const int* cls_start;          // NPCLS+1
  const int* seg_cls_start;      // NPCLS+1
  int nmol;
  const int* pmol;               // molecule of each pair
  const int* mseg;               // ket segments of (class, molecule)
  const int* mact;               // per molecule: 1 = build its quartets (nullptr: all)
  const int4* seg;
  const double* Q;
  const int* pK;                 // primitive pairs per shell pair
  double thr_all, thr64;         // cutoff / weight, mixed cutoff / weight
  const FFLimit* ffq;            // per molecule: two-float below its Q_ab Q_cd ...
  double ffw;                    // ... or below this weighted bound (mixed precision), see ff_weighted_limit
  const double* pw;              // per-pair density weight (local mode) or nullptr
  const double* sw;              // per-segment max of pw (local mode)
  int* count;                    // NTIER per item
  const int* off;                // exclusive scans, NTIER x (nitems + 1)
  int4* tasks[NTIER];            // FP64, FP32, two-float
  int fine_div[2][NTIER], fine_kets[2][NTIER];   // finer tasks by (d classes, tier): divisor of lane_prims, most kets
};

__device__ __forceinline__ int count_ge(const double* Q, int lo, int hi, double thr) {
  // Q descending on [lo, hi): number of entries with Q >= thr
  int a = lo, b = hi;
  while (a < b) {
    int m = (a + b) >> 1;
    if (Q[m] >= thr) a = m + 1;
    else b = m;
  }
  return a - lo;
}

template <bool FILL>
__global__ void k_tasks(TaskGenArgs g) {
  const int it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= g.nitems) return;
  int k = 0;
  while (k + 1 < g.ncombo && it >= g.item_combo_start[k + 1]) ++k;
  const int X = g.cbra[k], Y = g.cket[k];
  const int i = g.cls_start[X] + (it - g.item_combo_start[k]);
  const double qi = (g.mact && !g.mact[g.pmol[i]]) ? 0.0 : g.Q[i];   // inactive molecule: no tasks
  int nt[NTIER] = {0, 0, 0}, wt[NTIER] = {0, 0, 0};
  if (FILL)
#pragma unroll
    for (int t = 0; t < NTIER; ++t) wt[t] = g.off[(size_t)t * (g.nitems + 1) + it];
  const double wi = g.pw ? g.pw[i] : 1.0;
  const int kb = g.pK[i];
  if (qi > 0) {
    const int m = g.pmol[i];
    const double ffq = g.ffq[m].off ? 0.0 : g.ffq[m].q;
    const int s_lo = g.mseg[2 * (Y * g.nmol + m)], s_hi = g.mseg[2 * (Y * g.nmol + m) + 1];
    for (int sidx = s_lo; sidx < s_hi; ++sidx) {
      const int4 s = g.seg[sidx];
      // bound of (bra|ket) contributions: Q_bra Q_ket max(w_bra, max w over the ket segment)
      double w = g.pw ? fmax(wi, g.sw[sidx]) : 1.0;
      if (g.square_w) w *= w;
      if (!(w > 0)) continue;
      const double ta = g.thr_all / (qi * w), t64 = g.thr64 / (qi * w);
      // one class: each unordered pair of pairs once.  Pairs are sorted by
      // primitive count (descending) within a (class, molecule), so with
      // (i | j >= i) the bra - staged once for the warp - is the pair with
      // more primitives and a lane's ket loop (a load of the ket pair's fields
      // per primitive) is the shorter one; (i | j <= i) the other way round
      int lo = s.x, hi = s.y;
      if (!g.all_pairs && X == Y) {
        if (g.ket_ge[k]) lo = max(lo, i);
        else hi = min(hi, i + 1);
      }
      if (lo >= hi) continue;
      const int keep = count_ge(g.Q, lo, hi, ta);
      const int k64 = count_ge(g.Q, lo, lo + keep, t64);
      // of the k64 quartets above the mixed cutoff, those below the two-float
      // limit (a suffix: Q is descending) go to the two-float list
      const int kd = ffq > 0 ? count_ge(g.Q, lo, lo + k64, fmax(ffq / qi, g.ffw / (qi * w))) : k64;
      // split the bra primitives so that one lane handles at most about
      // lane_prims primitive quartets per task (bounds the launch tail)
      const int first[NTIER] = {lo, lo + k64, lo + kd}, len[NTIER] = {kd, keep - k64, k64 - kd};
#pragma unroll
      for (int t = 0; t < NTIER; ++t) {
        if (len[t] <= 0) continue;
        const int d = X > 2 || Y > 2;
        const int lp = max(1, g.lane_prims[k] / g.fine_div[d][t]);
        const int tk = min(g.task_kets[k], g.fine_kets[d][t]);
        const int nch0 = min(kb, (kb * s.z + lp - 1) / lp);
        const int cs = (kb + nch0 - 1) / nch0;
        const int nch = (kb + cs - 1) / cs;
        if (FILL) {
          for (int ch = 0; ch < nch; ++ch) {
            const int w = (ch * cs) | (min(kb, (ch + 1) * cs) << 16);
            for (int o = 0; o < len[t]; o += tk)
              g.tasks[t][wt[t]++] = make_int4(i, first[t] + o, min(tk, len[t] - o), w);
          }
        } else {
          nt[t] += nch * ((len[t] + tk - 1) / tk);
        }
      }
    }
  }
  if (!FILL) {
#pragma unroll
    for (int t = 0; t < NTIER; ++t) g.count[NTIER * it + t] = nt[t];
  }
}

// Exclusive scans of the NTIER interleaved counts into off (NTIER rows of
// n + 1 entries) in three launches: tile sums, a one-block scan of the tile
// sums, and the tiles' own scans with their offsets.  A tile is 2048 items
// staged in shared memory with coalesced loads; each thread scans 8
// consecutive items.
constexpr int SCAN_THREADS = 256, SCAN_ITEMS = 8, SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

struct Cnt {
  int v[NTIER];
};

// Exclusive block scan of c over the block's 256 threads; totals in tot.
__device__ __forceinline__ void block_exscan(Cnt& c, Cnt& tot) {
  __shared__ Cnt wsum[SCAN_THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  Cnt inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
#pragma unroll
    for (int t = 0; t < NTIER; ++t) {
      const int x = __shfl_up_sync(0xffffffffu, inc.v[t], o);
      if (lane >= o) inc.v[t] += x;
    }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
#pragma unroll
  for (int t = 0; t < NTIER; ++t) {
    int before = 0, all = 0;
    for (int k = 0; k < SCAN_THREADS / 32; ++k) {
      if (k < w) before += wsum[k].v[t];
      all += wsum[k].v[t];
    }
    tot.v[t] = all;
    c.v[t] = before + inc.v[t] - c.v[t];
  }
  __syncthreads();
}

__device__ __forceinline__ void scan_load_tile(int n, const int* __restrict__ count, int tile, int* sm) {
  const int base = tile * SCAN_TILE;
  for (int e = threadIdx.x; e < NTIER * SCAN_TILE; e += SCAN_THREADS) {
    const int i = base + e / NTIER;
    sm[e] = i < n ? count[NTIER * (long)base + e] : 0;
  }
  __syncthreads();
}
__device__ __forceinline__ Cnt scan_thread_sum(const int* sm) {
  Cnt c = {};
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k)
#pragma unroll
    for (int t = 0; t < NTIER; ++t) c.v[t] += sm[NTIER * (threadIdx.x * SCAN_ITEMS + k) + t];
  return c;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(int n, const int* __restrict__ count,
                                                             int* __restrict__ part) {
  __shared__ int sm[NTIER * SCAN_TILE];
  scan_load_tile(n, count, blockIdx.x, sm);
  Cnt c = scan_thread_sum(sm), tot;
  block_exscan(c, tot);
  if (threadIdx.x < NTIER) part[NTIER * blockIdx.x + threadIdx.x] = tot.v[threadIdx.x];
}

// One block: exclusive scan of the tile sums in place, totals into off[t][n].
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_parts(int ntile, int n, int* __restrict__ part,
                                                             int* __restrict__ off) {
  Cnt carry = {};   // over chunks of 256 tiles
  for (int t0 = 0; t0 < ntile; t0 += SCAN_THREADS) {
    const int i = t0 + threadIdx.x;
    Cnt c, tot;
#pragma unroll
    for (int t = 0; t < NTIER; ++t) c.v[t] = i < ntile ? part[NTIER * i + t] : 0;
    block_exscan(c, tot);
#pragma unroll
    for (int t = 0; t < NTIER; ++t) {
      if (i < ntile) part[NTIER * i + t] = carry.v[t] + c.v[t];
      carry.v[t] += tot.v[t];
    }
  }
  if (threadIdx.x == 0)
    for (int t = 0; t < NTIER; ++t) off[(size_t)t * (n + 1) + n] = carry.v[t];
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply(int n, const int* __restrict__ count,
                                                             const int* __restrict__ part, int* __restrict__ off) {
  __shared__ int sm[NTIER * SCAN_TILE];
  scan_load_tile(n, count, blockIdx.x, sm);
  Cnt c = scan_thread_sum(sm), tot;
  block_exscan(c, tot);
  const int i0 = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
#pragma unroll
  for (int t = 0; t < NTIER; ++t) {
    int a = c.v[t] + part[NTIER * blockIdx.x + t];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      if (i0 + k < n) off[(size_t)t * (n + 1) + i0 + k] = a;
      a += sm[NTIER * (threadIdx.x * SCAN_ITEMS + k) + t];
    }
  }
}

// ranges[2 (NTIER k + t)], ..[+1]: first and last task of combo k in list t
__global__ void k_ranges(int ncombo, int n, const int* item_combo_start, const int* off, int* ranges) {
  const int k = threadIdx.x;
  if (k >= ncombo) return;
  for (int t = 0; t < NTIER; ++t) {
    ranges[2 * (NTIER * k + t)] = off[(size_t)t * (n + 1) + item_combo_start[k]];
    ranges[2 * (NTIER * k + t) + 1] = off[(size_t)t * (n + 1) + item_combo_start[k + 1]];
  }
}

// Density maxima.  Per shell block the largest |D| (Ds, rounded up to FP32, for
// the per-quartet screening), per shell its row maximum over the molecule's
// functions; per pair the block maximum (FP32 for the screening) and, for the
// task lists of incremental builds and the gradient, w = max(block, row A, row
// B) and the block maximum, and per ket segment the largest block maximum.
__global__ void k_shell_dmax(int ns, const int* __restrict__ f0, const int* __restrict__ nc,
                             const int* __restrict__ smol, const int* __restrict__ mn,
                             const long long* __restrict__ moff, const int* __restrict__ ms0,
                             const long long* __restrict__ soff, const double* __restrict__ D,
                             double* __restrict__ row, float* __restrict__ Ds) {
  const int s = blockIdx.x;
  if (s >= ns) return;
  const int m = smol[s], n = mn[m], s0 = ms0[m], nsm = ms0[m + 1] - s0;
  const double* Dm = D + moff[m] + (long long)f0[s] * n;
  float* out = Ds + soff[m] + (long long)(s - s0) * nsm;
  double v = 0;
  for (int j = threadIdx.x; j < nsm; j += blockDim.x) {
    const int g = f0[s0 + j], w = nc[s0 + j];
    double x = 0;
    for (int a = 0; a < nc[s]; ++a)
      for (int b = 0; b < w; ++b) x = fmax(x, fabs(Dm[(long long)a * n + g + b]));
    out[j] = __double2float_ru(x);
    v = fmax(v, x);
  }
  __shared__ double sh[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = fmax(v, sh[w]);
    row[s] = v;
  }
}

// A quartet (AB|CD) feeds J_AB (dD_CD), J_CD (dD_AB) and K_AC, K_AD, K_BC, K_BD
// (dD_BD, dD_BC, dD_AD, dD_AC); every exchange block holds a bra shell, so
// max(pw[bra], pb[ket]) bounds all six density factors.
// One launch also makes the kernels' copies of the density, where asked for:
// FP32 (d32) and two-float (dff), the latter scaled by 2^-e with e the exponent
// of max |D| (clamped to +-400; 0 when the maximum is 0 or not finite), so that
// any density an FP64 build takes stays inside the FP32 exponent range; and it
// zeroes the work-queue heads and the two-float accumulator (gff, where asked for).
struct PrepArgs {
  int np, ns;
  const int *pA, *pB, *pmol, *f0, *nc, *mn;
  const long long* moff;
  const double* D;
  const double* row;
  double *pw, *pb;
  float* pbf;
  size_t nn;
  float* d32;
  ff* dff;
  int* dexp;
  double* gff;
  int* counters;
  int ncounters;
};
__global__ void __launch_bounds__(128) k_density_prep(PrepArgs a) {
  const size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  if (i0 < (size_t)a.ncounters) a.counters[i0] = 0;
  for (size_t p = i0; p < (size_t)a.np; p += step) {
    const int A = a.pA[p], B = a.pB[p], m = a.pmol[p], n = a.mn[m];
    const double* Dm = a.D + a.moff[m];
    double b = 0;
    for (int x = 0; x < a.nc[A]; ++x)
      for (int y = 0; y < a.nc[B]; ++y) b = fmax(b, fabs(Dm[(long)(a.f0[A] + x) * n + a.f0[B] + y]));
    a.pw[p] = fmax(b, fmax(a.row[A], a.row[B]));
    a.pb[p] = b;
    a.pbf[p] = __double2float_ru(b);
  }
  if (a.d32)
    for (size_t i = i0; i < a.nn; i += step) a.d32[i] = (float)a.D[i];
  if (!a.dff) return;
  double mx = 0;
  for (int s = threadIdx.x; s < a.ns; s += blockDim.x) mx = fmax(mx, a.row[s]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  __shared__ double sh[4];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = fmax(fmax(sh[0], sh[1]), fmax(sh[2], sh[3]));
  const int e = mx > 0 && mx <= 1.7976931348623157e308 ? min(400, max(-400, ilogb(mx))) : 0;
  const double sc = scalbn(1.0, -e);
  if (i0 == 0) *a.dexp = e;
  for (size_t i = i0; i < a.nn; i += step) {
    const double v = a.D[i] * sc;
    const float h = (float)v;
    a.dff[i] = ff(h, (float)(v - (double)h));
    if (a.gff) a.gff[i] = 0.0;
  }
}

__global__ void k_seg_max(int nseg, const int4* __restrict__ seg, const double* __restrict__ pw, double* __restrict__ sw) {
  const int s = blockIdx.x;
  if (s >= nseg) return;
  const int4 g = seg[s];
  double m = 0;
  for (int p = g.x + threadIdx.x; p < g.y; p += blockDim.x) m = fmax(m, pw[p]);
  __shared__ double sh[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, sh[w]);
    sw[s] = m;
  }
}

__global__ void k_to_float(size_t n, const double* __restrict__ x, float* __restrict__ y) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = (float)x[i];
}
static gbhf_status to_float(gbhf_ctx* c, size_t n, const double* d_x, float* d_y) {
  const int blocks = (int)std::min<size_t>((n + 255) / 256, (size_t)c->nsm * 4);
  k_to_float<<<std::max(blocks, 1), 256, 0, c->stream>>>(n, d_x, d_y);
  count_launch(c);
  GBHF_CUDA(c, cudaGetLastError());
  return GBHF_OK;
}

// Everything the kernels of the next build need of its density d_dD: maxima for
// the screening (c->tasks.Ds, pbf), FP32 and two-float copies, zeroed work-queue
// heads of st (ncounters), a zeroed c->gff (`fock`) and, with `segments`, the segment
// maxima of the weighted task lists.
static gbhf_status density_prep(gbhf_ctx* c, TaskLists& st, const double* d_dD, int precision, int ncounters,
                                bool segments, bool fock) {
  PairData& P = c->pairs;
  TaskLists& sh = c->tasks;   // per-shell and per-molecule arrays
  const int ns = (int)c->basis.shells.size();
  const size_t nst = (size_t)c->basis.stacked;   // all molecules' blocks
  GBHF_CUDA(c, st.row.alloc(ns));
  GBHF_CUDA(c, st.pw.alloc(std::max(P.npairs, 1)));
  GBHF_CUDA(c, st.pb.alloc(std::max(P.npairs, 1)));
  GBHF_CUDA(c, st.sw.alloc(std::max(P.nseg_total, 1)));
  GBHF_CUDA(c, st.counters.alloc(ncounters));
  GBHF_CUDA(c, sh.pbf.alloc(std::max(P.npairs, 1)));
  GBHF_CUDA(c, sh.Ds.alloc(std::max<size_t>(sh.ds_size, 1)));
  if (precision != GBHF_PREC_FP64) GBHF_CUDA(c, c->dfloat.alloc(nst));
  if (P.use_ff) {
    static_assert(sizeof(ff) == sizeof(double), "one block for both");
    GBHF_CUDA(c, c->dff.alloc(2 * nst));
    GBHF_CUDA(c, c->dff_exp.alloc(1));
    c->gff.p = reinterpret_cast<double*>(c->dff.p + nst);
  }
  k_shell_dmax<<<ns, 128, 0, c->stream>>>(ns, sh.f0.p, sh.nc.p, sh.smol.p, sh.mn.p, sh.moff.p, sh.ms0.p, sh.soff.p, d_dD,
                                          st.row.p, sh.Ds.p);
  const PrepArgs a{P.npairs,   ns,          P.A.p, P.B.p,  P.mol.p, sh.f0.p, sh.nc.p, sh.mn.p, sh.moff.p, d_dD, st.row.p,
                   st.pw.p,    st.pb.p,     sh.pbf.p, nst, precision != GBHF_PREC_FP64 ? c->dfloat.p : nullptr,
                   P.use_ff ? c->dff.p : nullptr, c->dff_exp.p, P.use_ff && fock ? c->gff.p : nullptr, st.counters.p, ncounters};
  const int blocks = (int)std::min<size_t>((std::max<size_t>(P.npairs, nst) + 127) / 128, (size_t)c->nsm * 8);
  k_density_prep<<<std::max(blocks, 1), 128, 0, c->stream>>>(a);
  if (segments && P.nseg_total > 0) {
    k_seg_max<<<P.nseg_total, 256, 0, c->stream>>>(P.nseg_total, P.seg_info.p, st.pb.p, st.sw.p);
    count_launch(c);
  }
  count_launch(c, 2);
  GBHF_CUDA(c, cudaGetLastError());
  sh.screened = true;
  return GBHF_OK;
}

// Quartet-class task lists of TL for the combos (cbra[k], cket[k]).
static gbhf_status build_task_lists(gbhf_ctx* c, TaskLists& TL, int ncombo, const int* cbra, const int* cket,
                                    const int* lane_prims, const int* task_kets, bool all_pairs, bool square_w,
                                    double thr_all, double thr64, double ffw, const double* pw,
                                    const double* sw) {
  PairData& P = c->pairs;
  int* h_ranges = TL.hranges;
  std::vector<int> ics(ncombo + 1, 0);
  for (int k = 0; k < ncombo; ++k) {
    const int X = cbra[k];
    ics[k + 1] = ics[k] + (P.cls_start[X + 1] - P.cls_start[X]);
  }
  TL.nitems = ics[ncombo];
  TL.combo_item_start = ics;
  TL.ncombo = ncombo;
  const int ni = TL.nitems;
  DBuf<int>& d_ics = TL.ics_d;
  DBuf<int>& d_cls = TL.cls_d;
  DBuf<int>& d_scs = TL.scs_d;
  GBHF_CUDA(c, d_ics.alloc(ncombo + 1));
  GBHF_CUDA(c, d_cls.alloc(NPCLS + 1));
  GBHF_CUDA(c, d_scs.alloc(NPCLS + 1));
  GBHF_CUDA(c, cudaMemcpyAsync(d_ics.p, ics.data(), (ncombo + 1) * sizeof(int), cudaMemcpyHostToDevice, c->stream));
  GBHF_CUDA(c, cudaMemcpyAsync(d_cls.p, P.cls_start, (NPCLS + 1) * sizeof(int), cudaMemcpyHostToDevice, c->stream));
  GBHF_CUDA(c, cudaMemcpyAsync(d_scs.p, P.seg_cls_start, (NPCLS + 1) * sizeof(int), cudaMemcpyHostToDevice, c->stream));
  GBHF_CUDA(c, TL.item_count.alloc(NTIER * (size_t)std::max(ni, 1)));
  GBHF_CUDA(c, TL.item_off.alloc(NTIER * ((size_t)ni + 1)));
  GBHF_CUDA(c, TL.ranges.alloc(2 * NTIER * ncombo));
  GBHF_CUDA(c, TL.stats.alloc(3 * NTIER * ncombo));
  // 32-ket groups that a task of the s/p J/K kernels scans: the queue of survivors
  // then fills whole batches, and the bra is staged once for all of them, while
  // there are tasks enough for every warp ((H2O)64 mixed build in order: 65.9 ms
  // at 1, 57.3 at 4, 56.2 at 8, 55.8 at 16; (H2O)16 mixed SCF 40.4, 39.3, 39.6, 40.3).
  // Below that a task of several groups is a longer serial chain.  FP64 Fock builds at 1
  // and 4: (H2O)2/STO-3G 0.168 and 0.195 ms, (H2O)8/6-31G 1.40 and 1.55, 10 waters 1.76
  // and 1.90, 12 2.59 and 2.55, 16 6.31 and 5.68; gradients: (H2O)4/STO-3G 0.92 and
  // 1.18, (H2O)8/6-31G 6.11 and 6.06.
  const int scan = P.npairs >= 65536 ? 8 : P.npairs >= (all_pairs ? 2048 : 4096) ? 4 : 1;
  TaskGenArgs g;
  g.nitems = ni;
  g.ncombo = ncombo;
  for (int k = 0; k < NCOMBO_MAX; ++k) {
    g.cbra[k] = k < ncombo ? cbra[k] : 0;
    g.cket[k] = k < ncombo ? cket[k] : 0;
    g.lane_prims[k] = k < ncombo ? std::max(1, lane_prims[k]) : 1;
    g.task_kets[k] = k < ncombo ? std::min(32, std::max(1, task_kets[k])) : 32;
    // (the s/p kernels only)
    if (k < (all_pairs ? NGCOMBO_SP : NCOMBO_SP) && g.task_kets[k] == 32) g.task_kets[k] *= scan;
    // the (ss|ss) and (ps|ps) quartets with the bra of more primitives: the
    // FP32 launches gain 13-14% (fewer ket-field loads per primitive
    // quartet); (pp|pp) FP64 lost 18% that way (its launch is tail-bound)
    g.ket_ge[k] = k < ncombo && cbra[k] == cket[k] && cbra[k] <= 1 ? 1 : 0;
  }
  // Finer tasks where a list is too short to keep the SMs busy to its end.
  // - d classes (a warp per quartet), below 4096 shell pairs: twelfths.  6-31G*
  //   gradient of 1, 2, 3 (mixed), 5 waters 11.4, 15.3, 10.4, 23.7 -> 6.9, 9.3, 6.9,
  //   18.6 ms, Fock build 1.46, 1.96, 1.40, 3.46 -> 0.90, 1.42, 1.09, 3.32.  With
  //   5050 pairs (10 waters) the gradient lost 2%.
  // - FP64 gradient tasks of s/p classes, quarters: the two-float list leaves few of
  //   them, and one ran for a third of the launch.  (H2O)8 7.88 -> 7.47 ms.
  // - two-float gradient tasks, at most 64 kets ((H2O)8 7.47 -> 7.10 ms, (H2O)12 mixed
  //   7.35 -> 6.66), below 4096 pairs halves ((H2O)4 2.75 -> 2.56).
  // The s/p Fock builds gain nothing of the kind ((H2O)16 FP64 6.7 -> 7.4 ms with
  // halved two-float tasks).
  const bool few = P.npairs < 4096;
  for (int t = 0; t < NTIER; ++t) {
    g.fine_div[0][t] = !all_pairs ? 1 : (t == TIER_64 ? 4 : (t == TIER_FF && few ? 2 : 1));
    g.fine_kets[0][t] = all_pairs && t == TIER_FF ? 64 : 1 << 20;
    g.fine_div[1][t] = few ? 12 : 1;
    g.fine_kets[1][t] = 1 << 20;
  }
  g.all_pairs = all_pairs ? 1 : 0;
  g.square_w = square_w ? 1 : 0;
  g.item_combo_start = d_ics.p;
  g.cls_start = d_cls.p;
  g.seg_cls_start = d_scs.p;
  g.seg = P.seg_info.p;
  g.Q = P.Q.p;
  g.pK = P.K.p;
  g.nmol = c->basis.nmol;
  g.pmol = P.mol.p;
  g.mseg = P.mseg.p;
  g.mact = c->mol_active;
  g.thr_all = thr_all;
  g.thr64 = thr64;
  g.ffq = P.ffq.p;
  g.ffw = ffw;
  g.pw = pw;
  g.sw = sw;
  g.count = TL.item_count.p;
  g.off = TL.item_off.p;
  for (int t = 0; t < NTIER; ++t) g.tasks[t] = nullptr;
  if (ni > 0) {
    k_tasks<false><<<(ni + 127) / 128, 128, 0, c->stream>>>(g);
    count_launch(c);
  }
  {
    const int ntile = std::max(1, (ni + SCAN_TILE - 1) / SCAN_TILE);
    GBHF_CUDA(c, TL.scan_part.alloc(NTIER * (size_t)ntile));
    k_scan_tiles<<<ntile, SCAN_THREADS, 0, c->stream>>>(ni, TL.item_count.p, TL.scan_part.p);
    k_scan_parts<<<1, SCAN_THREADS, 0, c->stream>>>(ntile, ni, TL.scan_part.p, TL.item_off.p);
    k_scan_apply<<<ntile, SCAN_THREADS, 0, c->stream>>>(ni, TL.item_count.p, TL.scan_part.p, TL.item_off.p);
    count_launch(c, 3);
  }
  // the per-class ranges follow from the offsets alone: one copy and one
  // synchronisation give the host both the ranges and the list sizes
  k_ranges<<<1, 64, 0, c->stream>>>(ncombo, ni, d_ics.p, TL.item_off.p, TL.ranges.p);
  count_launch(c);
  GBHF_CUDA(c, cudaGetLastError());
  GBHF_CUDA(c, cudaMemcpyAsync(h_ranges, TL.ranges.p, 2 * NTIER * ncombo * sizeof(int), cudaMemcpyDeviceToHost,
                               c->stream));
  GBHF_CUDA(c, cudaStreamSynchronize(c->stream));
  for (int t = 0; t < NTIER; ++t) {
    const int tot = ncombo > 0 ? h_ranges[2 * (NTIER * (ncombo - 1) + t) + 1] : 0;
    GBHF_CUDA(c, TL.tasks[t].alloc(std::max(tot, 1)));
    g.tasks[t] = TL.tasks[t].p;
  }
  if (ni > 0) {
    k_tasks<true><<<(ni + 127) / 128, 128, 0, c->stream>>>(g);
    count_launch(c);
  }
  GBHF_CUDA(c, cudaGetLastError());
  return GBHF_OK;
}

// d combos evaluated by the generated lane-per-ket code (few components per
// quartet); the others go to the warp-per-quartet kernels of jkd.cu.
static bool gen_dclass(int k) { return (k >= 6 && k <= 11) || k == 15; }

// Default task budgets.  J/K (which 0): lane_prims bounds the primitive
// quartets one lane evaluates in one task, per class (ss|ss) (ps|ss) (ps|ps)
// (pp|ss) (pp|ps) (pp|pp) ...: about the same arithmetic per task, so that the
// longest task - the tail of a persistent launch - stays short ((ss|ss) and
// (ps|ss) take less than that: their launches are short, so the tail is a
// larger share of them, while more tasks cost the overlapped SCF next to
// nothing - 0.1 ms of 48 on (H2O)16/6-31G).  A task never
// splits the ket primitives, so a lane always evaluates at least K_ket of them.
// For the warp-per-quartet d classes it bounds the primitive quartets of one
// quartet in one task, and such a task holds one quartet (a launch then spreads
// its quartets over every resident warp).  Gradient (which 1): the derivative
// code does about twice the ERI work per primitive quartet.
void default_budgets(gbhf_ctx* c, int which) {
  static const int jk_lp[NCOMBO] = {96, 64, 48, 96, 32, 8, 48, 16, 8, 8, 16, 8, 36, 36, 36, 16, 36, 36,
                                    36, 36, 36};
  static const int jk_tk[NCOMBO] = {32, 32, 32, 32, 32, 32, 32, 32, 32, 32, 32, 32, 1, 1, 1, 32, 1, 1, 1, 1, 1};
  static const int gr_lp_sp[NGCOMBO_SP] = {128, 64, 24, 64, 24, 8, 24, 8, 4};
  for (int k = 0; k < NCOMBO_MAX; ++k) {
    if (which == 0) {
      c->jk_lp[k] = k < NCOMBO ? jk_lp[k] : 1;
      c->jk_tk[k] = k < NCOMBO ? jk_tk[k] : 32;
    } else {
      c->gr_lp[k] = k < NGCOMBO_SP ? gr_lp_sp[k] : (grad_gen_combo(k) ? 8 : 36);
      c->gr_tk[k] = grad_gen_combo(k) ? 32 : 1;
    }
  }
}

// Kets per task: 32 (a lane per ket) for the lane-per-ket classes, else free.
bool lane_per_ket(int which, int k) {
  return which == 0 ? (k < NCOMBO_SP || gen_dclass(k)) : grad_gen_combo(k);
}

// Weighted bound below which a quartet of a mixed-precision build runs in two
// floats (error 2^-45 of its value) instead of FP64: 2^18 times the mixed cutoff,
// at which that error is an eighth of what FP32 leaves on a quartet at the cutoff.
// Without a mixed cutoff only P.ffq decides (ff_limits in setup.cu).
static double ff_weighted_limit(int precision, double thr64) {
  return precision == GBHF_PREC_FP64 ? 0.0 : 262144.0 * thr64;
}

// J/K lists: the classes with bra class >= ket class, unique quartets, with
// the context's task budgets.
static gbhf_status build_tasks(gbhf_ctx* c, int precision, double thr_all, double thr64, const double* pw = nullptr,
                               const double* sw = nullptr) {
  return build_task_lists(c, c->tasks, NCOMBO, COMBO_BRA, COMBO_KET, c->jk_lp, c->jk_tk, false, false, thr_all,
                          thr64, ff_weighted_limit(precision, thr64), pw, sw);
}

gbhf_status ensure_shell_arrays(gbhf_ctx* c) {
  TaskLists& st = c->tasks;
  if (st.f0_gen == c->basis_gen) return GBHF_OK;
  const Basis& b = c->basis;
  const size_t ns = b.shells.size();
  std::vector<int> f0(ns), nc(ns), at(ns), sm(ns);
  std::vector<double> sc(6 * std::max<size_t>(ns, 1), 1.0);
  for (size_t s = 0; s < ns; ++s) {
    f0[s] = b.shells[s].f0 - b.mol_fn_off[b.shells[s].mol];   // first function within its molecule
    nc[s] = b.shells[s].ncomp;
    at[s] = b.shells[s].atom;
    sm[s] = b.shells[s].mol;
    for (int k = 0; k < 6; ++k) sc[6 * s + k] = b.shells[s].scale[k];
  }
  // centres in three FP32 parts (float4 each): every bit of the coordinates
  std::vector<float> cen(12 * std::max<size_t>(ns, 1), 0.0f);
  for (size_t s = 0; s < ns; ++s)
    for (int x = 0; x < 3; ++x) {
      double r = b.xyz[3 * b.shells[s].atom + x];
      for (int k = 0; k < 3; ++k) {
        cen[12 * s + 4 * k + x] = (float)r;
        r -= (double)cen[12 * s + 4 * k + x];
      }
    }
  std::vector<int> mn(b.nmol), fmol(b.nbf), amol(b.natoms);
  for (int m = 0; m < b.nmol; ++m) {
    mn[m] = b.mol_fn_off[m + 1] - b.mol_fn_off[m];
    for (int i = b.mol_fn_off[m]; i < b.mol_fn_off[m + 1]; ++i) fmol[i] = m;
    for (int a = b.mol_atom_off[m]; a < b.mol_atom_off[m + 1]; ++a) amol[a] = m;
  }
  // shells of each molecule (contiguous: shells follow the functions)
  std::vector<int> ms0(b.nmol + 1, (int)ns);
  std::vector<long long> soff(b.nmol + 1, 0);
  for (size_t s = ns; s-- > 0;) ms0[sm[s]] = (int)s;
  for (int m = 0; m < b.nmol; ++m) soff[m + 1] = soff[m] + (long long)(ms0[m + 1] - ms0[m]) * (ms0[m + 1] - ms0[m]);
  st.ds_size = (size_t)soff[b.nmol];
  // all of them in one block and one copy (a new context's first build spends some 5 us on
  // every allocation and copy; water/STO-3G Fock 0.73 -> 0.71 ms with its set_basis)
  std::vector<unsigned char> host;
  std::vector<std::function<void()>> place;
  auto add = [&](auto& view, const auto& v) {
    place.push_back([&view, &st, off = host.size()] {
      view.p = reinterpret_cast<decltype(view.p)>(st.shell_block.p + off);
    });
    const unsigned char* p = reinterpret_cast<const unsigned char*>(v.data());
    host.insert(host.end(), p, p + v.size() * sizeof(v[0]));
    host.resize((host.size() + 15) / 16 * 16);
  };
  add(st.f0, f0);
  add(st.sscale, sc);
  add(st.ms0, ms0);
  add(st.soff, soff);
  add(st.cen, cen);
  add(st.nc, nc);
  add(st.atom, at);
  add(st.smol, sm);
  add(st.mn, mn);
  add(st.moff, b.mol_moff);
  add(st.fmol, fmol);
  add(st.amol, amol);
  add(st.mfo, b.mol_fn_off);
  add(st.mao, b.mol_atom_off);
  GBHF_CUDA(c, st.shell_block.alloc(host.size()));
  for (auto& p : place) p();
  GBHF_CUDA(c, cudaMemcpyAsync(st.shell_block.p, host.data(), host.size(), cudaMemcpyHostToDevice, c->stream));
  GBHF_CUDA(c, cudaStreamSynchronize(c->stream));
  st.f0_gen = c->basis_gen;
  return GBHF_OK;
}

// Gradient lists: every (bra class, ket class) combination, every ordered pair
// of shell pairs, bound Q_bra Q_ket max(w_bra, w_ket)^2 with the pair weights
// of D (|Gamma_abcd| <= that squared weight).
gbhf_status build_grad_tasks(gbhf_ctx* c, const double* d_D, double cutoff, double mixed_cutoff, int precision) {
  GBHF_TRY(ensure_pairs(c));
  GBHF_TRY(ensure_shell_arrays(c));
  TaskLists& gt = c->gtasks;
  GBHF_TRY(density_prep(c, gt, d_D, precision, NTIER * NCOMBO_MAX, true, false));
  // FP32 up to the cutoff, but never above a bound of 1/8: two floats take the
  // rest of what a larger cutoff gives to FP32
  const double t64 = precision == GBHF_PREC_FP64 ? 0.0 : std::min(mixed_cutoff, 0.125);
  GBHF_TRY(build_task_lists(c, gt, NCOMBO_MAX, GRAD_COMBO_BRA, GRAD_COMBO_KET, c->gr_lp, c->gr_tk, true, true,
                            cutoff, t64, ff_weighted_limit(precision, t64), gt.pw.p, gt.sw.p));
  return GBHF_OK;
}

gbhf_status jk_build(gbhf_ctx* c, const double* d_Dsq, double* d_G, int precision, double schwarz,
                     double mixed_cutoff, double weight, bool local_weights, bool with_j, const double** d_Gff) {
  const int wj = with_j ? 1 : 0;
  c->tasks.thr_exact = schwarz;   // per-quartet test in the kernels, on the density passed here
  GBHF_TRY(ensure_pairs(c));
  const PairData& P = c->pairs;
  TaskLists& st = c->tasks;
  GBHF_TRY(ensure_shell_arrays(c));
  if (local_weights || P.nprim_pairs >= SMALL_PRIM_PAIRS) {
    GBHF_TRY(density_prep(c, st, d_Dsq, precision, NTIER * NCOMBO, local_weights, true));
  } else {
    st.screened = false;
    GBHF_CUDA(c, st.counters.alloc(NTIER * NCOMBO));
    GBHF_CUDA(c, cudaMemsetAsync(st.counters.p, 0, NTIER * NCOMBO * sizeof(int), c->stream));
    if (precision != GBHF_PREC_FP64) {
      GBHF_CUDA(c, c->dfloat.alloc((size_t)c->basis.stacked));
      GBHF_TRY(to_float(c, (size_t)c->basis.stacked, d_Dsq, c->dfloat.p));
    }
  }
  if (local_weights) {
    // incremental build: bounds weighted by the local size of the density change
    const double t64 = precision == GBHF_PREC_FP64 ? 0.0 : mixed_cutoff;
    GBHF_TRY(build_tasks(c, precision, schwarz, t64, st.pw.p, st.sw.p));
    st.thr_all = -1;   // lists no longer match a uniform weight
    st.thr64 = -1;
  } else {
    if (!(weight > 0)) weight = 1e-300;
    const double thr_all = schwarz / weight;
    const double thr64 = precision == GBHF_PREC_FP64 ? 0.0 : mixed_cutoff / weight;
    if (thr_all != st.thr_all || thr64 != st.thr64 || !c->tasks.tasks[0].p) {
      GBHF_TRY(build_tasks(c, precision, thr_all, thr64));
      st.thr_all = thr_all;
      st.thr64 = thr64;
    }
  }
  if (!st.stats_pending) {   // the counters add up over builds until flush_jk_stats reads them
    GBHF_CUDA(c, cudaMemsetAsync(c->tasks.stats.p, 0, 3 * NTIER * NCOMBO * sizeof(unsigned long long), c->stream));
    st.stats_pending = true;
  }
  int nt[NCOMBO][NTIER];
  long total = 0;
  for (int k = 0; k < NCOMBO; ++k)
    for (int t = 0; t < NTIER; ++t) {
      nt[k][t] = st.hranges[2 * (NTIER * k + t) + 1] - st.hranges[2 * (NTIER * k + t)];
      total += nt[k][t];
    }
  const bool ev = c->prof.events;
  // FP64 lists, then two-float, then FP32, each heaviest class first.  Without
  // per-class profiling events the launches go round-robin to the side streams:
  // each is a persistent grid that fills the GPU, and the next one takes over SMs
  // as the tail of the previous one drains.  With profiling events they run in
  // order on the context stream so that each launch is timed alone.
  static const int order[NCOMBO] = {20, 19, 18, 17, 16, 15, 14, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2, 1, 0};
  static const int tiers[NTIER] = {TIER_64, TIER_FF, TIER_32};
  // with a million tasks the launches are long against their tails, and classes
  // that share an SM only push each other's Boys rows out of L1: one stream
  // ((H2O)64 mixed, 3.1 million tasks: 56.2 ms in order, 61.8 on eight streams;
  // (H2O)16, 170 thousand: 42.7 against 39.4 ms per SCF)
  const int nside = total >= (1l << 20) ? 1 : gbhf_ctx::NSIDE;
  // The two-float launches add into an accumulator of their own.  Theirs are many small
  // terms, and into the common one, near its final size once the FP64 launches are
  // through, each was rounded at that size: the FP64 Fock matrix of (H2O)8/6-31G was
  // 1.0e-14 rms from its exact value ((H2O)16 1.8e-14), against 7.8e-15 (1.2e-14) by
  // FP64 arithmetic alone and 2.8e-15 (3.8e-15) now.
  bool two_float = false;
  int ne = 0, nl = 0;
  int ev_combo[NTIER * NCOMBO], ev_prec[NTIER * NCOMBO];
  SideFork side(c->stream, c->fork_ev, c->side, c->join_ev, gbhf_ctx::NSIDE);
  if (ev) GBHF_CUDA(c, cudaEventRecord(c->evc[ne], c->stream));
  else GBHF_CUDA(c, side.fork());
  for (const int tier : tiers) {
    for (int oi = 0; oi < NCOMBO; ++oi) {
      const int k = order[oi];
      if (nt[k][tier] <= 0) continue;
      cudaStream_t strm = ev ? c->stream : c->side[nl % nside];
      ++nl;
      double* G = tier == TIER_FF ? c->gff.p : d_G;
      two_float |= tier == TIER_FF;
      if (k >= NCOMBO_SP && !gen_dclass(k)) GBHF_TRY(launch_jk_dclass(c, strm, k, tier, d_Dsq, G, nt[k][tier], wj));
      else if (tier == TIER_64) GBHF_TRY(launch_combo<double>(c, strm, k, tier, d_Dsq, G, nt[k][tier], wj));
      else if (tier == TIER_32) GBHF_TRY(launch_combo<float>(c, strm, k, tier, c->dfloat.p, G, nt[k][tier], wj));
      else GBHF_TRY(launch_jk_ff(c, strm, k, G, nt[k][tier], wj));
      if (ev) {
        ev_combo[ne] = k;
        ev_prec[ne] = tier == TIER_32 ? 1 : 0;   // two-float work counts as FP64 in the profile
        ++ne;
        GBHF_CUDA(c, cudaEventRecord(c->evc[ne], c->stream));
      }
    }
  }
  if (!ev) GBHF_CUDA(c, side.join());
  if (d_Gff) *d_Gff = two_float ? c->gff.p : nullptr;
  else if (two_float) GBHF_TRY(axpby(c, (size_t)c->basis.stacked, 1.0, d_G, 1.0, c->gff.p, d_G));
  // statistics: read with the per-class event times when those are taken,
  // else when the profile is read (no host synchronisation per build)
  if (!ev) return GBHF_OK;
  GBHF_TRY(flush_jk_stats(c));
  for (int e = 0; e < ne; ++e) {
    float ms = 0;
    GBHF_CUDA(c, cudaEventElapsedTime(&ms, c->evc[e], c->evc[e + 1]));
    c->prof.cls[ev_combo[e]][ev_prec[e]][3] += ms;
    (ev_prec[e] == 0 ? c->prof.jk_ms64 : c->prof.jk_ms32) += ms;
  }
  return GBHF_OK;
}

gbhf_status flush_jk_stats(gbhf_ctx* c) {
  TaskLists& st = c->tasks;
  if (!st.stats_pending) return GBHF_OK;
  unsigned long long hs[3 * NTIER * NCOMBO];
  GBHF_CUDA(c, cudaMemcpyAsync(hs, st.stats.p, sizeof(hs), cudaMemcpyDeviceToHost, c->stream));
  GBHF_CUDA(c, cudaStreamSynchronize(c->stream));
  st.stats_pending = false;
  for (int k = 0; k < NCOMBO; ++k)
    for (int t = 0; t < NTIER; ++t) {
      const int p = t == TIER_32 ? 1 : 0;   // two-float work counts as FP64 in the profile
      const unsigned long long* s = hs + 3 * (NTIER * k + t);
      c->prof.shellq += (double)s[0];
      c->prof.fnq += (double)s[1];
      (p == 0 ? c->prof.prim64 : c->prof.prim32) += (double)s[2];
      c->prof.cls[k][p][0] += (double)s[0];
      c->prof.cls[k][p][1] += (double)s[1];
      c->prof.cls[k][p][2] += (double)s[2];
    }
  return GBHF_OK;
}

}  // namespace gbhf
