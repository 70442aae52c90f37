// Symmetric eigen-solve by Householder tridiagonalisation, bisection and
// inverse iteration: eigenSolve (NumericalTools/EigenValues.hs:29-31; the
// reference calls LAPACK's dsyev family through hmatrix eigSH'), ascending
// eigenvalues with the eigenvectors as columns (sortEigenData,
// NumericalTools/VectorTools.hs:27-31).
//
// 1. k_sytrd_cluster: a thread-block cluster of 8 or 16 CTAs reduces A to
//    tridiagonal T = Q^T A Q with the rows of A spread over the CTAs' shared
//    memory (k_sytrd: the packed triangle in one CTA, for the smallest n and where
//    clusters are not available), n - 2 Householder reflectors H_k = I - tau_k v_k v_k^T
//    (v_k[k+1] = 1); n <= TRIDIAG_WIDE_MAX_N.
// 2. k_tri_prep: split T into unreduced blocks at negligible off-diagonals.
// 3. k_tri_vec: one warp per eigenvalue: 32-point multisection with Sturm
//    counts on its block, then inverse iteration (LU with partial pivoting of
//    T - lambda I in shared memory) from a fixed pseudo-random start.
// 4. k_tri_fix: eigenvalues closer than 1e-11 ||T|| within a block get their
//    vectors again by inverse iteration orthogonalised against the earlier
//    ones at every step; global ascending rank of every eigenvalue.
// 5. Two Newton-Schulz steps Z <- Z (3 I - Z^T Z) / 2 on the DMMA GEMM make
//    the vectors orthonormal to rounding (inverse-iteration vectors of close
//    eigenvalues are orthogonal only to eps ||T|| / gap).
// 6. k_tri_back: one warp per vector applies H_0 ... H_(n-3) and writes the
//    vector into the column of its rank.
#include <algorithm>
#include <cfloat>

#include <cooperative_groups.h>

#include "dense.cuh"
#include "gbhf_internal.h"

namespace gbhf {

namespace {

constexpr double kEps = DBL_EPSILON;

__host__ __device__ __forceinline__ long pidx(int i, int j) { return (long)i * (i + 1) / 2 + j; }   // j <= i

// The solver squares matrix elements (reflector norms) and vectors of size
// 1 / (eps ||T||) (inverse iteration), which leaves the FP64 range for elements
// below about 2^-460 or above 2^510.  A matrix whose largest element lies outside
// 2^-400 .. 2^400 is therefore reduced after scaling by 2^-x, x the exponent of
// that element (exact; scal[3] = x, and k_tri_fix scales the eigenvalues back).
__device__ __forceinline__ int scale_exponent(double amax) {
  if (!(amax > 0.0 && amax <= DBL_MAX)) return 0;
  const int x = ilogb(amax);
  return x < -400 || x > 400 ? x : 0;
}
// What decides whether the largest element is looked for at all: bit 0 an element of at
// least 2^-400, bit 1 one above 2^400 (no reduction of values in the common case, 5 us
// of a 7 x 7 solve).
__device__ __forceinline__ int range_bits(double a) {
  return (fabs(a) >= 0x1p-400 ? 1 : 0) | (fabs(a) > 0x1p400 ? 2 : 0);
}

// One CTA of 1024 threads.  Shared memory: packed lower triangle of A
// (n(n+1)/2), v (n), p / w (n).  Outputs: d (n), e (n - 1), tau (n), Vt (row k:
// reflector k, zero up to column k, 1 at column k + 1; rows 0 .. n - 3), scal[3].
__global__ void __launch_bounds__(1024) k_sytrd(int n, const double* __restrict__ A, double* __restrict__ d,
                                                double* __restrict__ e, double* __restrict__ tau,
                                                double* __restrict__ Vt, double* __restrict__ scal) {
  extern __shared__ double sm[];
  double* P = sm;
  double* sv = P + pidx(n, 0);   // n(n+1)/2 doubles before it
  double* sp = sv + n;
  __shared__ double s_bc[4];
  const int tid = threadIdx.x, nt = blockDim.x;
  int bits = 0;
  for (long q = tid; q < (long)n * n; q += nt) {
    const int i = (int)(q / n), j = (int)(q % n);
    if (j <= i) {
      P[pidx(i, j)] = A[q];
      bits |= range_bits(A[q]);
    }
  }
  const bool some = __syncthreads_or(bits & 1), large = __syncthreads_or(bits & 2);
  int sx = 0;
  if (!some || large) {
    double amax = 0.0;
    for (int q = tid; q < (int)pidx(n, 0); q += nt) amax = fmax(amax, fabs(P[q]));
    amax = block_reduce(amax, true);
    if (tid == 0) s_bc[0] = amax;
    __syncthreads();
    sx = scale_exponent(s_bc[0]);
    for (int q = tid; q < (int)pidx(n, 0); q += nt) P[q] = scalbn(P[q], -sx);
    __syncthreads();
  }
  if (tid == 0) scal[3] = sx;
  for (int k = 0; k + 2 < n; ++k) {
    const int m = n - 1 - k;   // trailing size, >= 2
    // Householder vector of column k below the diagonal
    double s = 0.0;
    for (int i = k + 2 + tid; i < n; i += nt) {
      const double x = P[pidx(i, k)];
      s += x * x;
    }
    s = block_reduce(s, false);
    if (tid == 0) {
      const double alpha = P[pidx(k + 1, k)];
      double beta = alpha, t = 0.0, scale = 0.0;
      if (s > 0.0) {
        beta = -copysign(sqrt(alpha * alpha + s), alpha);
        t = (beta - alpha) / beta;
        scale = 1.0 / (alpha - beta);
      }
      d[k] = P[pidx(k, k)];
      e[k] = beta;
      tau[k] = t;
      s_bc[0] = t;
      s_bc[1] = scale;
    }
    __syncthreads();
    const double t = s_bc[0], scale = s_bc[1];
    for (int i = tid; i < n; i += nt) {
      double v = 0.0;
      if (i == k + 1) v = 1.0;
      else if (i > k + 1) v = P[pidx(i, k)] * scale;
      sv[i] = v;
      Vt[(long)k * n + i] = v;
    }
    __syncthreads();
    if (t == 0.0) continue;   // uniform: s_bc is shared
    // p = t A22 v, G threads per row (G a power of two, G * m <= 1024)
    int G = 32;
    while (G > 1 && G * m > nt) G >>= 1;
    {
      const int row = k + 1 + tid / G, g = tid % G;
      double acc = 0.0;
      if (row < n) {
        for (int j = k + 1 + g; j < n; j += G) {
          const double a = j <= row ? P[pidx(row, j)] : P[pidx(j, row)];
          acc += a * sv[j];
        }
      }
      for (int o = G >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (row < n && g == 0) sp[row] = t * acc;
    }
    __syncthreads();
    // w = p - (t/2)(p.v) v
    double pv = 0.0;
    for (int i = k + 1 + tid; i < n; i += nt) pv += sp[i] * sv[i];
    pv = block_reduce(pv, false);
    if (tid == 0) s_bc[2] = -0.5 * t * pv;
    __syncthreads();
    const double c2 = s_bc[2];
    for (int i = k + 1 + tid; i < n; i += nt) sp[i] += c2 * sv[i];
    __syncthreads();
    // A22 -= v w^T + w v^T on the packed trailing triangle: local rows r and
    // m - 1 - r share a group (r + 1 + m - r = m + 1 elements per pair)
    {
      const int npair = (m + 1) / 2;
      int G2 = 32;
      while (G2 > 1 && G2 * npair > nt) G2 >>= 1;
      const int q = tid / G2, g = tid % G2;
      if (q < npair) {
        const int r1 = q, r2 = m - 1 - q;
        const int len = (r1 + 1) + (r2 != r1 ? r2 + 1 : 0);
        for (int u = g; u < len; u += G2) {
          int r, cidx;
          if (u <= r1) {
            r = r1;
            cidx = u;
          } else {
            r = r2;
            cidx = u - r1 - 1;
          }
          const int i = k + 1 + r, j = k + 1 + cidx;
          P[pidx(i, j)] -= sv[i] * sp[j] + sp[i] * sv[j];
        }
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    if (n >= 2) {
      d[n - 2] = P[pidx(n - 2, n - 2)];
      e[n - 2] = P[pidx(n - 1, n - 2)];
      tau[n - 2] = 0.0;
    }
    d[n - 1] = P[pidx(n - 1, n - 1)];
    tau[n - 1] = 0.0;
  }
}

// The same reduction by one thread-block cluster of CS CTAs: CTA r holds the
// full rows i = r (mod CS) of A in its shared memory, so that a row's product
// with the Householder vector needs no other CTA and the FP64 work of a step is
// split CS ways.  The rank-2 update of step k - 1 is applied in the same pass
// that forms the products of step k (one read and one write of A per step).
// Per step two cluster barriers:
//   A. every CTA forms its entries x_i of column k (with the pending update) and
//      writes them into every CTA's copy of x;
//   B. after the barrier one warp forms tau and the scale from x (the same bits in
//      every CTA), all form v; each warp updates own rows, A_il -= v'_i w'_l +
//      w'_i v'_l with the last step's v' and w', takes their products with v and
//      writes p_i = tau A_i v into every CTA's copy of p;
//   after the barrier w = p - (tau/2)(p.v) v, for all entries in every CTA.
// x is rewritten only after barrier B of its step and p only after barrier A of
// the next one, so one buffer of each is enough.  Outputs as k_sytrd.
//
// Bound: the two barriers and the serial scalar part of a step (2-3 us) and, from
// n of about 300 on, FP64 throughput (3 FMAs per element and step, 2 per cycle and
// SM): 16 CTAs above SY_WIDE_N (8 CTAs 3.67 ms at n = 256 for the whole solve, 16
// CTAs 3.46 at 257).  The solve at n = 208: 4.60 ms with the packed triangle spread
// over 8 CTAs (partial products summed over the CTAs, four block reductions a
// step) and the kernels below as they were, 2.73 now; at 333: 59.5 ms by Jacobi,
// 4.9 now.
constexpr int SY_THREADS = 512, SY_WARPS = SY_THREADS / 32;
constexpr int SY_WIDE_N = 256;

__host__ __device__ __forceinline__ int sy_ld(int n) { return n | 1; }
inline size_t sy_smem_bytes(int n, int cs) {
  return ((size_t)((n + cs - 1) / cs) * sy_ld(n) + 5 * (size_t)n) * sizeof(double);
}

template <int CS>
__global__ void __launch_bounds__(SY_THREADS)
    k_sytrd_cluster(int n, const double* __restrict__ A, double* __restrict__ d, double* __restrict__ e,
                    double* __restrict__ tau, double* __restrict__ Vt, double* __restrict__ scal) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ double sm[];
  __shared__ double s_bc[3], s_amax;
  __shared__ int s_bits;
  const int r = (int)cluster.block_rank(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nq = n > r ? (n - r + CS - 1) / CS : 0;   // rows owned: r + CS q
  const int ld = sy_ld(n);
  // the buffers that other CTAs write come first, at the same offsets in every CTA
  double* x = sm;
  double* p = x + n;
  double* v = p + n;        // this step's Householder vector
  double* vp = v + n;       // the last step's v and w
  double* wp = vp + n;
  double* P = wp + n;       // owned rows
  int bits = 0;
  for (int q = warp; q < nq; q += SY_WARPS)
    for (int j = lane; j < n; j += 32) {   // the lower triangle is what counts
      const int i = r + CS * q;
      const double a = j <= i ? A[(long)i * n + j] : A[(long)j * n + i];
      P[q * ld + j] = a;
      bits |= range_bits(a);
    }
  for (int i = tid; i < n; i += SY_THREADS) vp[i] = wp[i] = 0.0;
  bits = (__syncthreads_or(bits & 1) ? 1 : 0) | (__syncthreads_or(bits & 2) ? 2 : 0);
  if (tid == 0) s_bits = bits;
  cluster.sync();
  bits = lane < CS ? *cluster.map_shared_rank(&s_bits, lane) : 0;
  int sx = 0;
  if (!__any_sync(0xffffffffu, bits & 1) || __any_sync(0xffffffffu, bits & 2)) {   // by every thread of the cluster
    double amax = 0.0;
    for (int q = warp; q < nq; q += SY_WARPS)
      for (int j = lane; j < n; j += 32) amax = fmax(amax, fabs(P[q * ld + j]));
    amax = block_reduce(amax, true);
    if (tid == 0) s_amax = amax;
    cluster.sync();
    amax = lane < CS ? *cluster.map_shared_rank(&s_amax, lane) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    sx = scale_exponent(amax);
    for (int q = warp; q < nq; q += SY_WARPS)
      for (int j = lane; j < n; j += 32) P[q * ld + j] = scalbn(P[q * ld + j], -sx);
    __syncthreads();
  }
  if (r == 0 && tid == 0) scal[3] = sx;
  for (int k = 0; k + 2 < n; ++k) {
    const int q0 = k >= r ? (k - r) / CS + 1 : 0;   // first own row > k
    // A: column k of own rows > k, to every CTA
    {
      const double wk = wp[k], vk = vp[k];
      for (int idx = tid; idx < (nq - q0) * CS; idx += SY_THREADS) {
        const int q = q0 + idx / CS, dst = idx % CS, i = r + CS * q;
        const double xi = fma(-wp[i], vk, fma(-vp[i], wk, P[q * ld + k]));
        cluster.map_shared_rank(x, dst)[i] = xi;
      }
      if (k % CS == r && tid == 0) d[k] = fma(-2.0 * vk, wk, P[(k / CS) * ld + k]);
    }
    cluster.sync();
    if (warp == 0) {
      double s = 0.0;
      for (int i = k + 2 + lane; i < n; i += 32) s = fma(x[i], x[i], s);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) {
        const double alpha = x[k + 1];
        double beta = alpha, t = 0.0, scale = 0.0;
        if (s > 0.0) {
          beta = -copysign(sqrt(fma(alpha, alpha, s)), alpha);
          t = (beta - alpha) / beta;
          scale = 1.0 / (alpha - beta);
        }
        s_bc[0] = t;
        s_bc[1] = scale;
        if (r == 0) {
          e[k] = beta;
          tau[k] = t;
        }
      }
    }
    __syncthreads();
    const double t = s_bc[0], scale = s_bc[1];
    for (int i = k + 1 + tid; i < n; i += SY_THREADS) v[i] = i == k + 1 ? 1.0 : x[i] * scale;
    __syncthreads();
    for (int i = r + CS * tid; i < n; i += CS * SY_THREADS) Vt[(long)k * n + i] = i <= k ? 0.0 : v[i];
    // B: pending update of own rows and their products with v
    for (int q = q0 + warp; q < nq; q += SY_WARPS) {
      const int i = r + CS * q;
      double* row = P + q * ld;
      const double vi = vp[i], wi = wp[i];
      double acc = 0.0;
      for (int l = k + 1 + lane; l < n; l += 32) {
        const double a = fma(-wi, vp[l], fma(-vi, wp[l], row[l]));
        row[l] = a;
        acc = fma(a, v[l], acc);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane < CS) cluster.map_shared_rank(p, lane)[i] = t * acc;
    }
    cluster.sync();
    if (warp == 0) {
      double pv = 0.0;
      for (int i = k + 1 + lane; i < n; i += 32) pv = fma(p[i], v[i], pv);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) pv += __shfl_xor_sync(0xffffffffu, pv, o);
      if (lane == 0) s_bc[2] = -0.5 * t * pv;
    }
    __syncthreads();
    const double c2 = s_bc[2];
    for (int i = k + 1 + tid; i < n; i += SY_THREADS) {
      const double vi = v[i];
      vp[i] = vi;
      wp[i] = fma(c2, vi, p[i]);
    }
    __syncthreads();
  }
  // the last 2 x 2 block, with the pending update
  if (tid == 0) {
    const int i1 = n - 1, i2 = n - 2;
    if (n >= 2) {
      if (i2 % CS == r) d[i2] = fma(-2.0 * vp[i2], wp[i2], P[(i2 / CS) * ld + i2]);
      if (i1 % CS == r) e[i2] = fma(-wp[i1], vp[i2], fma(-vp[i1], wp[i2], P[(i1 / CS) * ld + i2]));
      if (r == 0) tau[i2] = 0.0;
    }
    if (i1 % CS == r) d[i1] = fma(-2.0 * vp[i1], wp[i1], P[(i1 / CS) * ld + i1]);
    if (r == 0) tau[i1] = 0.0;
  }
  cluster.sync();   // no CTA leaves while another may still write into its shared memory
}

template <int CS>
gbhf_status sytrd_config(gbhf_ctx* c, int n, cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr) {
  cfg = {};
  cfg.gridDim = dim3(CS);
  cfg.blockDim = dim3(SY_THREADS);
  cfg.dynamicSmemBytes = sy_smem_bytes(n, CS);
  cfg.stream = c->stream;
  attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = CS;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return GBHF_OK;
}

// Whether this device runs the cluster kernel at its largest size (checked once per context).
template <int CS>
bool sytrd_runs(gbhf_ctx* c, int max_n) {
  // the attributes belong to the kernel (per device, for the whole process): always
  // the largest size, so that no context lowers it under another's launch
  bool ok = cudaFuncSetAttribute(k_sytrd_cluster<CS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sy_smem_bytes(max_n, CS)) == cudaSuccess;
  if (CS > 8)
    ok = ok && cudaFuncSetAttribute(k_sytrd_cluster<CS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  if (ok) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    sytrd_config<CS>(c, max_n, cfg, attr);
    int ncl = 0;
    ok = cudaOccupancyMaxActiveClusters(&ncl, k_sytrd_cluster<CS>, &cfg) == cudaSuccess && ncl >= 1;
  }
  (void)cudaGetLastError();   // a refused query leaves no error behind
  return ok;
}

template <int CS>
gbhf_status launch_sytrd(gbhf_ctx* c, int n, const double* d_A, TridiagWork& w) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  GBHF_TRY(sytrd_config<CS>(c, n, cfg, attr));
  GBHF_CUDA(c, cudaLaunchKernelEx(&cfg, k_sytrd_cluster<CS>, n, d_A, w.d.p, w.e.p, w.tau.p, w.Vt.p, w.scal.p));
  count_launch(c);
  return GBHF_OK;
}

// Unreduced blocks: e_i is dropped when e_i^2 <= eps^2 |d_i d_(i+1)| (or is
// zero).  blk[i] = first row of row i's block, blk[n + i] = its last row.
// Also e2 = e^2, and single-precision copies df = d, e2f = e^2 for the coarse
// bisection.  scal = {||T|| bound, pivmin, single-precision pivmin}.  One block
// of 256 threads; d and e are staged in shared memory (n <= 1024).
__global__ void __launch_bounds__(256) k_tri_prep(int n, const double* __restrict__ d, double* __restrict__ e,
                                                  int* __restrict__ blk, double* __restrict__ e2,
                                                  float* __restrict__ df, float* __restrict__ e2f,
                                                  double* __restrict__ scal, int* __restrict__ status) {
  __shared__ double sd[1025], se[1025];
  __shared__ bool cut[1024];
  __shared__ double s_red[8];
  const int tid = threadIdx.x;
  for (int i = tid; i < n; i += blockDim.x) {
    sd[i] = d[i];
    se[i] = i + 1 < n ? e[i] : 0.0;
  }
  __syncthreads();
  double tn = 0.0;
  for (int i = tid; i < n; i += blockDim.x) {
    double r = fabs(sd[i]);
    if (i > 0) r += fabs(se[i - 1]);
    if (i + 1 < n) r += fabs(se[i]);
    if (status && !(r <= DBL_MAX)) atomicOr(status, GBHF_DEV_ERR_NOTCONV);
    tn = fmax(tn, r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
  if ((tid & 31) == 0) s_red[tid >> 5] = tn;
  __syncthreads();
  __syncthreads();
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tn = fmax(tn, s_red[w]);
  // a row ends its block where the next off-diagonal is negligible
  double emax2 = 0.0;
  for (int i = tid; i < n; i += blockDim.x) {
    const double ee = se[i] * se[i];
    const bool split = i + 1 == n || se[i] == 0.0 || ee <= kEps * kEps * fabs(sd[i] * sd[i + 1]);
    cut[i] = split;
    if (!split) emax2 = fmax(emax2, ee);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) emax2 = fmax(emax2, __shfl_xor_sync(0xffffffffu, emax2, o));
  __syncthreads();   // s_red read above
  if ((tid & 31) == 0) s_red[tid >> 5] = emax2;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) emax2 = fmax(emax2, s_red[w]);
    scal[0] = fmax(tn, DBL_MIN);
    scal[1] = DBL_MIN * fmax(1.0, emax2);
    scal[2] = (double)FLT_MIN * fmax(1.0, emax2);
  }
  for (int i = tid; i < n; i += blockDim.x) {
    int lo = i, hi = i;
    while (lo > 0 && !cut[lo - 1]) --lo;
    while (!cut[hi]) ++hi;
    blk[i] = lo;
    blk[n + i] = hi;
    if (cut[i]) se[i] = 0.0;
  }
  __syncthreads();
  for (int i = tid; i < n; i += blockDim.x) {
    const double ee = se[i] * se[i];
    if (i + 1 < n) e[i] = se[i];
    e2[i] = ee;
    df[i] = (float)sd[i];
    e2f[i] = (float)ee;
  }
}

// 1/q to about an ulp with three FP64 instructions: the single-precision
// estimate of the truncated q (exponents moved with integer operations), then
// r0 (1 + h + h^2), h = 1 - q r0: |h| <= 2^-20 + 2^-23 (the estimate sees q's high
// word), so the neglected h^3 is below 2^-59; outside the
// single-precision range the plain quotient.
__device__ __forceinline__ double recip_nr(double q) {
  const int hi = __double2hiint(q), ahi = hi & 0x7fffffff;
  if ((unsigned)(ahi - 0x39b00000) >= 0x0c800000u) return 1.0 / q;   // |q| outside [2^-100, 2^100)
  const float xf = __int_as_float((ahi - 0x38000000) << 3);
  float yf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(xf));
  const int yb = __float_as_int(yf);
  const double r0 = __hiloint2double(((yb >> 3) + 0x38000000) | (hi & 0x80000000), yb << 29);
  const double h = fma(-q, r0, 1.0);
  return fma(r0, fma(h, h, h), r0);
}

// Eigenvalues of T - x I below zero in the block [s, t] (Sturm count); e2 = e^2.
// Five FP64 instructions per row (16 cycles of the SM's FP64 pipe each); signs
// and the pivot test on the high words.
__device__ int sturm_count(const double* __restrict__ d, const double* __restrict__ e2, int s, int t, double x,
                           double pivmin) {
  const int phi = __double2hiint(pivmin);
  auto guard = [&](double q) {
    if ((__double2hiint(q) & 0x7fffffff) <= phi && fabs(q) < pivmin) q = -pivmin;
    return q;
  };
  double q = guard(d[s] - x);
  int c = (unsigned)__double2hiint(q) >> 31;
  for (int i = s + 1; i <= t; ++i) {
    q = guard(fma(-e2[i - 1], recip_nr(q), d[i] - x));
    c += (unsigned)__double2hiint(q) >> 31;
  }
  return c;
}

// The same in single precision (coarse bracketing only).
__device__ int sturm_count_f(const float* __restrict__ d, const float* __restrict__ e2, int s, int t, float x,
                             float pivmin) {
  float q = d[s] - x;
  if (fabsf(q) < pivmin) q = -pivmin;
  int c = q < 0.0f;
  for (int i = s + 1; i <= t; ++i) {
    q = (d[i] - x) - __fdividef(e2[i - 1], q);
    if (fabsf(q) < pivmin) q = -pivmin;
    c += q < 0.0f;
  }
  return c;
}

// Pseudo-random start in (-1, 1) for vector k, element i (a fixed integer hash).
__device__ __forceinline__ double start_value(int k, int i) {
  unsigned h = (unsigned)k * 0x9E3779B1u ^ ((unsigned)i + 0x7F4A7C15u) * 0x85EBCA77u;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  h *= 0x297A2D39u;
  h ^= h >> 15;
  return ((double)(h >> 8) + 0.5) * (2.0 / 16777216.0) - 1.0;
}

// Inverse iteration for eigenvalue lam of block [s, t] (m = t - s + 1 >= 2),
// executed by one warp.  w: 6 m doubles of this warp's shared memory.  The
// result (unit norm) goes to zrow[s .. t]; with nprev > 0 every iterate is
// orthogonalised against rows prev[0 .. nprev) (global rows of the same
// block, unit norm) first.
__device__ void inverse_iteration(const double* __restrict__ d, const double* __restrict__ e, int s, int t,
                                  double lam, double tnorm, int seed, double* w, double* __restrict__ zrow,
                                  const double* __restrict__ prev, long prev_stride, int nprev) {
  const int lane = threadIdx.x & 31;
  const int m = t - s + 1;
  double* u0 = w;          // reciprocal pivots
  double* u1 = w + m;      // first and second superdiagonal of U, divided by the pivot
  double* u2 = w + 2 * m;
  double* l = w + 3 * m;   // multipliers
  double* piv = w + 4 * m; // 1: rows i, i + 1 exchanged
  double* x = w + 5 * m;
  const double eps_piv = kEps * tnorm;
  if (lane == 0) {
    // current row (r0, r1) at columns (i, i + 1)
    double r0 = d[s] - lam, r1 = e[s];
    for (int i = 0; i + 1 < m; ++i) {
      const double sub = e[s + i], nd = d[s + i + 1] - lam, ns1 = (i + 2 < m) ? e[s + i + 1] : 0.0;
      if (fabs(r0) >= fabs(sub)) {
        if (r0 == 0.0) r0 = eps_piv;
        const double rc = recip_nr(r0), mlt = sub * rc;
        u0[i] = rc;
        u1[i] = r1;
        u2[i] = 0.0;
        l[i] = mlt;
        piv[i] = 0.0;
        r0 = nd - mlt * r1;
        r1 = ns1;
      } else {
        const double rc = recip_nr(sub), mlt = r0 * rc;
        u0[i] = rc;
        u1[i] = nd;
        u2[i] = ns1;
        l[i] = mlt;
        piv[i] = 1.0;
        r0 = r1 - mlt * nd;
        r1 = -mlt * ns1;
      }
    }
    if (r0 == 0.0) r0 = eps_piv;
    u0[m - 1] = 1.0 / r0;
    u1[m - 1] = u2[m - 1] = 0.0;
  }
  __syncwarp();
  for (int i = lane; i < m; i += 32) {
    u1[i] *= u0[i];
    u2[i] *= u0[i];
    x[i] = start_value(seed, i);
  }
  __syncwarp();
  // the serial chains of a solve are one FP64 FMA per row; a solve that grows
  // its unit input to within a factor of 100 m of 1 / (eps ||T||) is followed by
  // one more, at most four in all
  bool last = false;
  for (int it = 0; it < 4; ++it) {
    if (lane == 0) {
      double xi = x[0];
#pragma unroll 4
      for (int i = 0; i + 1 < m; ++i) {
        double xn = x[i + 1];
        if (piv[i] != 0.0) {
          const double tmp = xi;
          xi = xn;
          xn = tmp;
        }
        x[i] = xi;
        xi = fma(-l[i], xi, xn);
      }
      x[m - 1] = xi;
      double x1 = 0.0, x2 = 0.0;
#pragma unroll 4
      for (int i = m - 1; i >= 0; --i) {
        const double v = fma(-u1[i], x1, fma(-u2[i], x2, x[i] * u0[i]));
        x[i] = v;
        x2 = x1;
        x1 = v;
      }
    }
    __syncwarp();
    for (int p = 0; p < nprev; ++p) {
      const double* pr = prev + p * prev_stride + s;
      double dot = 0.0;
      for (int i = lane; i < m; i += 32) dot += pr[i] * x[i];
      for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      for (int i = lane; i < m; i += 32) x[i] -= dot * pr[i];
      __syncwarp();
    }
    double nrm = 0.0;
    for (int i = lane; i < m; i += 32) nrm += x[i] * x[i];
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
    for (int i = lane; i < m; i += 32) x[i] *= inv;
    __syncwarp();
    if (last) break;
    last = it > 0 && inv * 0.01 < m * kEps * tnorm;   // (the start vector is not normalised)
  }
  for (int i = lane; i < m; i += 32) zrow[s + i] = x[i];
  __syncwarp();
}

// One step of 32-point multisection: the new bracket from the counts at the
// 32 interior points x (one per lane); invariant count(lo) <= j < count(hi).
template <typename R>
__device__ __forceinline__ void multisect(R x, int c, int j, R& lo, R& hi) {
  const unsigned le = __ballot_sync(0xffffffffu, c <= j);
  const int lo_lane = le ? 31 - __clz(le) : -1;             // highest lane with count <= j
  const unsigned gt = ~le;
  const int hi_lane = gt ? __ffs(gt) - 1 : 32;              // lowest lane with count > j
  const R xlo = __shfl_sync(0xffffffffu, x, lo_lane < 0 ? 0 : lo_lane);
  const R xhi = __shfl_sync(0xffffffffu, x, hi_lane > 31 ? 31 : hi_lane);
  const R nlo = lo_lane >= 0 ? xlo : lo;
  R nhi = hi_lane <= 31 ? xhi : hi;
  if (!(nhi > nlo)) {   // counts not monotone in rounding: keep a valid bracket
    const R xn = __shfl_sync(0xffffffffu, x, (lo_lane >= 0 && lo_lane < 31) ? lo_lane + 1 : 31);
    nhi = (lo_lane >= 0 && lo_lane < 31) ? xn : hi;
  }
  lo = nlo;
  hi = nhi > nlo ? nhi : nlo;
}

// One warp per eigenvalue index k (the k-th row's block, local index k - s).
// Zt row k receives the vector (zeros outside the block), lam[k] the value.
// The bracket is first narrowed to ~1e-4 of the block's Gershgorin bound with
// single-precision Sturm counts (64 times the FP64 rate on this GPU), widened
// by a margin well above their error, checked with two FP64 counts (else the
// whole interval is kept), then refined in FP64.
__global__ void k_tri_vec(int n, const double* __restrict__ d, const double* __restrict__ e,
                          const double* __restrict__ e2, const float* __restrict__ df,
                          const float* __restrict__ e2f, const int* __restrict__ blk,
                          const double* __restrict__ scal, double* __restrict__ lam, double* __restrict__ Zt) {
  extern __shared__ double smw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int k = blockIdx.x * (blockDim.x >> 5) + wib;
  if (k >= n) return;   // whole warps leave together
  double* w = smw + (long)wib * 6 * n;
  const int s = blk[k], t = blk[n + k], j = k - s;
  const double tnorm = scal[0], pivmin = scal[1];
  const float pivf = (float)scal[2];
  double* zrow = Zt + (long)k * n;
  for (int i = lane; i < n; i += 32) zrow[i] = (i == k && s == t) ? 1.0 : 0.0;
  if (s == t) {
    if (lane == 0) lam[k] = d[k];
    return;
  }
  // Gershgorin interval of the block
  double lo = INFINITY, hi = -INFINITY;
  for (int i = s + lane; i <= t; i += 32) {
    const double r = (i > s ? fabs(e[i - 1]) : 0.0) + (i < t ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const double tb = fmax(fabs(lo), fabs(hi));
  lo -= 2.0 * kEps * tb + 2.0 * pivmin;
  hi += 2.0 * kEps * tb + 2.0 * pivmin;
  {
    // coarse: three FP32 rounds (width / 33^3), then a margin of 2e-4 tb on each side
    float lof = (float)lo, hif = (float)hi;
    for (int it = 0; it < 3; ++it) {
      const float x = lof + (hif - lof) * ((float)(lane + 1) / 33.0f);
      multisect<float>(x, sturm_count_f(df, e2f, s, t, x, pivf), j, lof, hif);
    }
    const double lo2 = fmax(lo, (double)lof - 2e-4 * tb), hi2 = fmin(hi, (double)hif + 2e-4 * tb);
    int cv = 0;
    if (lane < 2) cv = sturm_count(d, e2, s, t, lane == 0 ? lo2 : hi2, pivmin);
    const int c_lo = __shfl_sync(0xffffffffu, cv, 0), c_hi = __shfl_sync(0xffffffffu, cv, 1);
    if (c_lo <= j && c_hi > j) {
      lo = lo2;
      hi = hi2;
    }
  }
  for (int it = 0; it < 40; ++it) {
    if (hi - lo <= 2.0 * kEps * fmax(fabs(lo), fabs(hi)) + 0.5 * kEps * tb + pivmin) break;
    const double x = lo + (hi - lo) * ((double)(lane + 1) / 33.0);
    multisect<double>(x, sturm_count(d, e2, s, t, x, pivmin), j, lo, hi);
  }
  const double lambda = 0.5 * (lo + hi);
  if (lane == 0) lam[k] = lambda;
  inverse_iteration(d, e, s, t, lambda, tnorm, k, w, zrow, nullptr, 0, 0);
}

// One block.  Warp 0 recomputes the vectors of eigenvalues within 1e-11 ||T||
// of the previous one in the same block, orthogonalised against the earlier
// members of that run; then every thread ranks the eigenvalues (ascending,
// ties by index) and writes evals in sorted order.
__global__ void __launch_bounds__(256) k_tri_fix(int n, const double* __restrict__ d, const double* __restrict__ e,
                          const int* __restrict__ blk, const double* __restrict__ scal,
                          const double* __restrict__ lam, double* __restrict__ Zt, int* __restrict__ rank,
                          double* __restrict__ evals) {
  extern __shared__ double smw[];
  __shared__ double sl[TRIDIAG_WIDE_MAX_N];
  __shared__ unsigned char close[TRIDIAG_WIDE_MAX_N];
  const double tnorm = scal[0];
  const int sx = (int)scal[3];   // exponent of the scaling (scale_exponent)
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    sl[k] = lam[k];
    close[k] = k > 0 && blk[k] == blk[k - 1] && blk[k] != blk[n + k] && lam[k] - lam[k - 1] < 1e-11 * tnorm;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int run0 = 0;
    for (int k = 1; k < n; ++k) {
      if (!close[k]) {
        run0 = k;
        continue;
      }
      inverse_iteration(d, e, blk[k], blk[n + k], sl[k], tnorm, k + 7919, smw, Zt + (long)k * n,
                        Zt + (long)run0 * n, n, k - run0);
    }
  }
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const double v = sl[k];
    int r = 0;
    for (int q = 0; q < n; ++q) {
      const double u = sl[q];
      r += (u < v) || (u == v && q < k);
    }
    rank[k] = r;
    evals[r] = sx ? scalbn(v, sx) : v;
  }
}

__global__ void k_ns_mat(int n, const double* __restrict__ S, double* __restrict__ M) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < (long)n * n; q += (long)gridDim.x * blockDim.x) {
    const int i = (int)(q / n), j = (int)(q % n);
    M[q] = (i == j ? 1.5 : 0.0) - 0.5 * S[q];
  }
}

// z <- H_0 ... H_(n-3) z for every vector (rows of Zt), written to column
// rank[k] of evecs (n x n row-major).  One warp per vector, TB_WARPS vectors
// per block; each reflector row is loaded once per block into shared memory
// (double-buffered: row r - 1 loads while row r is applied), one barrier per
// reflector.
// TB_WARPS 2 (n <= 304: a block per SM) or 4: a warp's 3 n / 32 FP64 instructions
// per reflector take 16 cycles of its SM's FP64 pipe each (eight warps per block
// filled 26 of the 152 SMs at n = 208).
template <int TB_WARPS>
__global__ void __launch_bounds__(TB_WARPS * 32) k_tri_back(int n, const double* __restrict__ Vt,
                                                            const double* __restrict__ tau,
                                                            const double* __restrict__ Zt,
                                                            const int* __restrict__ rank,
                                                            double* __restrict__ evecs) {
  extern __shared__ double smw[];
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int k = blockIdx.x * TB_WARPS + wib;
  double* vbuf = smw;                       // 2 x n
  double* z = smw + 2 * n + (long)wib * n;  // this warp's vector
  if (k < n)
    for (int i = lane; i < n; i += 32) z[i] = Zt[(long)k * n + i];
  const int r0 = n - 3;
  if (r0 >= 0)
    for (int i = tid; i < n; i += blockDim.x) vbuf[(r0 & 1) * n + i] = Vt[(long)r0 * n + i];
  __syncthreads();
  for (int r = r0; r >= 0; --r) {
    // next row into the other buffer (read in the step after the barrier below)
    if (r > 0)
      for (int i = tid; i < n; i += blockDim.x) vbuf[((r - 1) & 1) * n + i] = Vt[(long)(r - 1) * n + i];
    const double tr = tau[r];
    if (k < n && tr != 0.0) {
      const double* v = vbuf + (r & 1) * n;
      double dot = 0.0;
      for (int i = r + 1 + lane; i < n; i += 32) dot += v[i] * z[i];
      for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      const double f = tr * dot;
      for (int i = r + 1 + lane; i < n; i += 32) z[i] -= f * v[i];
    }
    __syncthreads();
  }
  if (k < n) {
    const int col = rank[k];
    for (int i = lane; i < n; i += 32) evecs[(long)i * n + col] = z[i];
  }
}

}  // namespace

size_t tridiag_smem_bytes(int n) { return (size_t)(pidx(n, 0) + 2 * (long)n) * sizeof(double); }

// The widest cluster form that runs here: 16 CTAs, 8, or none.
static void check_sytrd(gbhf_ctx* c) {
  if (c->sytrd_checked) return;
  c->sytrd_checked = true;
  c->sytrd8 = sytrd_runs<8>(c, SY_WIDE_N);
  c->sytrd16 = sytrd_runs<16>(c, TRIDIAG_WIDE_MAX_N);
}

bool tridiag_takes(gbhf_ctx* c, int n) {
  if (c->force_jacobi) return false;
  if (n <= TRIDIAG_MAX_N) return tridiag_smem_bytes(n) <= c->smem_optin;
  if (n > TRIDIAG_WIDE_MAX_N || c->force_sytrd_single) return false;
  check_sytrd(c);
  return n <= SY_WIDE_N ? c->sytrd8 || c->sytrd16 : c->sytrd16;
}

// d_evecs (n x n): eigenvectors of A in columns, ascending eigenvalues.
gbhf_status eigh_tridiag(gbhf_ctx* c, int n, const double* d_A, double* d_evals, double* d_evecs) {
  TridiagWork& w = c->tri;
  const size_t nn = (size_t)n * n;
  GBHF_CUDA(c, w.d.alloc(n));
  GBHF_CUDA(c, w.e.alloc(n));
  GBHF_CUDA(c, w.tau.alloc(n));
  GBHF_CUDA(c, w.lam.alloc(n));
  GBHF_CUDA(c, w.scal.alloc(4));
  GBHF_CUDA(c, w.e2.alloc(n));
  GBHF_CUDA(c, w.df.alloc(n));
  GBHF_CUDA(c, w.e2f.alloc(n));
  GBHF_CUDA(c, w.Vt.alloc(nn));
  GBHF_CUDA(c, w.Zt.alloc(nn));
  GBHF_CUDA(c, w.Z2.alloc(nn));
  GBHF_CUDA(c, w.S.alloc(nn));
  GBHF_CUDA(c, w.M.alloc(nn));
  GBHF_CUDA(c, w.blk.alloc(2 * (size_t)n));
  GBHF_CUDA(c, w.rank.alloc(n));
  const size_t smem = tridiag_smem_bytes(n);   // of the one-CTA form, n <= TRIDIAG_MAX_N
  // The attribute belongs to the kernel (per device, for the whole process):
  // always the largest size, so that no context lowers it under another's launch.
  GBHF_CUDA(c, cudaFuncSetAttribute(k_sytrd, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)tridiag_smem_bytes(TRIDIAG_MAX_N)));
  if (n > 1) {
    GBHF_CUDA(c, cudaMemsetAsync(w.e.p, 0, n * sizeof(double), c->stream));
  }
  // above the one-CTA sizes a matrix with a non-finite entry is reported, as the
  // Jacobi solver reports it
  const bool wide = n > TRIDIAG_MAX_N;
  if (wide) {
    GBHF_CUDA(c, c->dev_status.alloc(1));
    GBHF_CUDA(c, cudaMemsetAsync(c->dev_status.p, 0, sizeof(int), c->stream));
  }
  // the cluster forms where the device runs them; below two rows per CTA one CTA
  check_sytrd(c);
  if (c->sytrd8 && !c->force_sytrd_single && n >= 16 && n <= SY_WIDE_N) {
    GBHF_TRY(launch_sytrd<8>(c, n, d_A, w));
  } else if (c->sytrd16 && !c->force_sytrd_single && n >= 32) {
    GBHF_TRY(launch_sytrd<16>(c, n, d_A, w));
  } else {
    k_sytrd<<<1, 1024, smem, c->stream>>>(n, d_A, w.d.p, w.e.p, w.tau.p, w.Vt.p, w.scal.p);
    count_launch(c);
    GBHF_LAUNCHED(c, "k_sytrd launch");
  }
  k_tri_prep<<<1, 256, 0, c->stream>>>(n, w.d.p, w.e.p, w.blk.p, w.e2.p, w.df.p, w.e2f.p, w.scal.p,
                                      wide ? c->dev_status.p : nullptr);
  count_launch(c);
  GBHF_LAUNCHED(c, "k_tri_prep launch");
  const int wpb = 2;   // warps per block: vectors spread over many SMs
  GBHF_CUDA(c, cudaFuncSetAttribute(k_tri_vec, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(wpb * 6 * TRIDIAG_WIDE_MAX_N * sizeof(double))));
  const size_t vsm = (size_t)wpb * 6 * n * sizeof(double);
  k_tri_vec<<<(n + wpb - 1) / wpb, 32 * wpb, vsm, c->stream>>>(n, w.d.p, w.e.p, w.e2.p, w.df.p, w.e2f.p, w.blk.p,
                                                               w.scal.p, w.lam.p, w.Zt.p);
  count_launch(c);
  GBHF_LAUNCHED(c, "k_tri_vec launch");
  k_tri_fix<<<1, 256, 6 * n * sizeof(double), c->stream>>>(n, w.d.p, w.e.p, w.blk.p, w.scal.p, w.lam.p, w.Zt.p,
                                                            w.rank.p, d_evals);
  count_launch(c);
  GBHF_LAUNCHED(c, "k_tri_fix launch");
  // Newton-Schulz: Zt <- (3 I - Zt Zt^T) Zt / 2, twice
  double* zin = w.Zt.p;
  double* zout = w.Z2.p;
  for (int step = 0; step < 2; ++step) {
    GBHF_TRY(gemm(c, false, true, n, n, n, 1.0, zin, n, zin, n, 0.0, w.S.p, n, true));
    k_ns_mat<<<std::max(1, std::min(c->nsm * 4, (int)((nn + 255) / 256))), 256, 0, c->stream>>>(n, w.S.p, w.M.p);
    count_launch(c);
    GBHF_LAUNCHED(c, "k_ns_mat launch");
    GBHF_TRY(gemm(c, false, false, n, n, n, 1.0, w.M.p, n, zin, n, 0.0, zout, n));
    std::swap(zin, zout);
  }
  if (n <= 304)
    k_tri_back<2><<<(n + 1) / 2, 64, 4 * (size_t)n * sizeof(double), c->stream>>>(n, w.Vt.p, w.tau.p, zin, w.rank.p,
                                                                                  d_evecs);
  else
    k_tri_back<4><<<(n + 3) / 4, 128, 6 * (size_t)n * sizeof(double), c->stream>>>(n, w.Vt.p, w.tau.p, zin, w.rank.p,
                                                                                   d_evecs);
  count_launch(c);
  GBHF_LAUNCHED(c, "k_tri_back launch");
  if (wide) {
    int st = 0;
    GBHF_CUDA(c, cudaMemcpyAsync(&st, c->dev_status.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    GBHF_CUDA(c, cudaStreamSynchronize(c->stream));
    if (st & GBHF_DEV_ERR_NOTCONV) return fail(c, GBHF_ERR_NOT_CONVERGED, "eigen-solver: non-finite matrix");
  }
  return GBHF_OK;
}

}  // namespace gbhf
