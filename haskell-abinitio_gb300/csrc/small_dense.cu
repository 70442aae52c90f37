// The SCF's dense steps for small matrices (n <= SMALL_DENSE_MAX_N), each as one
// launch of a thread-block cluster that holds every matrix in shared memory: the
// density by trace-correcting purification, S^(-1/2) by Newton-Schulz, the DIIS
// error.  At these sizes the general path spends its time in latency, not
// arithmetic: launches of a few microseconds each and, inside the purification, a
// grid barrier, atomics and dependent global loads per step (11 us per step at
// n = 13, where the 16 DMMA of the step take under 1 us).
//
// Every CTA of the cluster keeps a copy of all operands.  The 8 x 8 output tiles of
// a product go round the CTAs' warps; a warp writes its tile into every CTA's copy
// through distributed shared memory, and one cluster barrier ends the product.
//
// Measured against the general path's launches: density step (X^T F X to X P X^T)
// n = 13 0.352 -> 0.096 ms, 26 0.483 -> 0.150, 52 0.592 -> 0.275; DIIS error and its
// scalar products 13 0.129 -> 0.091, 39 0.159 -> 0.104; set-up with S^(-1/2) 13 0.71
// -> 0.23, 52 0.96 -> 0.50.  Larger n gives the FP64 pipes of eight SMs more work than
// the launches cost (density 0.415 ms at n = 65, 0.284 by the general path; DIIS error
// 0.126 at 52, 0.106 there): hence the limits.
#include <algorithm>

#include <cooperative_groups.h>

#include "dense.cuh"
#include "gbhf_internal.h"

namespace gbhf {

namespace {

namespace cg = cooperative_groups;

constexpr int SD_THREADS = 256, SD_WARPS = SD_THREADS / 32, SD_MAX_CS = 8, SD_NBUF = 5;

// Rows of n8 = n rounded up to 8 (padding zero), leading dimension 4 modulo 8:
// the fragments' 8 rows x 4 columns fall on different banks.
__host__ __device__ inline int sd_n8(int n) { return (n + 7) / 8 * 8; }
__host__ __device__ inline int sd_ld(int n) { return sd_n8(n) + 4; }
size_t sd_smem(int n, int nbuf) { return (size_t)nbuf * sd_n8(n) * sd_ld(n) * sizeof(double); }

struct Tile {
  int rt, ct;
  __device__ int row(int lane) const { return rt * 8 + (lane >> 2); }   // of this lane's two results
  __device__ int col(int lane) const { return ct * 8 + 2 * (lane & 3); }
};

// Tiles of this warp: all (sym = false) or those on and above the diagonal.
template <class F>
__device__ __forceinline__ void for_tiles(const cg::cluster_group& cl, int nt, bool sym, F&& f) {
  const int cs = (int)cl.num_blocks(), total = sym ? nt * (nt + 1) / 2 : nt * nt;
  for (int t = (int)cl.block_rank() + cs * (threadIdx.x >> 5); t < total; t += cs * SD_WARPS) {
    Tile w;
    if (sym) {
      int q = t;
      w.rt = 0;
      while (q >= nt - w.rt) {
        q -= nt - w.rt;
        ++w.rt;
      }
      w.ct = w.rt + q;
    } else {
      w.rt = t / nt;
      w.ct = t - w.rt * nt;
    }
    f(w);
  }
}

// One tile of A B by DMMA; a(row, k) and b(k, col) give the elements.
template <class A, class B>
__device__ __forceinline__ void tile_mul(Tile w, int n8, A&& a, B&& b, double& v0, double& v1) {
  const int lane = threadIdx.x & 31, r = w.rt * 8 + (lane >> 2), c = w.ct * 8 + (lane >> 2), q = lane & 3;
  double x0 = 0, x1 = 0, y0 = 0, y1 = 0;   // two chains
  for (int k = q; k < n8; k += 8) {
    dmma(x0, x1, a(r, k), b(k, c));
    dmma(y0, y1, a(r, k + 4), b(k + 4, c));
  }
  v0 = x0 + y0;
  v1 = x1 + y1;
}

// A tile into every CTA's copy of a matrix, with its mirror when sym.
__device__ __forceinline__ void put(const cg::cluster_group& cl, double* buf, int ld, Tile w, bool mirror, double v0,
                                    double v1) {
  const int lane = threadIdx.x & 31, r = w.row(lane), c = w.col(lane), cs = (int)cl.num_blocks();
  for (int d = 0; d < cs; ++d) {
    double* p = cl.map_shared_rank(buf, d);
    *reinterpret_cast<double2*>(p + r * ld + c) = make_double2(v0, v1);
    if (mirror && w.rt < w.ct) {
      p[c * ld + r] = v0;
      p[(c + 1) * ld + r] = v1;
    }
  }
}

// n x n from global memory, zero padded.
__device__ __forceinline__ void load_padded(double* dst, const double* __restrict__ src, int n, double scale = 1.0) {
  const int n8 = sd_n8(n), ld = sd_ld(n);
  for (int e = threadIdx.x; e < n8 * n8; e += SD_THREADS) {
    const int i = e / n8, j = e - i * n8;
    dst[i * ld + j] = i < n && j < n ? scale * src[i * n + j] : 0.0;
  }
}

// Gershgorin bounds of a matrix (every thread gets them); get(i, j) gives an element.
template <class G>
__device__ __forceinline__ void gershgorin(int n, G&& get, double& lo, double& hi) {
  __shared__ double s_lo[SD_WARPS], s_hi[SD_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  lo = 1e300;
  hi = -1e300;
  for (int i = warp; i < n; i += SD_WARPS) {
    double r = 0;
    for (int j = lane; j < n; j += 32)
      if (j != i) r += fabs(get(i, j));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    const double d = get(i, i);
    lo = fmin(lo, d - r);
    hi = fmax(hi, d + r);
  }
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  lo = s_lo[0];
  hi = s_hi[0];
  for (int w = 1; w < SD_WARPS; ++w) {
    lo = fmin(lo, s_lo[w]);
    hi = fmax(hi, s_hi[w]);
  }
}

// Sum of n8 values in shared memory by one warp, to *out.
__device__ __forceinline__ void warp_sum(const double* v, int n8, double* out) {
  const int lane = threadIdx.x & 31;
  double s = 0;
  for (int i = lane; i < n8; i += 32) s += v[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) *out = s;
}

// D = X (2 P) X^T with P the projector of X^T F X onto its ne lowest eigenvectors:
// the steps of k_tc2_fused.  A tile's owner sends both candidates for the next P
// (P^2 and 2 P - P^2) and their diagonals; after the barrier every CTA adds the
// same diagonals, so all take the same decision and the next P is already there.
// rec: tr(P - P^2), steps, device status (0).
__global__ void __launch_bounds__(SD_THREADS) k_density_small(int n, int ne, int max_steps, double tol,
                                                              const double* __restrict__ F,
                                                              const double* __restrict__ X, double* __restrict__ D,
                                                              double* __restrict__ rec) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double dg[2][2][SMALL_DENSE_MAX_N];   // [step parity][P^2, 2 P - P^2] diagonals
  __shared__ double s_t[2];
  const cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n8 = sd_n8(n), ld = sd_ld(n), nt = n8 / 8, cs = (int)cl.num_blocks();
  double *fb = sm, *xb = fb + n8 * ld, *tb = xb + n8 * ld, *pb = tb + n8 * ld;
  load_padded(fb, F, n);
  load_padded(xb, X, n);
  cl.sync();   // all copies loaded, all CTAs running
  for_tiles(cl, nt, false, [&](Tile w) {
    double v0, v1;
    tile_mul(w, n8, [&](int r, int k) { return xb[k * ld + r]; }, [&](int k, int c) { return fb[k * ld + c]; }, v0, v1);
    put(cl, tb, ld, w, false, v0, v1);
  });
  cl.sync();
  for_tiles(cl, nt, true, [&](Tile w) {
    double v0, v1;
    tile_mul(w, n8, [&](int r, int k) { return tb[r * ld + k]; }, [&](int k, int c) { return xb[k * ld + c]; }, v0, v1);
    put(cl, pb, ld, w, true, v0, v1);
  });
  cl.sync();
  {   // the spectrum mapped onto [0, 1], reversed
    double lo, hi;
    gershgorin(n, [&](int i, int j) { return pb[i * ld + j]; }, lo, hi);
    const double sc = hi > lo ? 1.0 / (hi - lo) : 0.0;
    __syncthreads();
    for (int e = tid; e < n * n; e += SD_THREADS) {
      const int i = e / n, j = e - i * n;
      const double v = sc * ((i == j ? hi : 0.0) - pb[i * ld + j]);
      pb[i * ld + j] = v;
      if (i == j) dg[1][0][i] = v;
    }
    for (int i = n + tid; i < n8; i += SD_THREADS) dg[1][0][i] = 0.0;
    __syncthreads();
    if (warp == 0) warp_sum(dg[1][0], n8, &s_t[0]);
    __syncthreads();
  }
  double t1 = s_t[0], den = 0.0;
  // dg[1] is written again, by any CTA, only after the barrier of step 0
  double *cur = pb, *sq_buf = fb, *ex_buf = tb;
  int steps = 0;
  for (int step = 0; step < max_steps; ++step) {
    const int par = step & 1;
    for_tiles(cl, nt, true, [&](Tile w) {
      double v0, v1;
      tile_mul(w, n8, [&](int r, int k) { return cur[r * ld + k]; }, [&](int k, int c) { return cur[c * ld + k]; }, v0,
               v1);
      const int r = w.row(lane), c = w.col(lane);
      const double e0 = __fma_rn(2.0, cur[r * ld + c], -v0), e1 = __fma_rn(2.0, cur[r * ld + c + 1], -v1);
      put(cl, sq_buf, ld, w, true, v0, v1);
      put(cl, ex_buf, ld, w, true, e0, e1);
      if (w.rt == w.ct && (r == c || r == c + 1))
        for (int d = 0; d < cs; ++d) {
          cl.map_shared_rank(&dg[par][0][0], d)[r] = r == c ? v0 : v1;
          cl.map_shared_rank(&dg[par][1][0], d)[r] = r == c ? e0 : e1;
        }
    });
    cl.sync();
    if (warp < 2) warp_sum(dg[par][warp], n8, &s_t[warp]);
    __syncthreads();
    const double t2 = s_t[0], te = s_t[1];
    den = t1 - t2;
    steps = step + 1;
    if (fabs(den) < tol * max(1, ne)) break;   // the same decision in every thread of the cluster
    const bool sq = fabs(t2 - ne) < fabs(2 * t1 - t2 - ne);
    double* next = sq ? sq_buf : ex_buf;
    (sq ? sq_buf : ex_buf) = cur;
    cur = next;
    t1 = sq ? t2 : te;
  }
  if (cl.block_rank() == 0 && tid == 0) {
    rec[0] = den;
    rec[1] = steps;
    rec[2] = 0.0;
  }
  // one of the other buffers: all CTAs are past the barrier after its last readers
  double* yb = sq_buf;
  for_tiles(cl, nt, false, [&](Tile w) {
    double v0, v1;
    tile_mul(w, n8, [&](int r, int k) { return xb[r * ld + k]; }, [&](int k, int c) { return cur[k * ld + c]; }, v0, v1);
    put(cl, yb, ld, w, false, 2.0 * v0, 2.0 * v1);
  });
  cl.sync();   // also: no CTA leaves while another may still write into its copies
  for_tiles(cl, nt, true, [&](Tile w) {
    double v[2];
    tile_mul(w, n8, [&](int r, int k) { return yb[r * ld + k]; }, [&](int k, int c) { return xb[c * ld + k]; }, v[0],
             v[1]);
    const int r = w.row(lane), c = w.col(lane);
    for (int h = 0; h < 2; ++h)
      if (r < n && c + h < n) {
        D[r * n + c + h] = v[h];
        if (w.rt < w.ct) D[(c + h) * n + r] = v[h];
      }
  });
}

// S^(-1/2): the iteration of inv_sqrt_dev, checked for convergence at the same
// steps.  out: the last max |Z Y - I|, iterations.
__global__ void __launch_bounds__(SD_THREADS) k_inv_sqrt_small(int n, const double* __restrict__ S,
                                                               double* __restrict__ X, double* __restrict__ out) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double errs[SD_MAX_CS * SD_WARPS];
  const cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n8 = sd_n8(n), ld = sd_ld(n), nt = n8 / 8, cs = (int)cl.num_blocks();
  double *Y = sm, *Z = Y + n8 * ld, *M = Z + n8 * ld, *T = M + n8 * ld, *U = T + n8 * ld;
  double lo, g1;
  gershgorin(n, [&](int i, int j) { return S[i * n + j]; }, lo, g1);
  load_padded(Y, S, n, 1.0 / g1);
  for (int e = tid; e < n8 * n8; e += SD_THREADS) {
    const int i = e / n8, j = e - i * n8;
    Z[i * ld + j] = i == j && i < n ? 1.0 : 0.0;
  }
  cl.sync();
  double err = 1;
  int it = 0;
  for (; it < 100; ++it) {
    const bool check = it % 3 == 2;
    double e = 0;
    for_tiles(cl, nt, false, [&](Tile w) {
      double v[2];
      tile_mul(w, n8, [&](int r, int k) { return Z[r * ld + k]; }, [&](int k, int c) { return Y[k * ld + c]; }, v[0],
               v[1]);
      const int r = w.row(lane), c = w.col(lane);
      for (int h = 0; h < 2; ++h) {
        const bool diag = r == c + h;
        if (r < n && c + h < n) e = fmax(e, fabs(v[h] - (diag ? 1.0 : 0.0)));
        v[h] = (diag && r < n ? 3.0 : 0.0) - v[h];
      }
      put(cl, M, ld, w, false, v[0], v[1]);
    });
    if (check) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e = fmax(e, __shfl_xor_sync(0xffffffffu, e, o));
      if (lane < cs) cl.map_shared_rank(errs, lane)[(int)cl.block_rank() * SD_WARPS + warp] = e;
    }
    cl.sync();
    if (check) {
      err = 0;
      for (int i = 0; i < cs * SD_WARPS; ++i) err = fmax(err, errs[i]);
      if (err < 1e-14) break;   // the same decision in every thread of the cluster
    }
    for_tiles(cl, nt, false, [&](Tile w) {
      double v0, v1;
      tile_mul(w, n8, [&](int r, int k) { return Y[r * ld + k]; }, [&](int k, int c) { return M[k * ld + c]; }, v0, v1);
      put(cl, T, ld, w, false, 0.5 * v0, 0.5 * v1);
      tile_mul(w, n8, [&](int r, int k) { return M[r * ld + k]; }, [&](int k, int c) { return Z[k * ld + c]; }, v0, v1);
      put(cl, U, ld, w, false, 0.5 * v0, 0.5 * v1);
    });
    cl.sync();
    double* q = Y;
    Y = T;
    T = q;
    q = Z;
    Z = U;
    U = q;
  }
  // (the last barrier of the loop also keeps the CTAs until all remote writes are done)
  const double root = sqrt(g1);
  for (int e = (int)cl.block_rank() * SD_THREADS + tid; e < n * n; e += cs * SD_THREADS) {
    const int i = e / n;
    X[e] = Z[i * ld + e - i * n] / root;
  }
  if (cl.block_rank() == 0 && tid == 0) {
    out[0] = err;
    out[1] = it;
  }
}

// e = X^T (F D S - (F D S)^T) X, as diis_error_dev.
__global__ void __launch_bounds__(SD_THREADS) k_diis_error_small(int n, const double* __restrict__ F,
                                                                 const double* __restrict__ S,
                                                                 const double* __restrict__ D,
                                                                 const double* __restrict__ X, double* __restrict__ E) {
  extern __shared__ __align__(16) double sm[];
  const cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31;
  const int n8 = sd_n8(n), ld = sd_ld(n), nt = n8 / 8;
  double *fb = sm, *sb = fb + n8 * ld, *db = sb + n8 * ld, *xb = db + n8 * ld, *tb = xb + n8 * ld;
  load_padded(fb, F, n);
  load_padded(sb, S, n);
  load_padded(db, D, n);
  load_padded(xb, X, n);
  cl.sync();
  for_tiles(cl, nt, false, [&](Tile w) {
    double v0, v1;
    tile_mul(w, n8, [&](int r, int k) { return db[r * ld + k]; }, [&](int k, int c) { return sb[k * ld + c]; }, v0, v1);
    put(cl, tb, ld, w, false, v0, v1);
  });
  cl.sync();
  for_tiles(cl, nt, false, [&](Tile w) {   // F D S over D
    double v0, v1;
    tile_mul(w, n8, [&](int r, int k) { return fb[r * ld + k]; }, [&](int k, int c) { return tb[k * ld + c]; }, v0, v1);
    put(cl, db, ld, w, false, v0, v1);
  });
  cl.sync();
  for_tiles(cl, nt, false, [&](Tile w) {   // (F D S - S D F) X over S
    double v0, v1;
    tile_mul(w, n8, [&](int r, int k) { return db[r * ld + k] - db[k * ld + r]; },
             [&](int k, int c) { return xb[k * ld + c]; }, v0, v1);
    put(cl, sb, ld, w, false, v0, v1);
  });
  cl.sync();
  for_tiles(cl, nt, false, [&](Tile w) {
    double v[2];
    tile_mul(w, n8, [&](int r, int k) { return xb[k * ld + r]; }, [&](int k, int c) { return sb[k * ld + c]; }, v[0],
             v[1]);
    const int r = w.row(lane), c = w.col(lane);
    for (int h = 0; h < 2; ++h)
      if (r < n && c + h < n) E[r * n + c + h] = v[h];
  });
}

// One CTA to n = 16 (at most four tiles: eight CTAs were 10% slower), four to n = 32
// (n = 26: 0.294 ms with one, 0.150 with four, 0.156 with eight), then the portable
// eight (n = 52: 1.06 with one, 0.352 with four, 0.276 with eight).
int sd_cluster(int n) {
  const int nt = sd_n8(n) / 8;
  return nt <= 2 ? 1 : (nt <= 4 ? 4 : SD_MAX_CS);
}

void sd_config(gbhf_ctx* c, int n, int nbuf, int cs, cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr) {
  cfg = {};
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(SD_THREADS);
  cfg.dynamicSmemBytes = sd_smem(n, nbuf);
  cfg.stream = c->stream;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cs;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
}

template <class K>
bool sd_runs(gbhf_ctx* c, K kernel, int nbuf) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sd_config(c, SMALL_DENSE_MAX_N, nbuf, SD_MAX_CS, cfg, attr);
  int ncl = 0;
  const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)cfg.dynamicSmemBytes) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&ncl, kernel, &cfg) == cudaSuccess && ncl >= 1;
  if (!ok) cudaGetLastError();
  return ok;
}

}  // namespace

bool small_dense_takes(gbhf_ctx* c, int n) {
  if (n > SMALL_DENSE_MAX_N) return false;
  if (c->small_dense < 0)   // once per context: the device has the shared memory and the clusters
    c->small_dense = sd_runs(c, k_density_small, SD_NBUF - 1) && sd_runs(c, k_inv_sqrt_small, SD_NBUF) &&
                     sd_runs(c, k_diis_error_small, SD_NBUF);
  return c->small_dense == 1;
}

gbhf_status density_small(gbhf_ctx* c, int n, int ne, const double* d_F, const double* d_X, double* d_D, double* d_rec) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sd_config(c, n, SD_NBUF - 1, sd_cluster(n), cfg, attr);
  GBHF_CUDA(c, cudaLaunchKernelEx(&cfg, k_density_small, n, ne, 200, 1e-13, d_F, d_X, d_D, d_rec));
  count_launch(c);
  return GBHF_OK;
}

gbhf_status inv_sqrt_small(gbhf_ctx* c, int n, const double* d_S, double* d_X, double* d_out) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sd_config(c, n, SD_NBUF, sd_cluster(n), cfg, attr);
  GBHF_CUDA(c, cudaLaunchKernelEx(&cfg, k_inv_sqrt_small, n, d_S, d_X, d_out));
  count_launch(c);
  return GBHF_OK;
}

gbhf_status diis_error_small(gbhf_ctx* c, int n, const double* d_F, const double* d_S, const double* d_D,
                             const double* d_X, double* d_e) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  sd_config(c, n, SD_NBUF, sd_cluster(n), cfg, attr);
  GBHF_CUDA(c, cudaLaunchKernelEx(&cfg, k_diis_error_small, n, d_F, d_S, d_D, d_X, d_e));
  count_launch(c);
  return GBHF_OK;
}

}  // namespace gbhf
