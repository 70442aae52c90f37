// Per-quartet screening of the direct builds, done by the warp that owns a task
// before any quartet of it is evaluated.
//
// A task lists the kets of one bra pair that pass the Schwarz bound; most of
// them drop by the density (a quartet touches six density blocks, and only near
// pairs hold large ones).  Evaluated lane by lane as they came, 16 of 32 lanes of
// an average (ps|ss) task of (H2O)40/6-31G did work, and each test gathered the
// density elements themselves (12 for (ps|ss), 54 for (pp|pp)).  Here the warp
// scans the task's kets 32 at a time against the largest |D| of every shell
// block (four gathers from two rows that stay in L1, the rest coalesced),
// queues the survivors in shared memory and evaluates them in full batches.
// Magnitudes are rounded up to FP32 and the threshold down, so a quartet that
// the FP64 test would keep is kept; a density above the FP32 range has infinite
// maxima, and where those meet a zero block (NaN) the quartet is kept as well.
#pragma once
#include "gbhf_internal.h"
#include "warp_queue.cuh"

namespace gbhf {

struct QuartetScreen {
  const int4* pinfo;        // per pair: shells A, B and their first functions within the molecule
  const float* Qf;          // Schwarz bound of each pair
  const float* pbf;         // largest |D_ab| of each pair's block
  const float* Ds;          // largest |D| of each shell block, stacked ns_m x ns_m
  const int* ms0;           // first shell of each molecule (nmol + 1)
  const long long* soff;    // offset of the molecule's block in Ds
  float thr;
};

// Without maxima of the current density (small systems) every quartet passes: Ds is null.
inline QuartetScreen quartet_screen(const gbhf_ctx* c, double thr) {
  return {c->pairs.pinfo.p, c->pairs.Qf.p, c->tasks.pbf.p,  c->tasks.screened ? c->tasks.Ds.p : nullptr,
          c->tasks.ms0.p,   c->tasks.soff.p, (float)(thr * (1.0 - 3e-7))};
}

// The gradient leaves out the quartets with all four shells on one atom: their four
// derivatives add up to zero there (translational invariance), in floating point to the
// rounding of terms that are the largest of all for steep shells.
struct OneCentre {
  int at;   // the atom of both bra shells, else -1
  __device__ __forceinline__ OneCentre(const int* __restrict__ shell_atom, int4 pab) {
    const int a = shell_atom[pab.x];
    at = a == shell_atom[pab.y] ? a : -1;
  }
  __device__ __forceinline__ bool holds(const int* __restrict__ shell_atom, int4 pcd) const {
    return at >= 0 && shell_atom[pcd.x] == at && shell_atom[pcd.y] == at;
  }
};

// The bra's part of the bound.
struct BraScreen {
  float q, dab;
  const float *ra, *rb;   // rows of Ds, indexed by global shell
  __device__ __forceinline__ BraScreen(const QuartetScreen& s, int ib, int4 pab, int mol) {
    ra = rb = nullptr;
    q = dab = 0.0f;
    if (!s.Ds) return;
    const int s0 = s.ms0[mol], ns = s.ms0[mol + 1] - s0;
    const float* d = s.Ds + s.soff[mol] - s0;
    ra = d + (long long)(pab.x - s0) * ns;
    rb = d + (long long)(pab.y - s0) * ns;
    q = s.Qf[ib];
    dab = s.pbf[ib];
  }
  // Q_ab Q_cd max |D| over ab, cd, ac, ad, bc, bd against the threshold
  __device__ __forceinline__ bool jk_pass(const QuartetScreen& s, int jk) const {
    if (!s.Ds) return true;
    const int4 p = s.pinfo[jk];
    const float d = fmaxf(fmaxf(fmaxf(ra[p.x], ra[p.y]), fmaxf(rb[p.x], rb[p.y])), fmaxf(dab, s.pbf[jk]));
    return !(q * s.Qf[jk] * d < s.thr);
  }
  // Q_ab Q_cd times a bound of |Gamma| = |jcoef D_ab D_cd - (D_ac D_bd + D_ad D_bc) / 4|
  __device__ __forceinline__ bool gamma_pass(const QuartetScreen& s, int jk, float jcoef, const OneCentre& one,
                                             const int* __restrict__ shell_atom) const {
    const int4 p = s.pinfo[jk];
    if (one.holds(shell_atom, p)) return false;
    if (!s.Ds) return true;
    const float g = fabsf(jcoef) * dab * s.pbf[jk] + 0.25f * (ra[p.x] * rb[p.y] + ra[p.y] * rb[p.x]);
    return !(q * s.Qf[jk] * g * 1.000001f < s.thr);
  }
};

}  // namespace gbhf
