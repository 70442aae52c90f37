// The two-float instances of the J/K kernel.
#include "jk_kern.cuh"

namespace gbhf {

gbhf_status launch_jk_ff(gbhf_ctx* c, cudaStream_t strm, int k, double* G, int nt, int wj) {
  return launch_combo<ff>(c, strm, k, TIER_FF, c->dff.p, G, nt, wj);
}

}  // namespace gbhf
