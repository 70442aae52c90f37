// The two-float instances of the two-electron gradient kernel.
#include "grad_kern.cuh"

namespace gbhf {

gbhf_status launch_grad_ff(gbhf_ctx* c, cudaStream_t strm, int k, double* grad, int nt) {
  return launch_grad_combo<ff>(c, strm, k, TIER_FF, c->dff.p, grad, nt);
}

}  // namespace gbhf
