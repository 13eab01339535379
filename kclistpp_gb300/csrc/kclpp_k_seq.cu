// kclpp_k_seq.cu -- instantiates the MODE_SEQ clique kernels up to k = 6 (one
// translation unit per mode so that the library builds in parallel; the Seq
// kernels of k = 7, 8, whose recursions take longest to compile, have their own).
#include "kclpp_kernels.cuh"

namespace kclpp {
cudaError_t launch_seq_deep(int k, const TierLaunch &t, dev::PassArgs a, cudaStream_t st);

cudaError_t launch_seq(int k, const TierLaunch &t, dev::PassArgs a, cudaStream_t st) {
  return k <= 6 ? launch_mode<dev::MODE_SEQ, 3, 6>(k, t, a, st) : launch_seq_deep(k, t, a, st);
}
}  // namespace kclpp
