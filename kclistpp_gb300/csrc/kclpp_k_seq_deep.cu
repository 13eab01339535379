// kclpp_k_seq_deep.cu -- instantiates the MODE_SEQ clique kernels of k = 7, 8.
#include "kclpp_kernels.cuh"

namespace kclpp {
cudaError_t launch_seq_deep(int k, const TierLaunch &t, dev::PassArgs a, cudaStream_t st) {
  return launch_mode<dev::MODE_SEQ, 7, 8>(k, t, a, st);
}
}  // namespace kclpp
