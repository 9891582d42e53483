// float32 scaling form of the one-read dense Sinkhorn (fused_impl.cuh).
#include "fused_impl.cuh"

namespace otg {
template <> int fu_launch_scal<float>(FusedArgs<float>& A, const FuPlan& f, cudaStream_t st) {
  return f.res ? fu_start_resident<float, FU_SCAL>(A, f, st) : fu_start_streamed<float, FU_SCAL>(A, f, st);
}
}  // namespace otg
