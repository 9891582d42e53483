// float64 scaling form of the one-read dense Sinkhorn (fused_impl.cuh).
#include "fused_impl.cuh"

namespace otg {
template <> int fu_launch_scal<double>(FusedArgs<double>& A, const FuPlan& f, cudaStream_t st) {
  return f.res ? fu_start_resident<double, FU_SCAL>(A, f, st) : fu_start_streamed<double, FU_SCAL>(A, f, st);
}
}  // namespace otg
