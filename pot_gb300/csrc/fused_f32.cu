// float32 log form of the one-read dense Sinkhorn (fused_impl.cuh) and its host side.
#include "fused_impl.cuh"

namespace otg {
template <> int fu_launch_log<float>(FusedArgs<float>& A, const FuPlan& f, bool abs, cudaStream_t st) {
  (void)abs;
  return f.res ? fu_start_resident<float, FU_LOG>(A, f, st) : fu_start_streamed<float, FU_LOG>(A, f, st);
}

int fused_launch_f32(const OtgDenseProblem* p, const FusedState& fs, cudaStream_t st) { return fused_run<float>(p, fs, st); }
size_t fused_bytes_f32(int64_t n, int64_t m, int requested_grid) { return fused_run_bytes<float>(n, m, requested_grid); }
bool fused_holds_gibbs_f32(const OtgDenseProblem* p) { return fused_run_holds_gibbs<float>(p); }
}  // namespace otg
