// float64 log form of the one-read dense Sinkhorn (fused_impl.cuh) and its host side.
#include "fused_impl.cuh"

namespace otg {
template <> int fu_launch_log<double>(FusedArgs<double>& A, const FuPlan& f, bool abs, cudaStream_t st) {
  return abs ? fu_start_resident<double, FU_ABS>(A, f, st) : f.res ? OTG_ERR_UNSUPPORTED : fu_start_streamed<double, FU_LOG>(A, f, st);
}

int fused_launch_f64(const OtgDenseProblem* p, const FusedState& fs, cudaStream_t st) { return fused_run<double>(p, fs, st); }
size_t fused_bytes_f64(int64_t n, int64_t m, int requested_grid) { return fused_run_bytes<double>(n, m, requested_grid); }
bool fused_holds_gibbs_f64(const OtgDenseProblem* p) { return fused_run_holds_gibbs<double>(p); }
}  // namespace otg
