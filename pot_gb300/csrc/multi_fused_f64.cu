// float64 instances of the one-read batch kernel (multi_fused.cuh).
#include <cmath>
#include "multi_common.cuh"
#include "multi_fused.cuh"
#include "launch.cuh"

namespace otg {

namespace {
template <bool LOGF, int NK>
int start(const MultiArgs<double>& A, int grid, size_t smem, int32_t* leaving, cudaStream_t st) {
  const void* k = (const void*)multi_fused_kernel<double, LOGF, NK>;
  if (!allow_smem(k, smem)) return OTG_ERR_CUDA;
  MultiArgs<double> a = A;
  void* args[] = {&a, &leaving};
  return cudaLaunchCooperativeKernel(k, dim3(grid), dim3(MT_THREADS), args, smem, st) == cudaSuccess ? OTG_OK : OTG_ERR_CUDA;
}
template <bool LOGF>
int start_nk(const MultiArgs<double>& A, int NK, int grid, size_t smem, int32_t* leaving, cudaStream_t st) {
  switch (NK) {
    case 2: return start<LOGF, 2>(A, grid, smem, leaving, st);
    case 4: return start<LOGF, 4>(A, grid, smem, leaving, st);
    case 8: return start<LOGF, 8>(A, grid, smem, leaving, st);
    default: return start<LOGF, 16>(A, grid, smem, leaving, st);
  }
}
}  // namespace

int multi_fused_launch(const MultiArgs<double>& A, bool logf, int NK, int grid, size_t smem, int32_t* leaving, cudaStream_t st) {
  return logf ? start_nk<true>(A, NK, grid, smem, leaving, st) : start_nk<false>(A, NK, grid, smem, leaving, st);
}
}  // namespace otg
