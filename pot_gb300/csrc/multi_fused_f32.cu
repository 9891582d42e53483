// float32 instances of the one-read batch kernel (multi_fused.cuh).
#include <cmath>
#include "multi_common.cuh"
#include "multi_fused.cuh"
#include "launch.cuh"

namespace otg {

bool multi_fused_plan(int dtype, int max_ldm, size_t smem_max, MultiFusedPlan& f) {
  const int es = dtype == OTG_F64 ? 8 : 4, W = 16 / es;
  const int V = (max_ldm + W - 1) / W;
  f.NK = V <= 64 ? 2 : V <= 128 ? 4 : V <= 256 ? 8 : 16;
  f.G = 1;
  while (f.G < FU_WARPS && f.G * 32 * f.NK < V) f.G *= 2;
  if (f.G * 32 * f.NK < V) return false;
  const int NG = FU_WARPS / f.G;
  f.mp = f.NK * f.G * 32 * W;
  const size_t fixed = (size_t)NG * f.mp * es + 12 * 1024;  // v, and the kernel's static arrays
  const size_t chunk = (size_t)NG * ((size_t)(16 / f.NK) * f.mp * es + 16);  // a batch, and its barrier
  f.NC = MF_RING;
  while (f.NC > 2 && fixed + f.NC * chunk > smem_max) --f.NC;
  f.smem = (size_t)NG * f.mp * es + f.NC * chunk;
  return fixed + f.NC * chunk <= smem_max;
}

namespace {
template <bool LOGF, int NK>
int start(const MultiArgs<float>& A, int grid, size_t smem, int32_t* leaving, cudaStream_t st) {
  const void* k = (const void*)multi_fused_kernel<float, LOGF, NK>;
  if (!allow_smem(k, smem)) return OTG_ERR_CUDA;
  MultiArgs<float> a = A;
  void* args[] = {&a, &leaving};
  return cudaLaunchCooperativeKernel(k, dim3(grid), dim3(MT_THREADS), args, smem, st) == cudaSuccess ? OTG_OK : OTG_ERR_CUDA;
}
template <bool LOGF>
int start_nk(const MultiArgs<float>& A, int NK, int grid, size_t smem, int32_t* leaving, cudaStream_t st) {
  switch (NK) {
    case 2: return start<LOGF, 2>(A, grid, smem, leaving, st);
    case 4: return start<LOGF, 4>(A, grid, smem, leaving, st);
    case 8: return start<LOGF, 8>(A, grid, smem, leaving, st);
    default: return start<LOGF, 16>(A, grid, smem, leaving, st);
  }
}
}  // namespace

int multi_fused_launch(const MultiArgs<float>& A, bool logf, int NK, int grid, size_t smem, int32_t* leaving, cudaStream_t st) {
  return logf ? start_nk<true>(A, NK, grid, smem, leaving, st) : start_nk<false>(A, NK, grid, smem, leaving, st);
}
}  // namespace otg
