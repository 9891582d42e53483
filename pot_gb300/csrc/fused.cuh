// Dense Sinkhorn that reads the cost once per iteration: host interface.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include "../../include/pot_gb300.h"

namespace otg {

// Where a launch of the one-read solver keeps its state (all in the caller's
// workspace; the caller clears the history, `info` and `bar`).
struct FusedState {
  void *u0, *u1, *v0, *v1, *rowc;  // state vectors, rowc: per-row constant (log2 a or 1/a)
  void* fref;                      // absorbed row potentials (float64 log form)
  void* space;                     // fused_bytes() of scratch
  double* hist;
  int* info;
  unsigned* bar;
  uint64_t timeout_ns;
};

// Scratch bytes of the one-read solver for this shape; 0: it does not take it.
size_t fused_bytes(int dtype, int64_t n, int64_t m, int requested_grid);

// Launches the one-read solver when it takes the problem (method, shape,
// alignment); returns OTG_ERR_UNSUPPORTED when it does not.
int fused_launch(const OtgDenseProblem* p, const FusedState& fs, cudaStream_t st);

// Whether that launch (scaling form) makes K = exp(-M/reg) by itself once: in
// shared memory, or with the copy into whole-vector rows.
bool fused_holds_gibbs(const OtgDenseProblem* p);

// Per-type parts (fused_f32.cu, fused_f64.cu).
int fused_launch_f32(const OtgDenseProblem* p, const FusedState& fs, cudaStream_t st);
int fused_launch_f64(const OtgDenseProblem* p, const FusedState& fs, cudaStream_t st);
size_t fused_bytes_f32(int64_t n, int64_t m, int requested_grid);
size_t fused_bytes_f64(int64_t n, int64_t m, int requested_grid);
bool fused_holds_gibbs_f32(const OtgDenseProblem* p);
bool fused_holds_gibbs_f64(const OtgDenseProblem* p);

inline size_t fused_bytes(int dtype, int64_t n, int64_t m, int requested_grid) {
  return dtype == OTG_F64 ? fused_bytes_f64(n, m, requested_grid) : fused_bytes_f32(n, m, requested_grid);
}
inline int fused_launch(const OtgDenseProblem* p, const FusedState& fs, cudaStream_t st) {
  return p->dtype == OTG_F64 ? fused_launch_f64(p, fs, st) : fused_launch_f32(p, fs, st);
}
inline bool fused_holds_gibbs(const OtgDenseProblem* p) {
  return p->dtype == OTG_F64 ? fused_holds_gibbs_f64(p) : fused_holds_gibbs_f32(p);
}

}  // namespace otg
