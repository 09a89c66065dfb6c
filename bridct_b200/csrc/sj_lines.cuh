// Line operations of the plain (Shao-Johnson, FP32 CUDA-core) form.
//
// A "line" is one row or one column of an h x w array.  Three line operations exist, one per reference
// mode (include/bridct.h:24-28):
//   FWD: y = Q x        orthonormal DCT-II      (reference: col_fN then x norm, rect.c:8-15)
//   INV: y = Q^T x      orthonormal DCT-III     (x norm then col_tN)
//   RT : y = Q^T Q x    normalized round trip   (col_fN, x corr, col_tN)
// The 2D transform is a column pass then a row pass; the per-axis factors of the reference's
// normalization table (src/plan.c:92-107, norm[r,c] = s_h(r) s_w(c)) are separable, so each pass
// folds its own factor into its line operation instead of reading an h*w table.
//
// Here: lines that one thread owns whole in registers, scalar (the generated straight-line programs of
// sj_generated.cuh).  Two lines per thread, and lines split over several threads: sj_split.cuh.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "sj_generated.cuh"

namespace bridct {

enum LineMode { LM_FWD = 0, LM_INV = 1, LM_RT = 2 };

// Programmatic dependent launch: the plain kernels are launched with programmatic stream
// serialization, so a kernel's CTAs may be scheduled while the previous kernel in the stream is
// still finishing.  griddep_wait() blocks until every prerequisite grid has completed and its
// memory is visible; each kernel calls it before its first global access, so results are exactly
// those of a serialized launch (without a prerequisite it returns at once).  griddep_trigger()
// lets the next kernel's CTAs be scheduled once every CTA of this one has reached it.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <int N> struct RegLine;
#define BRIDCT_REGLINE(N)                                                                  \
  template <> struct RegLine<N> {                                                          \
    static __device__ __forceinline__ void fwd(float (&v)[N]) { sj_line_fwd_##N(v); }      \
    static __device__ __forceinline__ void inv(float (&v)[N]) { sj_line_inv_##N(v); }      \
    static __device__ __forceinline__ void rt(float (&v)[N]) { sj_line_rt_##N(v); }        \
  };
BRIDCT_REGLINE(8)
BRIDCT_REGLINE(128)
#undef BRIDCT_REGLINE

template <int N, int MODE>
__device__ __forceinline__ void reg_line_apply(float (&v)[N]) {
  if (MODE == LM_FWD) RegLine<N>::fwd(v);
  else if (MODE == LM_INV) RegLine<N>::inv(v);
  else RegLine<N>::rt(v);
}

// One thread, one line: load, transform, store (shared memory, element stride es).
template <int N, int MODE>
__device__ __forceinline__ void reg_line(float* line, int es) {
  float v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = line[i * es];
  reg_line_apply<N, MODE>(v);
#pragma unroll
  for (int i = 0; i < N; ++i) line[i * es] = v[i];
}

}  // namespace bridct
