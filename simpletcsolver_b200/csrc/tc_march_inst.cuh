// Definitions behind tc_march_launch.cuh, for the instantiating files.
#pragma once
#include "tc_march_f32.cuh"
#include "tc_march_launch.cuh"

namespace tcgpu {
namespace march {

template <int NW, int PAIRS, int NG, int IMPL, class T, bool TILE>
void launch_one(Args<T> A, const double * dtp, cudaStream_t st) {
  using L = Layout<NW, PAIRS, NG, T>;
  const long long columns = (long long)((A.g.ny + L::JT - 1) / L::JT) * (TILE ? (A.g.nx + L::NT - 1) / L::NT : 1);
  A.KC = march_planes(columns, A.g.nz, 1);
  auto kernel = predict_kernel<NW, PAIRS, NG, IMPL, T, TILE>;
  // the limit belongs to the current CUDA context, so it is set with every launch (steps
  // replay a graph: twice per device context); a failure stays the thread's last error,
  // which the capture of a step and the end of each entry point report
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES) != cudaSuccess) return;
  kernel<<<(unsigned)(columns * (A.g.nz / A.KC)), L::THREADS, L::BYTES, st>>>(A, dtp);
}

// warps per line by its length, line pairs, and 1 or 2 groups of field warps per line:
// 4, 8 or 12 field warps, the fastest of the splits measured at each length
#ifndef TC_MARCH_INSTANCES
#define TC_MARCH_INSTANCES(X) X(1, 4, 1) X(2, 4, 1) X(3, 2, 2) X(4, 2, 1) X(6, 1, 2) X(8, 1, 1)
#endif

template <int IMPL, class T>
void launch(Args<T> A, bool tiles, const double * dtp, cudaStream_t st) {
  if constexpr (IMPL < 0 || (IMPL == 1 && sizeof(T) == 8))
    if (tiles) return launch_one<8, 1, 1, IMPL, T, true>(A, dtp, st);
  switch (sizeof(T) == 8 ? predict_warps(A.g.nx) : predict_warps32(A.g.nx)) {
#define X(NW, PAIRS, NG)                                                   \
  case NW:                                                                 \
    if constexpr (sizeof(T) == 8 || (NW & (NW - 1)) == 0) /* predict_warps32 */ \
      return launch_one<NW, PAIRS, NG, IMPL, T, false>(A, dtp, st);          \
    else                                                                     \
      return;
    TC_MARCH_INSTANCES(X)
#undef X
  }
}
}  // namespace march
}  // namespace tcgpu
