// Launch of the marching predict kernel for one implicit mask;
// declared here, instantiated in tc_march_inst*.cu (the instances compile in parallel).
#pragma once
#include "tc_march.cuh"

namespace tcgpu {
namespace march {

template <int IMPL, class T>
void launch(Args<T> A, bool tiles, const double * dtp, cudaStream_t st);

}  // namespace march
}  // namespace tcgpu
