#include "tc_march_inst.cuh"

namespace tcgpu {
namespace march {
template void launch<0, float>(Args<float>, bool, const double *, cudaStream_t);
template void launch<-1, float>(Args<float>, bool, const double *, cudaStream_t);
}  // namespace march
}  // namespace tcgpu
