#include "tc_march_inst.cuh"

namespace tcgpu {
namespace march {
template void launch<0, double>(Args<double>, bool, const double *, cudaStream_t);
}  // namespace march
}  // namespace tcgpu
