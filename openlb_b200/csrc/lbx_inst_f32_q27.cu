// FP32 kernel instantiations, 27 directions.
#define LBX_KERNEL_TU
#include "lbx_kernels.cuh"

namespace lbx {
LBX_INSTANTIATE(27, float)
}  // namespace lbx
