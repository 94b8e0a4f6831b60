// FP32 kernel instantiations, 9 directions.
#define LBX_KERNEL_TU
#include "lbx_kernels.cuh"

namespace lbx {
LBX_INSTANTIATE(9, float)
}  // namespace lbx
