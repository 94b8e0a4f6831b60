// FP32 kernel instantiations, 19 directions.
#define LBX_KERNEL_TU
#include "lbx_kernels.cuh"

namespace lbx {
LBX_INSTANTIATE(19, float)
}  // namespace lbx
