// binary16 deviation storage (float collision) instantiations, 9 directions.
#define LBX_KERNEL_TU
#include "lbx_kernels.cuh"

namespace lbx {
LBX_INSTANTIATE(9, __half)
}  // namespace lbx
