// binary16 deviation storage (float collision) instantiations, 27 directions.
#define LBX_KERNEL_TU
#include "lbx_kernels.cuh"

namespace lbx {
LBX_INSTANTIATE(27, __half)
}  // namespace lbx
