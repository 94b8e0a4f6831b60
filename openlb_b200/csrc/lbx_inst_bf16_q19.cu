// bfloat16 deviation storage (float collision) instantiations, 19 directions.
#define LBX_KERNEL_TU
#include "lbx_kernels.cuh"

namespace lbx {
LBX_INSTANTIATE(19, __nv_bfloat16)
}  // namespace lbx
