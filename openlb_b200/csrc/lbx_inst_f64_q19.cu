// FP64 kernel instantiations, 19 directions (the unit is built like every other without FMA
// contraction, so the operation sequence of lbx_collision.cuh rounds exactly like the reference's
// CPU build).
#define LBX_KERNEL_TU
#include "lbx_kernels.cuh"

namespace lbx {
LBX_INSTANTIATE(19, double)
}  // namespace lbx
