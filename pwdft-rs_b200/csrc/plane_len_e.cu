// Two-stage passes of the lengths 81 to 120.
#include "plane_kernels.cuh"

namespace pwgpu {
PW_PAIRS_E(PW_PLANE_LEN)
}  // namespace pwgpu
