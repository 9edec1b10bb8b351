// Two-stage passes of the lengths 54 to 80.
#include "plane_kernels.cuh"

namespace pwgpu {
PW_PAIRS_D(PW_PLANE_LEN)
}  // namespace pwgpu
