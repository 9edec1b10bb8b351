// Two-stage passes of the lengths 24 to 32.
#include "plane_kernels.cuh"

namespace pwgpu {
PW_PAIRS_B(PW_PLANE_LEN)
}  // namespace pwgpu
