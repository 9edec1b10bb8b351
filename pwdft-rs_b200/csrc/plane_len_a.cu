// Two-stage passes of the lengths 12 to 20.
#include "plane_kernels.cuh"

namespace pwgpu {
PW_PAIRS_A(PW_PLANE_LEN)
}  // namespace pwgpu
