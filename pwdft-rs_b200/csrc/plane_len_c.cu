// Two-stage passes of the lengths 36 to 50.
#include "plane_kernels.cuh"

namespace pwgpu {
PW_PAIRS_C(PW_PLANE_LEN)
}  // namespace pwgpu
