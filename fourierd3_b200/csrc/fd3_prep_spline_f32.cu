// Call preparation with B-spline weights for float32 meshes (split for parallel compilation).
#include "fd3_prep.cuh"

namespace fd3 {
template int launch_prep<float, false>(const PrepDev&, cudaStream_t);
}  // namespace fd3
