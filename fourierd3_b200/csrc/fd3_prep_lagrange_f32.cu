// Call preparation with Lagrange weights for float32 meshes (split for parallel compilation).
#include "fd3_prep.cuh"

namespace fd3 {
template int launch_prep<float, true>(const PrepDev&, cudaStream_t);
}  // namespace fd3
