// Explicit instantiation of the spread kernels for float32 meshes (split for parallel compilation).
#include "fd3_mesh_impl.cuh"

namespace fd3 {
template int launch_spread<float>(const MeshGeom&, int, const double*, const int*, const int*, const MeshRecords&, float*,
                               cudaStream_t);
}  // namespace fd3
