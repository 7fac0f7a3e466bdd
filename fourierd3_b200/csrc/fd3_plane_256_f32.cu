#include "fd3_plane.cuh"
namespace fd3 {
template int launch_plane_ny<float, 256>(bool, int, int, const void*, void*, cudaStream_t);
}
