// Dispatch of the single-CTA (y, z) plane transforms on the plane's sizes.
#include "fd3_internal.h"

namespace fd3 {

template <typename T, int NY>
int launch_plane_ny(bool inverse, int nz, int nplanes, const void* in, void* out, cudaStream_t s);

static bool plane_length(int n) { return n == 16 || n == 32 || n == 64 || n == 128 || n == 256; }

bool plane_applies(const MeshGeom& mg, bool is_double) {
  return plane_length(mg.n[1]) && plane_length(mg.n[2]) && mg.n[1] * mg.n[2] <= (is_double ? 16384 : 32768);
}

int launch_plane(const MeshGeom& mg, bool is_double, bool inverse, int nchannels, const void* in, void* out,
                 cudaStream_t s) {
  const long long planes = (long long)nchannels * mg.n[0];
  if (!plane_applies(mg, is_double) || planes > (1LL << 30)) {
    set_error("fft", "the single-CTA plane transforms do not apply to this mesh");
    return FD3_EINVAL;
  }
#define FD3_PLANE(NY)                                                                        \
  case NY:                                                                                   \
    return is_double ? launch_plane_ny<double, NY>(inverse, mg.n[2], (int)planes, in, out, s) \
                     : launch_plane_ny<float, NY>(inverse, mg.n[2], (int)planes, in, out, s);
  switch (mg.n[1]) {
    FD3_PLANE(16)
    FD3_PLANE(32)
    FD3_PLANE(64)
    FD3_PLANE(128)
    FD3_PLANE(256)
  }
#undef FD3_PLANE
  return FD3_EINVAL;
}

}  // namespace fd3
