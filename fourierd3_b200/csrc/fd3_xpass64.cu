// Dispatch of the float64 x-pass on the x length, and the pencil widths of both precisions' x-passes.
#include "fd3_xpass64.cuh"

namespace fd3 {

extern template int launch_x64<4, 4>(const X64Args&, X64Shape);
extern template int launch_x64<4, 8>(const X64Args&, X64Shape);
extern template int launch_x64<8, 8>(const X64Args&, X64Shape);
extern template int launch_x64<8, 16>(const X64Args&, X64Shape);
extern template int launch_x64<16, 16>(const X64Args&, X64Shape);

template <>
int launch_xfilter<double>(const MeshGeom& mg, const CellInfo* ci, const GreenPair* gp, const GreenPairF* gpf,
                           const float4* gtab, const Tables* tab, const float* deconv, int spme, void* spec,
                           double* part, int* n_blocks, cudaStream_t s) {
  (void)gpf;
  (void)gtab;
  const X64Shape sh = x64_shape(mg);
  if (sh.LKZ < 0) return FD3_EINVAL;
  const X64Args a{&mg, ci, gp, tab, deconv, spme, reinterpret_cast<double2*>(spec), part, n_blocks, s};
  switch (mg.n[0]) {
    case 16: return launch_x64<4, 4>(a, sh);
    case 32: return launch_x64<4, 8>(a, sh);
    case 64: return launch_x64<8, 8>(a, sh);
    case 128: return launch_x64<8, 16>(a, sh);
    case 256: return launch_x64<16, 16>(a, sh);
    default: return FD3_EINVAL;
  }
}

bool xpass64_twice_per_sm(const MeshGeom& mg) { return x64_shape(mg).two != 0; }

int xfilter_pencil(const MeshGeom& mg, int is_double) {
  if (!is_double) return xfilter_kz<float>(mg);
  const X64Shape sh = x64_shape(mg);
  return sh.LKZ < 0 ? 0 : 1 << sh.LKZ;
}

}  // namespace fd3
