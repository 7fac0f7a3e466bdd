// (y, z) plane transforms of the real mesh, one pass over it each way, for planes that fit one CTA's
// shared memory (float up to 256 x 128 points, double up to 128 x 128); larger float planes take the
// cluster kernels of fd3_yzfft.cu, the rest cuFFT. (the reference's torch.fft.rfftn / irfftn over the
// mesh, kspace_filter_d3.py:55-68, of which the x axis is transformed by the x-pass)
//
// Layouts as cuFFT's batched 2D transforms leave them: plane p = (channel, x) of the real mesh at
// rho + p NY NZ, of the half spectrum at spec + p NY (NZ / 2 + 1). Unnormalised.
//
// A row of NZ reals is N = NZ / 2 complex values z[m] = x[2m] + i x[2m+1]; its transform is an N-point
// FFT (A1 x A2 register DFTs) and the real/half-complex split. kz = 0 and kz = N come out real and
// travel as one packed column, so a plane is NY x N complex values in shared memory throughout.
//   forward: rows straight from global memory into the first register pass; second pass and split
//     (the partner Z[N - k] by a shuffle); y FFTs (B1 x B2) of the N columns, the second pass straight
//     from registers to the spectrum.
//   inverse: the mirror image.
// That is three shared-memory round trips per value (cuFFT's 2D transform is two kernels and an
// extra trip through L2 or HBM each way). The row layout of the z passes pads every k1 group by one
// value, and rows are an odd number of values apart, so neither z pass collides on banks; the y passes
// walk columns, lanes on consecutive values. Against cuFFT's 2D transforms, 8 channels, forward and inverse:
// 64^3 float 17.4 and 17.4 -> 12.3 and 12.3 us, double 25.8 and 27.6 -> 19.7 and 18.4; 128^3 float 67 and 62 -> 55
// and 57 (2.5 TB/s; instruction issue and shared-memory latency), double 130 and 126 -> 98 and 109;
// 256 x 256 x 128 float 245 and 236 -> 211 and 206.
#pragma once
#include "fd3_xfilter.cuh"

namespace fd3 {

// N = first x second register DFTs
template <int N>
struct Split2 {
  static constexpr int a = N <= 16 ? 4 : N <= 128 ? 8 : 16;
  static constexpr int b = N / a;
};

template <typename T, int NY, int NZ>
struct PlaneCfg {
  static constexpr int N = NZ / 2;
  static constexpr int A1 = Split2<N>::a, A2 = Split2<N>::b;
  static constexpr int B1 = Split2<NY>::a, B2 = Split2<NY>::b;
  static constexpr int GRP = A2 + 1;                       // padded k1 group of the z passes
  static constexpr int LD = A1 * GRP + ((A1 * GRP) % 2 == 0 ? 1 : 0);   // row pitch, odd
  static constexpr int kItems = NY * N / 16;
  static constexpr int kThreads = kItems >= 512 ? 512 : kItems >= 128 ? 256 : 128;
  static constexpr int TWN = 256;                          // twiddle table exp(-2 pi i j / TWN)
  static constexpr size_t kSmem = ((size_t)NY * LD + TWN) * 2 * sizeof(T);
  // CTAs per SM: what shared memory and 64 (float) or 112 (double) registers a thread allow
  static constexpr int kBySmem = (int)(220 * 1024 / kSmem), kByRegs = 65536 / (kThreads * (sizeof(T) == 4 ? 64 : 112));
  static constexpr int kMinBlocks = kBySmem < kByRegs ? (kBySmem < 1 ? 1 : kBySmem) : (kByRegs < 1 ? 1 : kByRegs);
};

// exp(-2 pi i j / N) from the table, conjugated for the inverse
template <typename T, int N, int SIGN>
__device__ __forceinline__ typename Cplx<T>::type plane_tw(const typename Cplx<T>::type* tw, int j) {
  auto w = tw[(j * (256 / N)) & 255];
  if (SIGN > 0) w.y = -w.y;
  return w;
}
template <typename C2>
__device__ __forceinline__ C2 plane_cmul(C2 a, C2 w) {
  return C2{a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x};
}

template <typename T>
__device__ __forceinline__ void plane_twiddles(typename Cplx<T>::type* tw) {
  for (int j = threadIdx.x; j < 256; j += blockDim.x) {
    double sn, cs;
    sincospi(-2.0 * j / 256.0, &sn, &cs);
    tw[j] = typename Cplx<T>::type{(T)cs, (T)sn};
  }
}

// Every warp of a pass is full or idle (NY A1 and NY A2 are multiples of 32), so its shuffles and warp
// barriers take whole warps.
template <typename T, int NY, int NZ>
__global__ void __launch_bounds__(PlaneCfg<T, NY, NZ>::kThreads, PlaneCfg<T, NY, NZ>::kMinBlocks)
    k_plane_forward(const T* __restrict__ rho, typename Cplx<T>::type* __restrict__ spec, int nplanes) {
  using C2 = typename Cplx<T>::type;
  using Cf = PlaneCfg<T, NY, NZ>;
  constexpr int N = Cf::N, A1 = Cf::A1, A2 = Cf::A2, B1 = Cf::B1, B2 = Cf::B2, LD = Cf::LD, GRP = Cf::GRP;
  constexpr int NT = Cf::kThreads, NZH = N + 1;
  extern __shared__ __align__(16) unsigned char pl_raw[];
  C2* tw = reinterpret_cast<C2*>(pl_raw);
  C2* B = tw + Cf::TWN;
  plane_twiddles<T>(tw);
  for (int p = blockIdx.x; p < nplanes; p += gridDim.x) {
    const C2* in = reinterpret_cast<const C2*>(rho + (size_t)p * NY * NZ);
    C2* out = spec + (size_t)p * NY * NZH;
    __syncthreads();   // twiddles written; the previous plane has been read
    // z pass 1: item (y, n2), lanes over n2
#pragma unroll 1
    for (int it = threadIdx.x; it < NY * A2; it += NT) {
      const int n2 = it % A2, y = it / A2;
      T re[A1], im[A1];
#pragma unroll
      for (int n1 = 0; n1 < A1; ++n1) {
        const C2 v = in[(size_t)y * N + A2 * n1 + n2];
        re[n1] = v.x;
        im[n1] = v.y;
      }
      dft_reg<T, A1, -1>(re, im);
      C2* row = B + y * LD + n2;
#pragma unroll
      for (int k1 = 0; k1 < A1; ++k1)
        row[k1 * GRP] = plane_cmul(C2{re[k1], im[k1]}, plane_tw<T, N, -1>(tw, n2 * k1));
    }
    __syncthreads();
    // z pass 2 and split: item (y, k1), the A1 lanes of a row in one warp
#pragma unroll 1
    for (int it = threadIdx.x; it < NY * A1; it += NT) {
      const int k1 = it % A1, y = it / A1;
      C2* row = B + y * LD;
      T re[A2], im[A2];
#pragma unroll
      for (int n2 = 0; n2 < A2; ++n2) {
        const C2 v = row[k1 * GRP + n2];
        re[n2] = v.x;
        im[n2] = v.y;
      }
      __syncwarp();   // the row's values are in registers: its natural order may be written over them
      dft_reg<T, A2, -1>(re, im);
      const int lane = threadIdx.x & 31;
      const int partner = (lane & ~(A1 - 1)) | ((A1 - k1) & (A1 - 1));
#pragma unroll
      for (int k2 = 0; k2 < A2; ++k2) {
        // Z[N - k], k = k1 + A1 k2: the partner's value A2 - 1 - k2, or this lane's (A2 - k2) mod A2
        const T pr = __shfl_sync(0xffffffffu, re[A2 - 1 - k2], partner);
        const T pi = __shfl_sync(0xffffffffu, im[A2 - 1 - k2], partner);
        const T cx = k1 == 0 ? re[(A2 - k2) % A2] : pr;
        const T cy = k1 == 0 ? im[(A2 - k2) % A2] : pi;
        const T ax = re[k2], ay = im[k2];
        const int k = k1 + A1 * k2;
        if (k == 0) {   // X[0] and X[N], both real: the packed column
          row[0] = C2{ax + ay, ax - ay};
        } else {
          // X[k] = ((a + b) - i W_NZ^k (a - b)) / 2 with b = conj(c)
          const C2 w = plane_tw<T, NZ, -1>(tw, k);
          const T sx = ax + cx, sy = ay - cy, dx = ax - cx, dy = ay + cy;
          row[k] = C2{T(0.5) * (sx + w.x * dy + w.y * dx), T(0.5) * (sy - w.x * dx + w.y * dy)};
        }
      }
    }
    __syncthreads();
    // y pass 1: item (n2, c), lanes over the columns; in place
#pragma unroll 1
    for (int it = threadIdx.x; it < N * B2; it += NT) {
      const int c = it % N, n2 = it / N;
      T re[B1], im[B1];
#pragma unroll
      for (int n1 = 0; n1 < B1; ++n1) {
        const C2 v = B[(B2 * n1 + n2) * LD + c];
        re[n1] = v.x;
        im[n1] = v.y;
      }
      dft_reg<T, B1, -1>(re, im);
#pragma unroll
      for (int k1 = 0; k1 < B1; ++k1)
        B[(B2 * k1 + n2) * LD + c] = plane_cmul(C2{re[k1], im[k1]}, plane_tw<T, NY, -1>(tw, n2 * k1));
    }
    __syncthreads();
    // y pass 2: item (k1, c) to the spectrum; the packed column stays here until every ky is known
#pragma unroll 1
    for (int it = threadIdx.x; it < N * B1; it += NT) {
      const int c = it % N, k1 = it / N;
      T re[B2], im[B2];
#pragma unroll
      for (int n2 = 0; n2 < B2; ++n2) {
        const C2 v = B[(B2 * k1 + n2) * LD + c];
        re[n2] = v.x;
        im[n2] = v.y;
      }
      dft_reg<T, B2, -1>(re, im);
#pragma unroll
      for (int k2 = 0; k2 < B2; ++k2) {
        if (c == 0)
          B[(B2 * k1 + k2) * LD] = C2{re[k2], im[k2]};
        else
          out[(size_t)(k1 + B1 * k2) * NZH + c] = C2{re[k2], im[k2]};
      }
    }
    __syncthreads();
    // C = Y0 + i YN with Y0, YN the transforms of real columns:
    // Y0[ky] = (C[ky] + C*[-ky]) / 2, YN[ky] = (C[ky] - C*[-ky]) / (2 i); ky = k1 + B1 k2 at row B2 k1 + k2
    for (int ky = threadIdx.x; ky < NY; ky += NT) {
      const int km = (NY - ky) & (NY - 1);
      const C2 c = B[(B2 * (ky % B1) + ky / B1) * LD], m = B[(B2 * (km % B1) + km / B1) * LD];
      out[(size_t)ky * NZH] = C2{T(0.5) * (c.x + m.x), T(0.5) * (c.y - m.y)};
      out[(size_t)ky * NZH + N] = C2{T(0.5) * (c.y + m.y), T(0.5) * (m.x - c.x)};
    }
  }
}

template <typename T, int NY, int NZ>
__global__ void __launch_bounds__(PlaneCfg<T, NY, NZ>::kThreads, PlaneCfg<T, NY, NZ>::kMinBlocks)
    k_plane_inverse(const typename Cplx<T>::type* __restrict__ spec, T* __restrict__ rho, int nplanes) {
  using C2 = typename Cplx<T>::type;
  using Cf = PlaneCfg<T, NY, NZ>;
  constexpr int N = Cf::N, A1 = Cf::A1, A2 = Cf::A2, B1 = Cf::B1, B2 = Cf::B2, LD = Cf::LD, GRP = Cf::GRP;
  constexpr int NT = Cf::kThreads, NZH = N + 1;
  extern __shared__ __align__(16) unsigned char pl_raw[];
  C2* tw = reinterpret_cast<C2*>(pl_raw);
  C2* B = tw + Cf::TWN;
  plane_twiddles<T>(tw);
  for (int p = blockIdx.x; p < nplanes; p += gridDim.x) {
    const C2* in = spec + (size_t)p * NY * NZH;
    C2* out = reinterpret_cast<C2*>(rho + (size_t)p * NY * NZ);
    __syncthreads();
    // inverse y pass 1 from the spectrum: item (n2, c), lanes over the columns
#pragma unroll 1
    for (int it = threadIdx.x; it < N * B2; it += NT) {
      const int c = it % N, n2 = it / N;
      T re[B1], im[B1];
#pragma unroll
      for (int n1 = 0; n1 < B1; ++n1) {
        const C2* rowp = in + (size_t)(B2 * n1 + n2) * NZH;
        const C2 v = rowp[c];
        re[n1] = v.x;
        im[n1] = v.y;
        if (c == 0) {   // H[ky][0] + i H[ky][N]: one transform gives both real columns
          const C2 h = rowp[N];
          re[n1] -= h.y;
          im[n1] += h.x;
        }
      }
      dft_reg<T, B1, 1>(re, im);
#pragma unroll
      for (int k1 = 0; k1 < B1; ++k1)
        B[(B2 * k1 + n2) * LD + c] = plane_cmul(C2{re[k1], im[k1]}, plane_tw<T, NY, 1>(tw, n2 * k1));
    }
    __syncthreads();
    // inverse y pass 2 in place: row B2 k1 + k2 then holds y = k1 + B1 k2
#pragma unroll 1
    for (int it = threadIdx.x; it < N * B1; it += NT) {
      const int c = it % N, k1 = it / N;
      T re[B2], im[B2];
#pragma unroll
      for (int n2 = 0; n2 < B2; ++n2) {
        const C2 v = B[(B2 * k1 + n2) * LD + c];
        re[n2] = v.x;
        im[n2] = v.y;
      }
      dft_reg<T, B2, 1>(re, im);
#pragma unroll
      for (int k2 = 0; k2 < B2; ++k2) B[(B2 * k1 + k2) * LD + c] = C2{re[k2], im[k2]};
    }
    __syncthreads();
    // pack Z[k] = (X[k] + X*[N-k]) + i W_NZ^-k (X[k] - X*[N-k]) and inverse z pass 1: item (row, n2), the
    // A2 lanes of a row in one warp
#pragma unroll 1
    for (int it = threadIdx.x; it < NY * A2; it += NT) {
      const int n2 = it % A2, y = it / A2;
      C2* row = B + y * LD;
      T re[A1], im[A1];
#pragma unroll
      for (int n1 = 0; n1 < A1; ++n1) {
        const int k = A2 * n1 + n2;
        const C2 a = row[k];
        if (k == 0) {   // X[0] + i X[N], both real
          re[n1] = a.x + a.y;
          im[n1] = a.x - a.y;
        } else {
          const C2 b = row[N - k];   // b = X[N-k]; its conjugate enters
          const C2 w = plane_tw<T, NZ, 1>(tw, k);
          const T sx = a.x + b.x, sy = a.y - b.y, dx = a.x - b.x, dy = a.y + b.y;
          // i w (dx + i dy) = i (w.x dx - w.y dy) - (w.x dy + w.y dx)
          re[n1] = sx - (w.x * dy + w.y * dx);
          im[n1] = sy + (w.x * dx - w.y * dy);
        }
      }
      __syncwarp();   // the row's values are in registers: the padded layout may be written over them
      dft_reg<T, A1, 1>(re, im);
#pragma unroll
      for (int k1 = 0; k1 < A1; ++k1)
        row[k1 * GRP + n2] = plane_cmul(C2{re[k1], im[k1]}, plane_tw<T, N, 1>(tw, n2 * k1));
    }
    __syncthreads();
    // inverse z pass 2 to the mesh: item (row, k1), lanes over k1
#pragma unroll 1
    for (int it = threadIdx.x; it < NY * A1; it += NT) {
      const int k1 = it % A1, q = it / A1;
      const int y = q / B2 + B1 * (q % B2);   // row q = B2 k1 + k2 of the y transform
      const C2* row = B + q * LD + k1 * GRP;
      T re[A2], im[A2];
#pragma unroll
      for (int n2 = 0; n2 < A2; ++n2) {
        const C2 v = row[n2];
        re[n2] = v.x;
        im[n2] = v.y;
      }
      dft_reg<T, A2, 1>(re, im);
#pragma unroll
      for (int k2 = 0; k2 < A2; ++k2) out[(size_t)y * N + k1 + A1 * k2] = C2{re[k2], im[k2]};
    }
  }
}

// ------------------------------------------------------------------ launch
template <typename T, int NY, int NZ>
static int launch_plane_t(bool inverse, int nplanes, const void* in, void* out, cudaStream_t s) {
  using C2 = typename Cplx<T>::type;
  using Cf = PlaneCfg<T, NY, NZ>;
  static_assert(NY * Cf::A1 % 32 == 0 && NY * Cf::A2 % 32 == 0, "whole warps");
  const void* kern = inverse ? reinterpret_cast<const void*>(k_plane_inverse<T, NY, NZ>)
                             : reinterpret_cast<const void*>(k_plane_forward<T, NY, NZ>);
  if (Cf::kSmem > 48 * 1024) {
    const int rc = allow_dynamic_smem(kern, Cf::kSmem);
    if (rc) return rc;
  }
  const int most = 148 * Cf::kMinBlocks;   // persistent: the twiddles once per CTA
  const int blocks = nplanes < most ? nplanes : most;
  if (inverse)
    k_plane_inverse<T, NY, NZ><<<blocks, Cf::kThreads, Cf::kSmem, s>>>((const C2*)in, (T*)out, nplanes);
  else
    k_plane_forward<T, NY, NZ><<<blocks, Cf::kThreads, Cf::kSmem, s>>>((const T*)in, (C2*)out, nplanes);
  FD3_LAUNCHED();
  return FD3_OK;
}

template <typename T, int NY>
int launch_plane_ny(bool inverse, int nz, int nplanes, const void* in, void* out, cudaStream_t s) {
  constexpr int most = sizeof(T) == 4 ? 32768 : 16384;
  switch (nz) {
    case 16: return launch_plane_t<T, NY, 16>(inverse, nplanes, in, out, s);
    case 32: return launch_plane_t<T, NY, 32>(inverse, nplanes, in, out, s);
    case 64: return launch_plane_t<T, NY, 64>(inverse, nplanes, in, out, s);
    case 128:
      if constexpr (NY * 128 <= most) return launch_plane_t<T, NY, 128>(inverse, nplanes, in, out, s);
      break;
    case 256:
      if constexpr (NY * 256 <= most) return launch_plane_t<T, NY, 256>(inverse, nplanes, in, out, s);
      break;
  }
  return FD3_EINVAL;
}

}  // namespace fd3
