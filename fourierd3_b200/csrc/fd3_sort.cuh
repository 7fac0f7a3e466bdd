// Device pieces of the counting sorts and the bin grid, shared by the cell list and the call's
// preparation.
#pragma once
#include "fd3_internal.h"

namespace fd3 {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;

// Exclusive scan of in[n] by one CTA of kScanThreads; out[n] = total.
__device__ __forceinline__ void scan_exclusive_block(const int* __restrict__ in, int n, int* __restrict__ out) {
  __shared__ int warp_tot[32];
  __shared__ int carry_s;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int base = 0; base < n; base += kScanThreads * kScanItems) {
    int v[kScanItems];
    int local = 0;
    const int i0 = base + threadIdx.x * kScanItems;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      v[k] = (i0 + k < n) ? in[i0 + k] : 0;
      local += v[k];
    }
    int incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      int w = warp_tot[lane];
      int wi = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += t;
      }
      warp_tot[lane] = wi - w;   // exclusive warp offsets
    }
    __syncthreads();
    int run = carry_s + warp_tot[wid] + incl - local;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (i0 + k < n) out[i0 + k] = run;
      run += v[k];
    }
    __syncthreads();
    if (threadIdx.x == kScanThreads - 1) carry_s = run;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry_s;
}

// Place of an id of the arrival-ordered segment [a, b) once the segment is sorted.
__device__ __forceinline__ int ranked_place(const int* __restrict__ arrival, int id, int a, int b) {
  int rank = 0;
#pragma unroll 4
  for (int q = a; q < b; ++q) rank += arrival[q] < id ? 1 : 0;
  return a + rank;
}

// ------------------------------------------------------------------ bin grid
struct GridDev {
  int nb[3], reach[3];
  double cell[9], inv[9];
  double rc2;
};
static inline GridDev to_dev(const CellGrid& g) {
  GridDev d;
  for (int a = 0; a < 3; ++a) {
    d.nb[a] = g.nb[a];
    d.reach[a] = g.reach[a];
  }
  for (int k = 0; k < 9; ++k) {
    d.cell[k] = g.cell[k];
    d.inv[k] = g.inv[k];
  }
  d.rc2 = g.rc2;
  return d;
}

}  // namespace fd3
