// Preparation of a call from its positions: the cell, the bin-sorted copy of the atoms (cell list),
// the atoms sorted by (mesh tile, species) with their stencil records, and the mixed form's Green
// table. (reference: src/fourierd3/calculator.py:94-123, src/fourierd3/core.py:254-267, 555)
//
// Both sorts go through the same four steps, each over all atoms: key and arrival slot (the atomic
// that counts the key), scan of the counts, scatter in arrival order, final place by rank inside the
// segment (see counting_sort) with the sorted copies written there and then. Every step is far below
// a microsecond of work for a few thousand atoms, so what bounds them is the launch chain: one CTA
// runs all of it in shared memory while it can (k_prep_small), otherwise one memset and four launches
// do both sorts, the records and the Green table (two streams of 8 launches and 3 memsets before:
// 62-74 us of stream time at 14 to 5,000 atoms).
#pragma once
#include "fd3_prep_args.cuh"

namespace fd3 {

__device__ __forceinline__ const CellInfo* prep_cell(const PrepDev& a) { return a.use_host ? &a.host : a.ci; }

// The call's cell for the kernels that follow; stale when the device copy differs.
__device__ __forceinline__ void prep_store_cell(const PrepDev& a) {
  if (!a.use_host) return;
  bool stale = false;
  if (a.d_cell)
    for (int k = 0; k < 9; ++k) stale |= a.d_cell[k] != a.host_cell[k];
  CellInfo c = a.host;
  c.stale = stale ? 1.0 : 0.0;
  *a.ci = c;
}

__device__ __forceinline__ int4 prep_bin(const PrepDev& a, int i) {
  const double x0 = a.pos[3 * i], x1 = a.pos[3 * i + 1], x2 = a.pos[3 * i + 2];
  int o[3], b[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double f = x0 * a.g.inv[c] + x1 * a.g.inv[3 + c] + x2 * a.g.inv[6 + c];
    const double fl = floor(f);
    o[c] = (int)fl;
    const int bb = (int)((f - fl) * a.g.nb[c]);
    b[c] = bb < 0 ? 0 : (bb >= a.g.nb[c] ? a.g.nb[c] - 1 : bb);
  }
  return make_int4(o[0], o[1], o[2], (b[0] * a.g.nb[1] + b[1]) * a.g.nb[2] + b[2]);
}

__device__ __forceinline__ int prep_mesh_key(const PrepDev& a, int i) {
  int base[3];
  double xl[3];
  mesh_locate<double>(a.pos, i, a.ps, prep_cell(a), a.m.n[0], a.m.n[1], a.m.n[2], a.P, base, xl);
  const int tx = base[0] / a.m.t[0], ty = base[1] / a.m.t[1], tz = base[2] / a.m.t[2];
  return ((tx * a.m.nt[1] + ty) * a.m.nt[2] + tz) * a.m.S + a.species[i];
}

__device__ __forceinline__ void prep_emit_bin(const PrepDev& a, int i, int4 o, int t) {
  a.xs[t] = make_double4(a.pos[3 * i], a.pos[3 * i + 1], a.pos[3 * i + 2], a.species ? (double)a.species[i] : 0.0);
  a.meta[t] = make_int4(o.x, o.y, o.z, i);
}

// Stencil record of atom i at sorted slot t: first node and species, the P weights per axis and their
// derivatives.
template <typename T, int P, bool LAG>
__device__ __forceinline__ void prep_emit_mesh(const PrepDev& a, int i, int t) {
  a.morder[t] = i;
  a.mslot[i] = t;
  int base[3];
  T xl[3];
  mesh_locate<T>(a.pos, i, a.ps, prep_cell(a), a.m.n[0], a.m.n[1], a.m.n[2], P, base, xl);
  a.rb[t] = make_int4(base[0], base[1], base[2], a.species[i]);
  T* rw = (T*)a.rw + (size_t)t * 3 * P;
  T* rdw = (T*)a.rdw + (size_t)t * 3 * P;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    T w[P], dw[P];
    stencil_weights<P, LAG, T>(xl[c], w, dw);
#pragma unroll
    for (int k = 0; k < P; ++k) {
      rw[c * P + k] = w[k];
      rdw[c * P + k] = dw[k];
    }
  }
}

// Green-table entries e0, e0 + step, ...
__device__ __forceinline__ void prep_green(const PrepDev& a, int e0, int step) {
  const int total = a.m.S * (a.m.S + 1) / 2 * (kGreenKnots + 1);
  for (int e = e0; e < total; e += step) a.gtab[e] = green_table_entry(a.m, prep_cell(a)->recip, a.gp, a.tab, e);
}

// ------------------------------------------------------------------ one CTA
constexpr int kPrepSmallThreads = 1024;
constexpr int kPrepSmallAtoms = 2048;
constexpr int kPrepSmallInts = 44 * 1024 / 4;   // counts of both sorts and 2 n ids, without the opt-in

// CTA 0 sorts; further CTAs, when there are any, fill the Green table beside it.
template <typename T, int P, bool LAG>
__global__ void __launch_bounds__(kPrepSmallThreads) k_prep_small(const __grid_constant__ PrepDev a) {
  extern __shared__ int ps_raw[];
  __shared__ int warp_tot[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (blockIdx.x > 0) {
    prep_green(a, (blockIdx.x - 1) * kPrepSmallThreads + tid, (gridDim.x - 1) * kPrepSmallThreads);
    return;
  }
  const int nc = a.K + a.Km;
  int* cnt = ps_raw;          // [K | Km]: counts, then segment starts (the mesh's after n bin entries)
  int* tb = cnt + nc;         // ids by bin, in arrival order
  int* tm = tb + (a.K ? a.n : 0);
  for (int e = tid; e < nc; e += kPrepSmallThreads) cnt[e] = 0;
  if (tid == 0) prep_store_cell(a);
  __syncthreads();
  constexpr int kItems = kPrepSmallAtoms / kPrepSmallThreads;
  int4 off[kItems];
  int bslot[kItems], mkey[kItems], mslot[kItems];
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int i = tid + q * kPrepSmallThreads;
    if (i < a.n) {
      if (a.K) {
        off[q] = prep_bin(a, i);
        a.off[i] = off[q];
        bslot[q] = atomicAdd(&cnt[off[q].w], 1);
      }
      if (a.Km) {
        mkey[q] = a.K + prep_mesh_key(a, i);
        mslot[q] = atomicAdd(&cnt[mkey[q]], 1);
      }
    }
  }
  __syncthreads();
  // exclusive scan of both count arrays at once: `each` consecutive entries per thread
  const int each = (nc + kPrepSmallThreads - 1) / kPrepSmallThreads;
  const int e0 = tid * each, e1 = e0 + each < nc ? e0 + each : nc;
  int local = 0;
  for (int e = e0; e < e1; ++e) local += cnt[e];
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    const int w = warp_tot[lane];
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    warp_tot[lane] = wi - w;
  }
  __syncthreads();
  int run = warp_tot[wid] + incl - local;
  const int nb = a.K ? a.n : 0;   // the mesh segments follow the n bin entries in the scan
  for (int e = e0; e < e1; ++e) {
    const int c = cnt[e], start = e < a.K ? run : run - nb;
    cnt[e] = start;
    if (e < a.K) a.bin_start[e] = start;
    else a.mstart[e - a.K] = start;
    run += c;
  }
  if (tid == 0) {
    if (a.K) a.bin_start[a.K] = a.n;
    if (a.Km) a.mstart[a.Km] = a.n;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int i = tid + q * kPrepSmallThreads;
    if (i < a.n) {
      if (a.K) tb[cnt[off[q].w] + bslot[q]] = i;
      if (a.Km) tm[cnt[mkey[q]] + mslot[q]] = i;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int i = tid + q * kPrepSmallThreads;
    if (i < a.n) {
      if (a.K) {
        const int k = off[q].w;
        prep_emit_bin(a, i, off[q], ranked_place(tb, i, cnt[k], k + 1 < a.K ? cnt[k + 1] : a.n));
      }
      if (a.Km) {
        const int k = mkey[q];
        prep_emit_mesh<T, P, LAG>(a, i, ranked_place(tm, i, cnt[k], k + 1 < nc ? cnt[k + 1] : a.n));
      }
    }
  }
}

// ------------------------------------------------------------------ several launches
static __global__ void __launch_bounds__(256) k_prep_keys(const __grid_constant__ PrepDev a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) prep_store_cell(a);
  if (i >= a.n) return;
  if (a.K) {
    const int4 o = prep_bin(a, i);
    a.off[i] = o;
    a.bslot[i] = atomicAdd(&a.counts[o.w], 1);
  }
  if (a.Km) {
    const int k = prep_mesh_key(a, i);
    a.mkeys[i] = k;
    a.mslot[i] = atomicAdd(&a.counts[a.K + k], 1);
  }
}

static __global__ void __launch_bounds__(kScanThreads) k_prep_scan(const __grid_constant__ PrepDev a) {
  if (blockIdx.x == 0 && a.K)
    scan_exclusive_block(a.counts, a.K, a.bin_start);
  else
    scan_exclusive_block(a.counts + a.K, a.Km, a.mstart);
}

static __global__ void __launch_bounds__(256) k_prep_scatter(const __grid_constant__ PrepDev a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  if (a.K) a.btmp[a.bin_start[a.off[i].w] + a.bslot[i]] = i;
  if (a.Km) a.mtmp[a.mstart[a.mkeys[i]] + a.mslot[i]] = i;
}

// blockIdx.y: 0 the bin-sorted atoms, 1 the mesh-sorted records, 2 the Green table (the first
// present ones).
template <typename T, int P, bool LAG>
__global__ void __launch_bounds__(256) k_prep_emit(const __grid_constant__ PrepDev a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int part = blockIdx.y + (a.K ? 0 : 1);
  if (part == 2) {
    prep_green(a, p, gridDim.x * blockDim.x);
  } else if (p < a.n) {
    if (part == 0) {
      const int i = a.btmp[p];
      const int4 o = a.off[i];
      prep_emit_bin(a, i, o, ranked_place(a.btmp, i, a.bin_start[o.w], a.bin_start[o.w + 1]));
    } else {
      const int i = a.mtmp[p], k = a.mkeys[i];
      prep_emit_mesh<T, P, LAG>(a, i, ranked_place(a.mtmp, i, a.mstart[k], a.mstart[k + 1]));
    }
  }
}

template <typename T, int P, bool LAG>
static int prep_t(const PrepDev& a, cudaStream_t s) {
  const bool green = a.gtab != nullptr;
  const int green_n = green ? a.m.S * (a.m.S + 1) / 2 * (kGreenKnots + 1) : 0;
  const int ints = a.K + a.Km + ((a.K ? 1 : 0) + (a.Km ? 1 : 0)) * a.n;
  if (a.n <= kPrepSmallAtoms && ints <= kPrepSmallInts) {
    int extra = (green_n + kPrepSmallThreads - 1) / kPrepSmallThreads;
    if (extra > 147) extra = 147;
    k_prep_small<T, P, LAG><<<1 + extra, kPrepSmallThreads, ints * sizeof(int), s>>>(a);
    FD3_LAUNCHED();
    return FD3_OK;
  }
  const int nb = (a.n + 255) / 256;
  FD3_CUDA(cudaMemsetAsync(a.counts, 0, sizeof(int) * (a.K + a.Km), s));
  k_prep_keys<<<nb, 256, 0, s>>>(a);
  FD3_LAUNCHED();
  k_prep_scan<<<(a.K ? 1 : 0) + (a.Km ? 1 : 0), kScanThreads, 0, s>>>(a);
  FD3_LAUNCHED();
  k_prep_scatter<<<nb, 256, 0, s>>>(a);
  FD3_LAUNCHED();
  k_prep_emit<T, P, LAG><<<dim3(nb, (a.K ? 1 : 0) + 1 + (green ? 1 : 0)), 256, 0, s>>>(a);
  FD3_LAUNCHED();
  return FD3_OK;
}

template <typename T, bool LAG>
int launch_prep(const PrepDev& a, cudaStream_t s) {
#define FD3_PREP_CASE(PP) \
  case PP:                \
    return prep_t<T, PP, LAG>(a, s);
  switch (a.P) {
    FD3_PREP_CASE(1)
    FD3_PREP_CASE(2)
    FD3_PREP_CASE(3)
    FD3_PREP_CASE(4)
    FD3_PREP_CASE(5)
    FD3_PREP_CASE(6)
    FD3_PREP_CASE(7)
    FD3_PREP_CASE(8)
  }
#undef FD3_PREP_CASE
  return FD3_EINVAL;
}

}  // namespace fd3
