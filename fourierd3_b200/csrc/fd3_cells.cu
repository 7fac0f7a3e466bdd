// Cell-list neighbour search, smooth-cutoff coordination numbers, C6 factors and the
// CN adjoint (reference: src/fourierd3/core.py:323-386, 449-478, 525-550 and the matscipy
// neighbour build at src/fourierd3/calculator.py:94-123).
//
// Design: atoms are counting-sorted into a bin grid whose bins are at least r_cut wide (in
// perpendicular height), so a neighbour lies within `reach` bins per axis. Bins are laid out
// with z fastest, so for a fixed (dx, dy) the bins bz-reach..bz+reach are one contiguous run of
// the bin-sorted atom array (split only at the periodic wrap). One warp handles one atom and
// strides its lanes over those runs, so the candidate loads are coalesced.
#include <math.h>
#include <stdio.h>

#include "fd3_sort.cuh"

namespace fd3 {

// ------------------------------------------------------------------ host geometry
static void inv3_host(const double* m, double* inv, double* det_out) {
  const double c00 = m[4] * m[8] - m[5] * m[7];
  const double c01 = m[2] * m[7] - m[1] * m[8];
  const double c02 = m[1] * m[5] - m[2] * m[4];
  const double c10 = m[5] * m[6] - m[3] * m[8];
  const double c11 = m[0] * m[8] - m[2] * m[6];
  const double c12 = m[2] * m[3] - m[0] * m[5];
  const double c20 = m[3] * m[7] - m[4] * m[6];
  const double c21 = m[1] * m[6] - m[0] * m[7];
  const double c22 = m[0] * m[4] - m[1] * m[3];
  const double det = m[0] * c00 + m[1] * c10 + m[2] * c20;
  const double a[9] = {c00, c01, c02, c10, c11, c12, c20, c21, c22};
  for (int k = 0; k < 9; ++k) inv[k] = a[k] / det;
  if (det_out) *det_out = det;
}

int make_cell_grid(const double* h_cell, double r_cut, CellGrid* g) {
  if (!h_cell || !g) {
    set_error("cell grid", "null cell");
    return FD3_EINVAL;
  }
  if (!(r_cut > 0)) return FD3_EINVAL;
  double det;
  inv3_host(h_cell, g->inv, &det);
  if (!(fabs(det) > 0) || !isfinite(det)) return FD3_EINVAL;
  for (int k = 0; k < 9; ++k) g->cell[k] = h_cell[k];
  for (int a = 0; a < 3; ++a) {
    // perpendicular height of the cell along axis a = 1 / |column a of inv(cell)|
    const double cn = sqrt(g->inv[0 * 3 + a] * g->inv[0 * 3 + a] + g->inv[1 * 3 + a] * g->inv[1 * 3 + a] +
                           g->inv[2 * 3 + a] * g->inv[2 * 3 + a]);
    const double h = 1.0 / cn;
    int nb = (int)floor(h / r_cut);
    if (nb < 1) nb = 1;
    if (nb > 512) nb = 512;
    g->nb[a] = nb;
    g->reach[a] = (int)ceil(r_cut * nb / h + 1e-9);
  }
  g->r_cut = r_cut;
  g->rc2 = r_cut * r_cut;
  return FD3_OK;
}

// ------------------------------------------------------------------ scan / sort
__global__ void __launch_bounds__(kScanThreads) k_scan_exclusive(const int* __restrict__ in, int n,
                                                                int* __restrict__ out) {
  scan_exclusive_block(in, n, out);
}

int scan_exclusive(const int* in, int n, int* out, cudaStream_t s) {
  k_scan_exclusive<<<1, kScanThreads, 0, s>>>(in, n, out);
  FD3_LAUNCHED();
  return FD3_OK;
}

// Counting sort of the ids 0..n-1 by key, ids ascending within a key. The atomic that counts a key
// also hands the id its arrival slot, so one scatter fills the segments in arrival order; the last
// kernel then gives every id its final place by its rank in its segment (the number of smaller ids
// there), which makes the order independent of the atomics. Its threads walk the segments in
// position order, so the lanes of a warp scan the same few segments (broadcast loads): m compares
// per id for a segment of m ids, all ids at once. (Sorting each segment in one warp, longer ones by
// insertion in one lane: a call at 12,000 HCNO atoms, 343 bins of 35, 51 us longer; one with 1.2 M edges in
// segments of 59 380 us longer.)
__global__ void __launch_bounds__(256) k_key_slots(const int* __restrict__ keys, int n, int* __restrict__ counts,
                                                  int* __restrict__ slot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) slot[i] = atomicAdd(&counts[keys[i]], 1);
}

__global__ void __launch_bounds__(256) k_scatter(const int* __restrict__ keys, int n, const int* __restrict__ starts,
                                                const int* __restrict__ slot, int* __restrict__ arrival) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) arrival[starts[keys[i]] + slot[i]] = i;
}

__global__ void __launch_bounds__(256) k_rank_segments(const int* __restrict__ keys, int n,
                                                      const int* __restrict__ starts,
                                                      const int* __restrict__ arrival, int* __restrict__ order) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int i = arrival[p], k = keys[i];
  order[ranked_place(arrival, i, starts[k], starts[k + 1])] = i;
}

// arrival: scratch of n ints; order also holds the arrival slots until the last kernel writes it.
int counting_sort(const int* keys, int n, int K, int* counts, int* starts, int* order, int* arrival,
                  cudaStream_t s) {
  const int tb = 256, nb = (n + tb - 1) / tb;
  FD3_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * K, s));
  if (n > 0) {
    k_key_slots<<<nb, tb, 0, s>>>(keys, n, counts, order);
    FD3_LAUNCHED();
  }
  int rc = scan_exclusive(counts, K, starts, s);
  if (rc || n <= 0) return rc;
  k_scatter<<<nb, tb, 0, s>>>(keys, n, starts, order, arrival);
  FD3_LAUNCHED();
  k_rank_segments<<<nb, tb, 0, s>>>(keys, n, starts, arrival, order);
  FD3_LAUNCHED();
  return FD3_OK;
}

// ------------------------------------------------------------------ cell list
__global__ void __launch_bounds__(256) k_bin_atoms(GridDev g, int n, const double* __restrict__ x, int* __restrict__ bin_of,
                            int4* __restrict__ off) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x0 = x[3 * i], x1 = x[3 * i + 1], x2 = x[3 * i + 2];
  int o[3], b[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double f = x0 * g.inv[a] + x1 * g.inv[3 + a] + x2 * g.inv[6 + a];
    const double fl = floor(f);
    o[a] = (int)fl;
    int bb = (int)((f - fl) * g.nb[a]);
    b[a] = bb < 0 ? 0 : (bb >= g.nb[a] ? g.nb[a] - 1 : bb);
  }
  const int bin = (b[0] * g.nb[1] + b[1]) * g.nb[2] + b[2];
  bin_of[i] = bin;
  off[i] = make_int4(o[0], o[1], o[2], bin);
}

__global__ void __launch_bounds__(256) k_gather_sorted(int n, const int* __restrict__ order, const double* __restrict__ x,
                                const int32_t* __restrict__ species, const int4* __restrict__ off,
                                double4* __restrict__ xs, int4* __restrict__ meta) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int i = order[t];
  xs[t] = make_double4(x[3 * i], x[3 * i + 1], x[3 * i + 2], species ? (double)species[i] : 0.0);
  const int4 o = off[i];
  meta[t] = make_int4(o.x, o.y, o.z, i);
}

int build_cell_list(const CellGrid& g, int n, const double* pos_ang, const int32_t* species, CellList& cl,
                    cudaStream_t s) {
  const int K = g.nb[0] * g.nb[1] * g.nb[2];
  const int tb = 256;
  if (n > 0) {
    k_bin_atoms<<<(n + tb - 1) / tb, tb, 0, s>>>(to_dev(g), n, pos_ang, cl.bin_of, cl.off);
    FD3_LAUNCHED();
  }
  // meta is written after the sort: until then it is the sort's scratch
  int rc = counting_sort(cl.bin_of, n, K, cl.bin_count, cl.bin_start, cl.order, reinterpret_cast<int*>(cl.meta), s);
  if (rc) return rc;
  if (n > 0) {
    k_gather_sorted<<<(n + tb - 1) / tb, tb, 0, s>>>(n, cl.order, pos_ang, species, cl.off, cl.xs, cl.meta);
    FD3_LAUNCHED();
  }
  return FD3_OK;
}

// The exact pair predicate (Angstrom, no FMA): d = (x_j - x_i) + S . cell, |d|^2 < r_cut^2.
__device__ __forceinline__ bool pair_inside(const GridDev& g, double xj0, double xj1, double xj2, double xi0,
                                            double xi1, double xi2, int S0, int S1, int S2, double& d0, double& d1,
                                            double& d2) {
  const double sh0 = dadd(dadd(dmul((double)S0, g.cell[0]), dmul((double)S1, g.cell[3])), dmul((double)S2, g.cell[6]));
  const double sh1 = dadd(dadd(dmul((double)S0, g.cell[1]), dmul((double)S1, g.cell[4])), dmul((double)S2, g.cell[7]));
  const double sh2 = dadd(dadd(dmul((double)S0, g.cell[2]), dmul((double)S1, g.cell[5])), dmul((double)S2, g.cell[8]));
  d0 = dadd(dsub(xj0, xi0), sh0);
  d1 = dadd(dsub(xj1, xi1), sh1);
  d2 = dadd(dsub(xj2, xi2), sh2);
  return dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2)) < g.rc2;
}

// Visit every candidate (j, S) of atom i. All lanes of the warp run the same number of
// iterations; `fn(hit, u, j, S, d)` gets the exact-predicate result (Angstrom, no FMA).
template <class Fn>
__device__ __forceinline__ void visit_neighbors(const GridDev& g, const int* __restrict__ bin_start,
                                                const double4* __restrict__ xs, const int4* __restrict__ meta,
                                                int i, double xi0, double xi1, double xi2, int4 offi, Fn&& fn) {
  const int lane = threadIdx.x & 31;
  const int bin = offi.w;
  const int bz = bin % g.nb[2];
  const int by = (bin / g.nb[2]) % g.nb[1];
  const int bx = bin / (g.nb[2] * g.nb[1]);
  for (int dx = -g.reach[0]; dx <= g.reach[0]; ++dx) {
    const int cx = bx + dx;
    const int sx = floordiv(cx, g.nb[0]);
    const int wx = cx - sx * g.nb[0];
    for (int dy = -g.reach[1]; dy <= g.reach[1]; ++dy) {
      const int cy = by + dy;
      const int sy = floordiv(cy, g.nb[1]);
      const int wy = cy - sy * g.nb[1];
      int zs = bz - g.reach[2];
      const int ze = bz + g.reach[2];
      while (zs <= ze) {
        const int sz = floordiv(zs, g.nb[2]);
        const int wz = zs - sz * g.nb[2];
        int len = g.nb[2] - wz;
        if (len > ze - zs + 1) len = ze - zs + 1;
        const int b0 = (wx * g.nb[1] + wy) * g.nb[2] + wz;
        const int a0 = bin_start[b0], a1 = bin_start[b0 + len];
        for (int u0 = a0; u0 < a1; u0 += 32) {
          const int u = u0 + lane;
          bool hit = false;
          int j = 0;
          int S0 = 0, S1 = 0, S2 = 0;
          double d0 = 0, d1 = 0, d2 = 0;
          if (u < a1) {
            const double4 xj = xs[u];
            const int4 mj = meta[u];
            j = mj.w;
            S0 = sx + offi.x - mj.x;
            S1 = sy + offi.y - mj.y;
            S2 = sz + offi.z - mj.z;
            hit = pair_inside(g, xj.x, xj.y, xj.z, xi0, xi1, xi2, S0, S1, S2, d0, d1, d2) &&
                  !(j == i && S0 == 0 && S1 == 0 && S2 == 0);
          }
          fn(hit, u, j, S0, S1, S2, d0, d1, d2);
        }
        zs += len;
      }
    }
  }
}

constexpr int kWarpsPerBlock = 8;

// Per-atom traversal straight from global memory: the path for bins whose neighbourhood does not
// fit the shared-memory stage (dense clusters, cells much narrower than the cutoff).
__device__ __noinline__ double cn_atom_global(const GridDev& g, const int* __restrict__ bin_start,
                                                 const double4* __restrict__ xs, const int4* __restrict__ meta,
                                                 const int4* __restrict__ off, const Tables* __restrict__ tab,
                                                 int t) {
  const double4 xi = xs[t];
  const int i = meta[t].w;
  const int4 offi = off[i];
  const double rci = tab->rcov[(int)xi.w];
  double acc = 0.0;
  visit_neighbors(g, bin_start, xs, meta, i, xi.x, xi.y, xi.z, offi,
                  [&](bool hit, int u, int, int, int, int, double d0, double d1, double d2) {
                    if (!hit) return;
                    const double v0 = d0 * kAngToBohr, v1 = d1 * kAngToBohr, v2 = d2 * kAngToBohr;
                    double f, df;
                    cn_edge(sqrt(v0 * v0 + v1 * v1 + v2 * v2), rci + tab->rcov[(int)xs[u].w], tab->r_cut, f, df);
                    acc += f;
                  });
  return warp_sum(acc);
}

// Sums of one atom's pairs, this lane's share: the CN force and the six virial components.
struct PairSums {
  double f0, f1, f2, xx, xy, xz, yy, yz, zz;
};
__device__ __noinline__ PairSums cn_adjoint_atom_global(const GridDev& g, const int* __restrict__ bin_start,
                                                        const double4* __restrict__ xs,
                                                        const int4* __restrict__ meta, const int4* __restrict__ off,
                                                        const Tables* __restrict__ tab, const double* __restrict__ gcn,
                                                        int t) {
  const double4 xi = xs[t];
  const int i = meta[t].w;
  const int4 offi = off[i];
  const double rci = tab->rcov[(int)xi.w];
  const double gi = gcn[i];
  PairSums p{0, 0, 0, 0, 0, 0, 0, 0, 0};
  visit_neighbors(g, bin_start, xs, meta, i, xi.x, xi.y, xi.z, offi,
                  [&](bool hit, int u, int j, int, int, int, double d0, double d1, double d2) {
                    if (!hit) return;
                    const double v0 = d0 * kAngToBohr, v1 = d1 * kAngToBohr, v2 = d2 * kAngToBohr;
                    const double r = sqrt(v0 * v0 + v1 * v1 + v2 * v2);
                    double fe, df;
                    cn_edge(r, rci + tab->rcov[(int)xs[u].w], tab->r_cut, fe, df);
                    if (r > 1e-6) {
                      const double a = df / r;
                      const double w = (gi + gcn[j]) * a;
                      p.f0 -= w * v0;
                      p.f1 -= w * v1;
                      p.f2 -= w * v2;
                      const double b = gi * a;
                      p.xx += b * v0 * v0; p.xy += b * v0 * v1; p.xz += b * v0 * v2;
                      p.yy += b * v1 * v1; p.yz += b * v1 * v2; p.zz += b * v2 * v2;
                    }
                  });
  return p;
}

// ------------------------------------------------------------------ bin-staged CN
// The candidates of a bin are the atoms of its (2 reach + 1)^3 neighbour bins, numbered through the
// neighbour bins in a fixed order. A CTA stages up to `cap` of them at a time in shared memory as
// image positions p_j = x_j + (S' - off_j) . cell, and its warps run the bin's own atoms against
// that stage (d = p_j - (x_i - off_i . cell)).
constexpr int kMaxNbrBins = 343;

// P4 = double4: absolute image positions (the plain form, and the exact pair predicate);
// P4 = float4 (mixed form): positions relative to the bin's own corner, so that float keeps
// ~1e-6 A over the few bins a stage spans.
struct NbrBins {
  int a0[kMaxNbrBins];
  int pref[kMaxNbrBins + 1];
  int img[kMaxNbrBins][3];
};

// Table of the neighbour bins of bin b. Returns the number of candidates, or -1 when the
// neighbourhood has more than kMaxNbrBins bins (a cell much narrower than the cutoff).
__device__ __forceinline__ int nbr_bins(const GridDev& g, int b, const int* __restrict__ bin_start, NbrBins& st) {
  const int nx = 2 * g.reach[0] + 1, ny = 2 * g.reach[1] + 1, nz = 2 * g.reach[2] + 1;
  const int nnb = nx * ny * nz;
  if (nnb > kMaxNbrBins) return -1;
  const int bz = b % g.nb[2], by = (b / g.nb[2]) % g.nb[1], bx = b / (g.nb[2] * g.nb[1]);
  for (int e = threadIdx.x; e < nnb; e += blockDim.x) {
    const int dz = e % nz - g.reach[2], dy = (e / nz) % ny - g.reach[1], dx = e / (nz * ny) - g.reach[0];
    const int cx = bx + dx, cy = by + dy, cz = bz + dz;
    const int sx = floordiv(cx, g.nb[0]), sy = floordiv(cy, g.nb[1]), sz = floordiv(cz, g.nb[2]);
    const int id = ((cx - sx * g.nb[0]) * g.nb[1] + (cy - sy * g.nb[1])) * g.nb[2] + (cz - sz * g.nb[2]);
    const int a0 = bin_start[id];
    st.a0[e] = a0;
    st.pref[e + 1] = bin_start[id + 1] - a0;
    st.img[e][0] = sx;
    st.img[e][1] = sy;
    st.img[e][2] = sz;
  }
  __syncthreads();
  if (threadIdx.x < 32) {   // one warp scans the bin sizes (27 bins at reach 1: one round)
    int carry = 0;
    for (int e0 = 0; e0 < nnb; e0 += 32) {
      const int e = e0 + (int)threadIdx.x;
      int v = e < nnb ? st.pref[e + 1] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if ((int)threadIdx.x >= o) v += u;
      }
      v += carry;
      if (e < nnb) st.pref[e + 1] = v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
    if (threadIdx.x == 0) st.pref[0] = 0;
  }
  __syncthreads();
  return st.pref[nnb];
}

// Neighbour bin of candidate c: the last entry with pref[e] <= c.
__device__ __forceinline__ int nbr_bin_of(const NbrBins& st, int nnb, int c) {
  int lo = 0, hi = nnb - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (st.pref[mid] <= c) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Stage candidates [c0, c1); org is subtracted from the staged positions (zero for double4). The
// staged w component is the candidate's covalent radius (the CN's only use of the species).
template <typename P4>
__device__ __forceinline__ void stage_candidates(const GridDev& g, const NbrBins& st, int c0, int c1,
                                                 const double4* __restrict__ xs, const int4* __restrict__ meta,
                                                 const double (&org)[3], const double* __restrict__ rcov, P4* p,
                                                 int* j) {
  const int nnb = (2 * g.reach[0] + 1) * (2 * g.reach[1] + 1) * (2 * g.reach[2] + 1);
  for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
    const int lo = nbr_bin_of(st, nnb, c);
    const int u = st.a0[lo] + (c - st.pref[lo]);
    const double4 xj = xs[u];
    const int4 mj = meta[u];
    const double S0 = st.img[lo][0] - mj.x, S1 = st.img[lo][1] - mj.y, S2 = st.img[lo][2] - mj.z;
    const double px = xj.x + S0 * g.cell[0] + S1 * g.cell[3] + S2 * g.cell[6];
    const double py = xj.y + S0 * g.cell[1] + S1 * g.cell[4] + S2 * g.cell[7];
    const double pz = xj.z + S0 * g.cell[2] + S1 * g.cell[5] + S2 * g.cell[8];
    const double wv = rcov[(int)xj.w];
    if constexpr (sizeof(P4) == sizeof(double4))
      p[c - c0] = make_double4(px, py, pz, wv);
    else
      p[c - c0] = make_float4((float)(px - org[0]), (float)(py - org[1]), (float)(pz - org[2]), (float)wv);
    j[c - c0] = mj.w;
  }
}

__device__ __forceinline__ void wrapped_pos(const GridDev& g, double4 x, int4 m, double& w0, double& w1,
                                            double& w2) {
  w0 = x.x - (m.x * g.cell[0] + m.y * g.cell[3] + m.z * g.cell[6]);
  w1 = x.y - (m.x * g.cell[1] + m.y * g.cell[4] + m.z * g.cell[7]);
  w2 = x.z - (m.x * g.cell[2] + m.y * g.cell[5] + m.z * g.cell[8]);
}

// The forward CN kernel also records, per atom, every in-cutoff pair: the neighbour id and one
// 4-wide record {f'(r)/r, Bohr vector d} (HitList, TE = double for the plain form, float for the
// mixed form), so the adjoint reads a pair with one vector load instead of searching the cell list
// a second time. An atom with more than `cap` such pairs (or one handled by the global-memory
// path) is marked n = -1 and the adjoint recomputes it.
// The dense bins of the mixed form, whose pairs are taken in float64, keep that precision in the same
// 16 bytes: {f'(r)/r as a double, the neighbour's slot in the bin-sorted atoms, its bin's image}, from
// which the adjoint forms d again in float64; their atoms are marked n = -2 - (number of pairs).
template <typename TE> struct Vec4;
template <> struct Vec4<float> { using type = float4; };
template <> struct Vec4<double> { using type = double4; };

template <typename TE>
struct HitList {
  int* j;
  typename Vec4<TE>::type* ad;
  int* n;
  int cap;
};

// Image of a neighbour bin in one word: at most 343 bins of 3 or more per axis, so |image| <= 18.
__device__ __forceinline__ int pack_image(const int (&m)[3]) {
  return (m[0] + 128) | (m[1] + 128) << 8 | (m[2] + 128) << 16;
}
__device__ __forceinline__ float4 exact_record(double a, int u, int image) {
  return make_float4(__int_as_float(__double2loint(a)), __int_as_float(__double2hiint(a)), __int_as_float(u),
                     __int_as_float(image));
}

// C6 weights and factors of one atom by a group of 8 lanes: softmax interpolation over the 7
// reference CNs (one lane each), the rank-r factors c_r = sum_p w_p V[s, p, r] (core.py:449-478,
// 525-532; ranks over the lanes), their CN derivative (times the cncorr slope) and the self term
// sum_r lambda_r c_r^2 phi_ss(0) (core.py:545-550), of which each lane returns its ranks' share.
// raw_cn is the CN before cncorr; cn receives the corrected one. Every lane of the warp takes part
// (`on` false: an idle group). Eight lanes per atom: a thread per atom is a chain of seven float64
// exponentials (6 us at any size), a warp per atom repeats the work 32-fold (+60 us at 139,968 atoms).
__device__ __forceinline__ double c6_group(bool on, int i, int s, double raw_cn, const Tables* __restrict__ tab,
                                           const double* __restrict__ V, int R, double* __restrict__ cn,
                                           double* __restrict__ c6, double* __restrict__ dc6, const RankOut& ro) {
  const int lane = threadIdx.x & 7;
  double cnv = raw_cn, slope = 1.0;
  if (tab->has_cncorr) {
    slope = tab->cncorr[2 * s + 1];
    cnv = slope * cnv + tab->cncorr[2 * s + 0];
  }
  const double ref = lane < 7 ? tab->cnref[7 * s + lane] : -1.0;
  const bool ok = ref != -1.0;
  const double diff = cnv - ref;
  double lg = ok ? -4.0 * (diff * diff) : -INFINITY;
  const double dl = ok ? -8.0 * diff : 0.0;
  double mx = lg;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  lg = lg == -INFINITY ? 0.0 : exp(lg - mx);
  double sum = lg;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const double w = lg * (1.0 / sum);   // softmax weight (0 in lane 7)
  double dlbar = w * dl;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) dlbar += __shfl_xor_sync(0xffffffffu, dlbar, o);
  const double wd = w * (dl - dlbar);
  double selfv = 0.0;
  for (int r0 = 0; r0 < R; r0 += 8) {
    const int r = r0 + lane;
    double c = 0.0, d = 0.0;
#pragma unroll
    for (int p = 0; p < 7; ++p) {
      const double wp = __shfl_sync(0xffffffffu, w, p, 8), wdp = __shfl_sync(0xffffffffu, wd, p, 8);
      const double v = r < R ? V[(7 * s + p) * R + r] : 0.0;
      c += wp * v;
      d += wdp * v;
    }
    if (on && r < R) {
      c6[(size_t)i * R + r] = c;
      dc6[(size_t)i * R + r] = slope * d;
      ro.put(i, r, R, c);
      selfv += tab->eigs[r] * c * c * tab->selfcont[s];
    }
  }
  if (on && lane == 0) cn[i] = cnv;
  return selfv;
}

// CN and C6 factors of the atoms of one bin (split over nsplit CTAs when there are few bins), plus
// the pair records.
// Per atom (one warp) the staged candidates are first tested against the cutoff 32 at a time
// (float64 distances in the plain form, float relative to the bin corner in the mixed form); the
// indices of the pairs inside are compacted in order into a per-warp ring of 64, and whenever 32
// are waiting all lanes evaluate the CN function for them and write their records contiguously. The CN function and the record stores thus run on full warps
// instead of on the ~15 % of lanes that hit in a given candidate batch.
// A bin holds ~15 atoms at r_cut 6 A (SiO2 density): 4 warps per CTA leave fewer idle warps
// waiting for a bin's last atom than 8 do, and more CTAs (bins) fit per SM.
// The stage holds what the box's mean density fills, with half as much again; a bin with more candidates (a
// dense cluster, or a tiny cell whose images are all candidates) restages them in pieces of `cap`
// for each round of its warps. (With one fixed stage of 768 and a per-atom traversal of global
// memory beyond it, every bin of an HCNO box, 936 candidates, took the traversal: CN 97 us and
// adjoint 178 us at 12,000 atoms.)
constexpr int kCnRing = 64;
constexpr int kCnWarps = 4;
constexpr int kCnSmem = 56 * 1024;   // stage bytes at most: three CTAs per SM (1,593 candidates in float64)
constexpr int kCnSmemPlain = 38 * 1024;   // ... without the shared-memory opt-in (8 KB are static)

template <typename TC> struct StagePos { using type = double4; };
template <> struct StagePos<float> { using type = float4; };

template <typename TE, typename TC, typename P4>
__device__ __forceinline__ void cn_hit(const NbrBins& st, int nnb, int cb, const P4* __restrict__ sp,
                                       const int* __restrict__ sj, int c, TC w0, TC w1, TC w2, TC rci, TC rc,
                                       const HitList<TE>& hl, size_t hb, int h, TC& acc) {
  const P4 pj = sp[c];
  const TC v0 = (TC)((pj.x - w0) * (TC)kAngToBohr);
  const TC v1 = (TC)((pj.y - w1) * (TC)kAngToBohr);
  const TC v2 = (TC)((pj.z - w2) * (TC)kAngToBohr);
  const TC r2 = v0 * v0 + v1 * v1 + v2 * v2;
  TC f = TC(0), a = TC(0);
  if (r2 > TC(1e-12)) {
    cn_pair<TC>(r2, rci + (TC)pj.w, rc, f, a);   // pj.w: the neighbour's covalent radius
    acc += f;
  }
  if (h < hl.cap) {
    hl.j[hb + h] = sj[c];
    if constexpr (sizeof(TE) < sizeof(TC)) {
      const int e = nbr_bin_of(st, nnb, cb + c);
      hl.ad[hb + h] = exact_record(a, st.a0[e] + (cb + c - st.pref[e]), pack_image(st.img[e]));
    } else {
      hl.ad[hb + h] = typename Vec4<TE>::type{(TE)a, (TE)v0, (TE)v1, (TE)v2};
    }
  }
}

// The atoms of bin b that this CTA takes (part of nsplit), in arithmetic TC: raw CN to cn[], records.
// ONCE: the candidates fit the stage.
template <typename TE, typename TC, bool ONCE>
__device__ __forceinline__ void cn_bin(const GridDev& g, const NbrBins& st, int total, int cap, int b, int s0, int s1,
                                       int part, int nsplit, const double4* __restrict__ xs,
                                       const int4* __restrict__ meta, const Tables* __restrict__ tab,
                                       double* __restrict__ cn, const HitList<TE>& hl, unsigned char* stage,
                                       int* __restrict__ rg) {
  using P4 = typename StagePos<TC>::type;
  P4* sp = reinterpret_cast<P4*>(stage);
  int* sj = reinterpret_cast<int*>(sp + cap);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int bz = b % g.nb[2], by = (b / g.nb[2]) % g.nb[1], bx = b / (g.nb[2] * g.nb[1]);
  double org[3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
    org[c] = sizeof(P4) == sizeof(double4)
                 ? 0.0
                 : ((double)bx / g.nb[0]) * g.cell[c] + ((double)by / g.nb[1]) * g.cell[3 + c] +
                       ((double)bz / g.nb[2]) * g.cell[6 + c];
  const unsigned lt = (1u << lane) - 1u;
  const TC rc = (TC)tab->r_cut;
  const TC rc2 = (TC)g.rc2;
  const int nnb = (2 * g.reach[0] + 1) * (2 * g.reach[1] + 1) * (2 * g.reach[2] + 1);
  if (ONCE) {
    stage_candidates<P4>(g, st, 0, total, xs, meta, org, tab->rcov, sp, sj);
    __syncthreads();
  }
  // rounds of one atom per warp (the same number for every warp where restaging takes barriers)
  for (int t0 = s0 + part * kCnWarps; t0 < s1; t0 += kCnWarps * nsplit) {
    const int t = t0 + wid;
    const bool on = t < s1;
    if (ONCE && !on) break;
    double wd0 = 0, wd1 = 0, wd2 = 0;
    int i = 0, s = 0;
    if (on) {
      const double4 xi = xs[t];
      const int4 mi = meta[t];
      wrapped_pos(g, xi, mi, wd0, wd1, wd2);
      i = mi.w;
      s = (int)xi.w;
    }
    const TC w0 = (TC)(wd0 - org[0]), w1 = (TC)(wd1 - org[1]), w2 = (TC)(wd2 - org[2]);
    const TC rci = (TC)tab->rcov[s];
    TC acc = TC(0);
    int produced = 0, consumed = 0;
    const size_t hb = (size_t)t * hl.cap;
    for (int cb = 0; cb < (ONCE ? 1 : total); cb += cap) {
      const int cnt = ONCE || total - cb < cap ? total - cb : cap;
      if (!ONCE) {
        __syncthreads();   // every warp has finished with the previous piece
        stage_candidates<P4>(g, st, cb, cb + cnt, xs, meta, org, tab->rcov, sp, sj);
        __syncthreads();
        if (!on) continue;
      }
      for (int c0 = 0; c0 < cnt; c0 += 32) {
        const int c = c0 + lane;
        bool hit = false;
        if (c < cnt) {
          const P4 pj = sp[c];
          const TC d0 = pj.x - w0, d1 = pj.y - w1, d2 = pj.z - w2;
          hit = d0 * d0 + d1 * d1 + d2 * d2 < rc2;
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) rg[(produced + __popc(m & lt)) & (kCnRing - 1)] = c;
        produced += __popc(m);
        __syncwarp();
        if (produced - consumed >= 32) {
          const int h = consumed + lane;
          cn_hit<TE, TC>(st, nnb, cb, sp, sj, rg[h & (kCnRing - 1)], w0, w1, w2, rci, rc, hl, hb, h, acc);
          consumed += 32;
          __syncwarp();
        }
      }
      // the ring holds indices into this piece: take the rest of it before the next
      if (consumed + lane < produced) {
        const int h = consumed + lane;
        cn_hit<TE, TC>(st, nnb, cb, sp, sj, rg[h & (kCnRing - 1)], w0, w1, w2, rci, rc, hl, hb, h, acc);
      }
      consumed = produced;
      __syncwarp();
    }
    const double cnv = warp_sum((double)acc);
    if (on && lane == 0) {
      hl.n[t] = produced > hl.cap ? -1 : sizeof(TE) < sizeof(TC) ? -2 - produced : produced;
      cn[i] = cnv;
    }
  }
}

// The mixed form (TE = float) takes bins of up to kCnFloat candidates in float and denser ones in
// float64, forward and (through their records) backward, so that the sums over more pairs keep the
// accuracy of the smaller ones.
constexpr int kCnFloat = 768;

// The other cases, out of line so that the common one keeps its registers (nine CTAs per SM in float):
// a bin whose candidates do not fit the stage, and the dense bins of the mixed form.
template <typename TE>
__device__ __noinline__ void cn_bin_dense(const GridDev& g, const NbrBins& st, int total, int stage_bytes, int b,
                                          int s0, int s1, int part, int nsplit, const double4* __restrict__ xs,
                                          const int4* __restrict__ meta, const Tables* __restrict__ tab,
                                          double* __restrict__ cn, const HitList<TE>& hl, unsigned char* stage,
                                          int* __restrict__ rg) {
  if (sizeof(TE) == 4 && total <= kCnFloat)
    cn_bin<TE, float, false>(g, st, total, stage_bytes / 20, b, s0, s1, part, nsplit, xs, meta, tab, cn, hl, stage,
                             rg);
  else if (sizeof(TE) == 4 && total <= stage_bytes / 36)
    cn_bin<TE, double, true>(g, st, total, stage_bytes / 36, b, s0, s1, part, nsplit, xs, meta, tab, cn, hl, stage,
                             rg);
  else
    cn_bin<TE, double, false>(g, st, total, stage_bytes / 36, b, s0, s1, part, nsplit, xs, meta, tab, cn, hl, stage,
                              rg);
}

// C6: the factors too (c6_group, after the CTA's atoms); without it k_c6_atoms follows.
template <typename TE, bool C6>
__global__ void __launch_bounds__(32 * kCnWarps, sizeof(TE) == 4 ? 9 : 7) k_cn_bins(
                                                const __grid_constant__ GridDev g, int stage_bytes,
                                                int nsplit, const int* __restrict__ bin_start,
                                                const double4* __restrict__ xs, const int4* __restrict__ meta,
                                                const int4* __restrict__ off, const Tables* __restrict__ tab,
                                                const double* __restrict__ V, int R, double* __restrict__ cn,
                                                double* __restrict__ c6, double* __restrict__ dc6,
                                                const __grid_constant__ HitList<TE> hl, RankOut ro,
                                                double* __restrict__ self_part) {
  extern __shared__ __align__(16) unsigned char cn_raw[];
  __shared__ NbrBins st;
  __shared__ int ring[kCnWarps][kCnRing];
  const int b = blockIdx.x / nsplit, part = blockIdx.x - b * nsplit;
  const int s0 = bin_start[b], s1 = bin_start[b + 1];
  double self[1] = {0.0};
  if (s0 + part * kCnWarps < s1) {
    int* rg = ring[threadIdx.x >> 5];
    const int total = nbr_bins(g, b, bin_start, st);
    if (total < 0) {
      for (int t = s0 + part * kCnWarps + (threadIdx.x >> 5); t < s1; t += kCnWarps * nsplit) {
        const double cnv = cn_atom_global(g, bin_start, xs, meta, off, tab, t);
        if ((threadIdx.x & 31) == 0) {
          hl.n[t] = -1;
          cn[meta[t].w] = cnv;
        }
      }
    } else {
      constexpr int each = sizeof(TE) == 4 ? 20 : 36;   // staged bytes per candidate
      if (total <= stage_bytes / each && (sizeof(TE) == 8 || total <= kCnFloat))
        cn_bin<TE, TE, true>(g, st, total, stage_bytes / each, b, s0, s1, part, nsplit, xs, meta, tab, cn, hl, cn_raw,
                             rg);
      else
        cn_bin_dense<TE>(g, st, total, stage_bytes, b, s0, s1, part, nsplit, xs, meta, tab, cn, hl, cn_raw, rg);
    }
    if constexpr (C6) {
    __syncthreads();   // the raw CNs are written
    constexpr int kGroups = 4 * kCnWarps;
    const int grp = threadIdx.x >> 3;
    const int rounds = (s1 - s0 - part * kCnWarps + kCnWarps * nsplit - 1) / (kCnWarps * nsplit);
    for (int a0 = 0; a0 < rounds * kCnWarps; a0 += kGroups) {
      const int a = a0 + grp;   // atom a of this CTA: warp a mod kCnWarps of round a / kCnWarps
      const int t = s0 + part * kCnWarps + a / kCnWarps * (kCnWarps * nsplit) + a % kCnWarps;
      const bool on = a < rounds * kCnWarps && t < s1;
      const int i = on ? meta[t].w : 0, s = on ? (int)xs[t].w : 0;
      self[0] += c6_group(on, i, s, on ? cn[i] : 0.0, tab, V, R, cn, c6, dc6, ro);
    }
    }
  }
  if constexpr (C6) block_sum_store<1>(self, self_part + blockIdx.x);
}

static double mean_candidates(const CellGrid& g, int n) {
  return (double)n / ((double)g.nb[0] * g.nb[1] * g.nb[2]) * (2 * g.reach[0] + 1) * (2 * g.reach[1] + 1) *
         (2 * g.reach[2] + 1);
}
static bool mostly_dense(const CellGrid& g, int n) { return mean_candidates(g, n) + 32 > kCnFloat; }

int64_t cn_max_blocks(int64_t bins) { return 4 * 148 + bins; }   // bins * ceil(4 * 148 / bins) at most

int launch_cn_c6_cells(const CellGrid& g, int n, const CellList& cl, const int32_t* species, const Tables* tab,
                       const double* eigvecs, int R, double* cn, double* c6, double* dc6,
                       const RankOut& ro, double* self_part, int* n_self_blocks, const HitStore& hs, cudaStream_t s) {
  const int K = g.nb[0] * g.nb[1] * g.nb[2];
  // stage: the mean number of candidates and half as much again, within kCnSmem
  const double want = 1.5 * mean_candidates(g, n) + 64;
  const int each = hs.is_double || mostly_dense(g, n) ? 36 : 20;   // double4 or float4, and the id
  int stage = want * each < kCnSmem ? ((int)want + 3) / 4 * 4 * each : kCnSmem / (4 * each) * (4 * each);
  if (!hs.is_double && each == 20 && stage > kCnFloat * 20) stage = kCnFloat * 20;
  // few bins: several CTAs share a bin's atoms (each stages the candidates) until the chip has four
  // CTAs per SM or every warp one atom. 27 bins of 24 atoms (648 SiO2 atoms, float64): 40 -> 9 us.
  const int per_bin = (n + K - 1) / K;
  int nsplit = (4 * 148 + K - 1) / K;
  const int most = (per_bin + kCnWarps - 1) / kCnWarps;
  if (nsplit > most) nsplit = most;
  if (nsplit < 1) nsplit = 1;
  const int grid = K * nsplit;
  // Where the bins alone fill the chip, the factors take a kernel of their own (8 us): the CN kernel
  // runs more CTAs per SM without them (139,968 atoms, mixed, both: 226 us with, 189 us without).
  const bool with_c6 = nsplit > 1 || K < 4 * 148;
  auto launch = [&](auto kern, auto hl) -> int {
    const int rc = stage > kCnSmemPlain ? allow_dynamic_smem(kern, kCnSmem) : FD3_OK;
    if (rc) return rc;
    kern<<<grid, 32 * kCnWarps, stage, s>>>(to_dev(g), stage, nsplit, cl.bin_start, cl.xs, cl.meta, cl.off, tab,
                                            eigvecs, R, cn, c6, dc6, hl, ro, self_part);
    FD3_LAUNCHED();
    return FD3_OK;
  };
  int rc;
  if (hs.is_double) {
    const HitList<double> hl{hs.j, (double4*)hs.ad, hs.n, hs.cap};
    rc = with_c6 ? launch(k_cn_bins<double, true>, hl) : launch(k_cn_bins<double, false>, hl);
  } else {
    const HitList<float> hl{hs.j, (float4*)hs.ad, hs.n, hs.cap};
    rc = with_c6 ? launch(k_cn_bins<float, true>, hl) : launch(k_cn_bins<float, false>, hl);
  }
  *n_self_blocks = grid;
  if (rc || with_c6) return rc;
  return launch_c6_atoms(n, species, tab, eigvecs, R, cn, c6, dc6, ro, self_part, n_self_blocks, s);
}

// One atom's recorded pairs of a dense bin of the mixed form, in float64; this lane's share.
__device__ __noinline__ PairSums cn_adjoint_atom_exact(const GridDev& g, const double4* __restrict__ xs,
                                                       const int4* __restrict__ meta, const double* __restrict__ gcn,
                                                       const HitList<float>& hl, int t, int nh) {
  double w0, w1, w2;
  wrapped_pos(g, xs[t], meta[t], w0, w1, w2);
  const double gi = gcn[meta[t].w];
  const size_t hb = (size_t)t * hl.cap;
  PairSums p{0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 2
  for (int e = threadIdx.x & 31; e < nh; e += 32) {
    const float4 q = hl.ad[hb + e];
    const double gj = gcn[hl.j[hb + e]];
    const double a = __hiloint2double(__float_as_int(q.y), __float_as_int(q.x));
    const int u = __float_as_int(q.z), im = __float_as_int(q.w);
    const double4 xj = xs[u];
    const int4 mj = meta[u];
    const double S0 = (im & 255) - 128 - mj.x, S1 = (im >> 8 & 255) - 128 - mj.y, S2 = (im >> 16) - 128 - mj.z;
    const double v0 = (xj.x + S0 * g.cell[0] + S1 * g.cell[3] + S2 * g.cell[6] - w0) * kAngToBohr;
    const double v1 = (xj.y + S0 * g.cell[1] + S1 * g.cell[4] + S2 * g.cell[7] - w1) * kAngToBohr;
    const double v2 = (xj.z + S0 * g.cell[2] + S1 * g.cell[5] + S2 * g.cell[8] - w2) * kAngToBohr;
    const double w = (gi + gj) * a;
    p.f0 -= w * v0;
    p.f1 -= w * v1;
    p.f2 -= w * v2;
    const double b = gi * a;
    p.xx += b * v0 * v0; p.xy += b * v0 * v1; p.xz += b * v0 * v2;
    p.yy += b * v1 * v1; p.yz += b * v1 * v2; p.zz += b * v2 * v2;
  }
  return p;
}

// One atom without a float record (hl.n[t] = nh < 0): its float64 records, or the cell list again.
template <typename TE, bool EXACT>
__device__ __forceinline__ PairSums cn_adjoint_atom_rest(const GridDev& g, const int* __restrict__ bin_start,
                                                         const double4* __restrict__ xs,
                                                         const int4* __restrict__ meta, const int4* __restrict__ off,
                                                         const Tables* __restrict__ tab,
                                                         const double* __restrict__ gcn, const HitList<TE>& hl, int t,
                                                         int nh) {
  if constexpr (EXACT)
    if (nh <= -2) return cn_adjoint_atom_exact(g, xs, meta, gcn, hl, t, -2 - nh);
  return cn_adjoint_atom_global(g, bin_start, xs, meta, off, tab, gcn, t);
}

// CN adjoint: dE/dx_i = -sum_(j,S) (g_i + g_j) f'(r) d / r  (the list is symmetric), and the
// strain virial W_ab = sum_i g_i sum_(j,S) f'(r) d_a d_b / r  (Bohr, Hartree). The force written
// is out_scale * (mesh gradient already in grad + CN gradient). One warp per atom streams the
// atom's recorded pairs; the others (n < 0, see cn_adjoint_atom_rest) are taken afterwards.
// A stale cell (ci->stale, see k_cellinfo) makes every force NaN.
// The kernel is bound by the latency of its dependent loads (count -> atom -> records -> g_j), so
// a warp fetches the next atom's count and index while it works on this one, issues all of a
// batch of 96 records' loads before the g_j loads that depend on them, and reads the atom's mesh
// gradient at the start. Lane l still sums the records l, l + 32, ... in that order.
//
// REST: the same kernel takes the atoms with n < 0, for the sizes where another launch costs more
// than the registers of that path (up to kAdjointOne atoms; 5,184: 16 us against 19, 139,968: 104
// against 78); otherwise k_cn_adjoint_rest follows. EXACT: from the float64 records,
// where the mixed form's bins are dense on average (otherwise its few dense ones are traversed again); the work
// is in the calls then, which spill at four CTAs per SM (12,000 HCNO atoms: call 782 us with four, 776 with three).
template <typename TE, bool REST, bool EXACT = false>
__global__ void __launch_bounds__(256, EXACT ? 3 : 4) k_cn_adjoint(const __grid_constant__ GridDev g, int n, const int* __restrict__ bin_start,
                                                        const double4* __restrict__ xs,
                                                        const int4* __restrict__ meta, const int4* __restrict__ off,
                                                        const Tables* __restrict__ tab,
                                                        const CellInfo* __restrict__ ci,
                                                        const double* __restrict__ gcn, double* __restrict__ grad,
                                                        double out_scale, double* __restrict__ vir_part,
                                                        HitList<TE> hl) {
  using V4 = typename Vec4<TE>::type;
  constexpr int kU = 3;   // records per lane per batch
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int stride = gridDim.x * kWarpsPerBlock;
  double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  int t = blockIdx.x * kWarpsPerBlock + wid;
  int nh_next = t < n ? hl.n[t] : -1;
  int i_next = t < n ? meta[t].w : 0;
  if (ci->stale != 0.0) out_scale = __longlong_as_double(0x7ff8000000000000LL);
  // grid-stride over atoms: the block's virial is reduced once, after all its atoms
  bool rest = false;
  for (; t < n; t += stride) {
    const int nh = nh_next, i = i_next;
    if (t + stride < n) {
      nh_next = hl.n[t + stride];
      i_next = meta[t + stride].w;
    }
    if (nh < 0) {
      rest = true;
    } else {
      const double gi = gcn[i];
      const double gq = lane < 3 ? grad[3 * i + lane] : 0.0;
      double f0 = 0, f1 = 0, f2 = 0;
      const size_t hb = (size_t)t * hl.cap;
      for (int e0 = 0; e0 < nh; e0 += 32 * kU) {
        V4 r4[kU];
        int jj[kU];
        double gj[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int e = e0 + 32 * u + lane;
          if (e < nh) {
            r4[u] = hl.ad[hb + e];
            jj[u] = hl.j[hb + e];
          } else {
            r4[u] = V4{0, 0, 0, 0};
            jj[u] = -1;
          }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) gj[u] = jj[u] >= 0 ? gcn[jj[u]] : 0.0;
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          if (jj[u] < 0) continue;
          const double a = (double)r4[u].x, v0 = (double)r4[u].y, v1 = (double)r4[u].z, v2 = (double)r4[u].w;
          const double w = (gi + gj[u]) * a;
          f0 -= w * v0;
          f1 -= w * v1;
          f2 -= w * v2;
          const double bb = gi * a;
          v[0] += bb * v0 * v0; v[1] += bb * v0 * v1; v[2] += bb * v0 * v2;
          v[4] += bb * v1 * v1; v[5] += bb * v1 * v2; v[8] += bb * v2 * v2;
        }
      }
      f0 = warp_sum(f0);
      f1 = warp_sum(f1);
      f2 = warp_sum(f2);
      const double q0 = __shfl_sync(0xffffffffu, gq, 0), q1 = __shfl_sync(0xffffffffu, gq, 1),
                   q2 = __shfl_sync(0xffffffffu, gq, 2);
      if (lane == 0) {
        grad[3 * i] = out_scale * (q0 + f0);
        grad[3 * i + 1] = out_scale * (q1 + f1);
        grad[3 * i + 2] = out_scale * (q2 + f2);
      }
    }
  }
  // the others in a loop of their own: the calls would cost the loop above its registers
  if (REST && rest)
    for (t = blockIdx.x * kWarpsPerBlock + wid; t < n; t += stride) {
      const int nh = hl.n[t];
      if (nh >= 0) continue;
      const int i = meta[t].w;
      const PairSums p = cn_adjoint_atom_rest<TE, EXACT>(g, bin_start, xs, meta, off, tab, gcn, hl, t, nh);
      v[0] += p.xx; v[1] += p.xy; v[2] += p.xz;
      v[4] += p.yy; v[5] += p.yz; v[8] += p.zz;
      const double f0 = warp_sum(p.f0), f1 = warp_sum(p.f1), f2 = warp_sum(p.f2);
      if (lane == 0) {
        grad[3 * i] = out_scale * (grad[3 * i] + f0);
        grad[3 * i + 1] = out_scale * (grad[3 * i + 1] + f1);
        grad[3 * i + 2] = out_scale * (grad[3 * i + 2] + f2);
      }
    }
  v[3] = v[1];
  v[6] = v[2];
  v[7] = v[5];
  block_sum_store<9>(v, vir_part + 9 * blockIdx.x);
}

// The atoms with n < 0, after k_cn_adjoint<TE, false>. A warp reads the counts of the 32 atoms that
// are its own (a grid stride apart) at once: outside the mixed form's dense boxes almost always none is.
template <typename TE>
__global__ void __launch_bounds__(256) k_cn_adjoint_rest(const __grid_constant__ GridDev g, int n,
                                                        const int* __restrict__ bin_start,
                                                        const double4* __restrict__ xs, const int4* __restrict__ meta,
                                                        const int4* __restrict__ off, const Tables* __restrict__ tab,
                                                        const CellInfo* __restrict__ ci,
                                                        const double* __restrict__ gcn, double* __restrict__ grad,
                                                        double out_scale, double* __restrict__ vir_part,
                                                        HitList<TE> hl) {
  const int lane = threadIdx.x & 31, stride = gridDim.x * kWarpsPerBlock;
  double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (ci->stale != 0.0) out_scale = __longlong_as_double(0x7ff8000000000000LL);
  for (int64_t t0 = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); t0 < n; t0 += 32 * (int64_t)stride) {
    const int64_t own = t0 + (int64_t)lane * stride;
    const int own_n = own < n ? hl.n[own] : 0;
    unsigned todo = __ballot_sync(0xffffffffu, own_n < 0);
    for (; todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1, nh = __shfl_sync(0xffffffffu, own_n, src);
      const int t = (int)(t0 + (int64_t)src * stride), i = meta[t].w;
      const PairSums p = cn_adjoint_atom_rest<TE, sizeof(TE) == 4>(g, bin_start, xs, meta, off, tab, gcn, hl, t, nh);
      v[0] += p.xx; v[1] += p.xy; v[2] += p.xz;
      v[4] += p.yy; v[5] += p.yz; v[8] += p.zz;
      const double f0 = warp_sum(p.f0), f1 = warp_sum(p.f1), f2 = warp_sum(p.f2);
      if (lane == 0) {
        grad[3 * i] = out_scale * (grad[3 * i] + f0);
        grad[3 * i + 1] = out_scale * (grad[3 * i + 1] + f1);
        grad[3 * i + 2] = out_scale * (grad[3 * i + 2] + f2);
      }
    }
  }
  v[3] = v[1];
  v[6] = v[2];
  v[7] = v[5];
  block_sum_store<9>(v, vir_part + 9 * blockIdx.x);
}

constexpr int kAdjointOne = 16384;
constexpr int kRestBlocks = 148 * 2;

int launch_cn_adjoint_cells(const CellGrid& g, int n, const CellList& cl, const Tables* tab, const CellInfo* ci,
                            const double* gcn, double* grad, double out_scale, double* vir_part, int* n_blocks,
                            const HitStore& hs, cudaStream_t s) {
  const int need = (n + kWarpsPerBlock - 1) / kWarpsPerBlock;
  const int blocks = need < 148 * 8 ? need : 148 * 8;   // resident grid, grid-stride over atoms
  *n_blocks = blocks;
  if (blocks == 0) return FD3_OK;
  const GridDev gd = to_dev(g);
  const bool one = n <= kAdjointOne;
  auto launch = [&](auto kern, int grid, double* part, auto hl) -> int {
    kern<<<grid, 32 * kWarpsPerBlock, 0, s>>>(gd, n, cl.bin_start, cl.xs, cl.meta, cl.off, tab, ci, gcn, grad,
                                              out_scale, part, hl);
    FD3_LAUNCHED();
    return FD3_OK;
  };
  auto both = [&](auto kern_one, auto kern, auto kern_rest, auto hl) -> int {
    if (one) return launch(kern_one, blocks, vir_part, hl);
    const int rc = launch(kern, blocks, vir_part, hl);
    if (rc) return rc;
    *n_blocks = blocks + kRestBlocks;
    return launch(kern_rest, kRestBlocks, vir_part + 9 * (size_t)blocks, hl);
  };
  if (hs.is_double)
    return both(k_cn_adjoint<double, true>, k_cn_adjoint<double, false>, k_cn_adjoint_rest<double>,
                HitList<double>{hs.j, (double4*)hs.ad, hs.n, hs.cap});
  return both(mostly_dense(g, n) ? k_cn_adjoint<float, true, true> : k_cn_adjoint<float, true>,
              k_cn_adjoint<float, false>, k_cn_adjoint_rest<float>,
              HitList<float>{hs.j, (float4*)hs.ad, hs.n, hs.cap});
}

// ------------------------------------------------------------------ edge-list path
// ------------------------------------------------------------------ edge-list path, fixed order
// Edges sorted by source and by destination, ids ascending within an atom (see counting_sort); both
// sorts share each launch. An edge list usually comes sorted by source (every neighbour search emits it
// row by row): the first kernel notes whether it does, the second then writes the source segments where
// the source changes (at most N writes in all, since the sources ascend) and the source half of the
// other steps has nothing to do.
//
// An edge whose source or destination is outside 0..n-1 raises *bad and is keyed to bucket e mod n (so no
// bucket grows with the number of bad edges); every consumer re-checks the range and skips it.
// 1.2 M edges sorted by source, 20,736 atoms: CN stage 150 us; with one sort after the other 224.
__device__ __forceinline__ int edge_key(const int64_t* __restrict__ src, const int64_t* __restrict__ dst, int64_t e,
                                        int n, int& kd, bool& ok) {
  const int64_t i = src[e], j = dst[e];
  ok = i >= 0 && i < n && j >= 0 && j < n;
  const int spill = (int)(e % n);
  kd = ok ? (int)j : spill;
  return ok ? (int)i : spill;
}

__global__ void __launch_bounds__(256) k_edge_keys(int64_t ne, int n, const int64_t* __restrict__ src,
                                                  const int64_t* __restrict__ dst, EdgeIndex ei) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  int kd, kd_prev;
  bool ok, ok_prev;
  const int ks = edge_key(src, dst, e, n, kd, ok);
  const int prev = e > 0 ? edge_key(src, dst, e - 1, n, kd_prev, ok_prev) : -1;
  ei.ks[e] = ks;
  ei.kd[e] = kd;
  ei.ord_d[e] = atomicAdd(&ei.cnt_d[kd], 1);   // arrival slot, until the last step
  if (!ok) *ei.bad = 1;
  if (ks < prev) *ei.unsorted = 1;
}

// Longer runs of atoms without edges are written by the whole CTA (two edges in the middle of 200,000 atoms: CN
// stage 1.0 ms with one thread writing them, 0.31 now; the same edges in descending order 0.30).
__global__ void __launch_bounds__(256) k_edge_slots(int ne, int n, EdgeIndex ei) {
  constexpr int kShort = 32;
  __shared__ int gaps, lo[257], hi[257], val[257];   // a gap before each edge, and one after the last
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (*ei.unsorted != 0) {
    if (e < ne) ei.ord_s[e] = atomicAdd(&ei.cnt_s[ei.ks[e]], 1);
    return;
  }
  if (threadIdx.x == 0) gaps = 0;
  __syncthreads();
  auto fill = [&](int a, int b, int v) {   // st_s[a .. b] = v
    if (b - a >= kShort) {
      const int k = atomicAdd(&gaps, 1);
      lo[k] = a;
      hi[k] = b;
      val[k] = v;
    } else {
      for (; a <= b; ++a) ei.st_s[a] = v;
    }
  };
  if (e < ne) {
    const int ks = ei.ks[e];
    ei.ord_s[e] = e;
    fill(e > 0 ? ei.ks[e - 1] + 1 : 0, ks, e);
    if (e == ne - 1) fill(ks + 1, n, ne);
  }
  __syncthreads();
  for (int k = 0; k < gaps; ++k)
    for (int a = lo[k] + (int)threadIdx.x; a <= hi[k]; a += blockDim.x) ei.st_s[a] = val[k];
}

__global__ void __launch_bounds__(kScanThreads) k_edge_scan(int n, EdgeIndex ei) {
  if (blockIdx.x == 0)
    scan_exclusive_block(ei.cnt_d, n, ei.st_d);
  else if (*ei.unsorted != 0)
    scan_exclusive_block(ei.cnt_s, n, ei.st_s);
}

// blockIdx.y: 0 destinations, 1 sources
__global__ void __launch_bounds__(256) k_edge_scatter(int ne, EdgeIndex ei) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne || (blockIdx.y == 1 && *ei.unsorted == 0)) return;
  if (blockIdx.y == 0)
    ei.arr_d[ei.st_d[ei.kd[e]] + ei.ord_d[e]] = e;
  else
    ei.arr_s[ei.st_s[ei.ks[e]] + ei.ord_s[e]] = e;
}

__global__ void __launch_bounds__(256) k_edge_rank(int ne, EdgeIndex ei) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= ne || (blockIdx.y == 1 && *ei.unsorted == 0)) return;
  const int* arr = blockIdx.y == 0 ? ei.arr_d : ei.arr_s;
  const int* st = blockIdx.y == 0 ? ei.st_d : ei.st_s;
  const int e = arr[p], k = (blockIdx.y == 0 ? ei.kd : ei.ks)[e];
  (blockIdx.y == 0 ? ei.ord_d : ei.ord_s)[ranked_place(arr, e, st[k], st[k + 1])] = e;
}

int launch_edge_index(int64_t n_edges, int n, const int64_t* src, const int64_t* dst, const EdgeIndex& ei,
                      cudaStream_t s) {
  // bad, unsorted and both count arrays in one fill; without edges every segment is empty
  FD3_CUDA(cudaMemsetAsync(ei.bad, 0, sizeof(int) * (2 + 2 * (size_t)n), s));
  if (n_edges <= 0) {
    FD3_CUDA(cudaMemsetAsync(ei.st_s, 0, sizeof(int) * (n + 1), s));
    FD3_CUDA(cudaMemsetAsync(ei.st_d, 0, sizeof(int) * (n + 1), s));
    return FD3_OK;
  }
  const int tb = 256, ne = (int)n_edges, nb = (int)((n_edges + tb - 1) / tb);
  k_edge_keys<<<nb, tb, 0, s>>>(n_edges, n, src, dst, ei);
  FD3_LAUNCHED();
  k_edge_slots<<<nb, tb, 0, s>>>(ne, n, ei);
  FD3_LAUNCHED();
  k_edge_scan<<<2, kScanThreads, 0, s>>>(n, ei);
  FD3_LAUNCHED();
  k_edge_scatter<<<dim3(nb, 2), tb, 0, s>>>(ne, ei);
  FD3_LAUNCHED();
  k_edge_rank<<<dim3(nb, 2), tb, 0, s>>>(ne, ei);
  FD3_LAUNCHED();
  return FD3_OK;
}

// CN of atom a: the sum of the smooth-cutoff function over its source edges in edge order
// (core.py:323-386, index_add_ on edge_index[0]); one warp per atom, lanes over the edges, a
// fixed butterfly reduction -- the same result on every run. NaN for every atom when an edge
// index was out of range (the range check the reference leaves to torch indexing). Edges with
// |r|^2 >= mask_r2 contribute nothing (mask_r2 = +inf: every edge counts, as in the reference).
__global__ void __launch_bounds__(256) k_cn_edges_seg(int n, int64_t ne, const int* __restrict__ st,
                                                     const int* __restrict__ ord, const double* __restrict__ x,
                                                     const int32_t* __restrict__ species,
                                                     const int64_t* __restrict__ src, const int64_t* __restrict__ dst,
                                                     const double* __restrict__ sh, const Tables* __restrict__ tab,
                                                     double mask_r2, const int* __restrict__ bad,
                                                     double* __restrict__ cn) {
  const int lane = threadIdx.x & 31;
  const int a = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (a >= n) return;
  const double rca = tab->rcov[species[a]];
  double sum = 0.0;
  for (int p = st[a] + lane; p < st[a + 1]; p += 32) {
    const int e = ord[p];
    const int64_t i = src[e], j = dst[e];
    if (i != a || j < 0 || j >= n) continue;
    const double v0 = x[3 * j] - x[3 * i] + sh[3 * (int64_t)e];
    const double v1 = x[3 * j + 1] - x[3 * i + 1] + sh[3 * (int64_t)e + 1];
    const double v2 = x[3 * j + 2] - x[3 * i + 2] + sh[3 * (int64_t)e + 2];
    const double r2 = v0 * v0 + v1 * v1 + v2 * v2;
    if (r2 >= mask_r2) continue;
    double f, df;
    cn_edge(sqrt(r2), rca + tab->rcov[species[j]], tab->r_cut, f, df);
    sum += f;
  }
  sum = warp_sum(sum);
  if (lane == 0) cn[a] = *bad ? __longlong_as_double(0x7ff8000000000000LL) : sum;
}

int launch_cn_edges_seg(int64_t n_edges, int n, const double* pos, const int32_t* species, const int64_t* src,
                        const int64_t* dst, const double* shift, const Tables* tab, double mask_r2,
                        const EdgeIndex& ei, double* cn, cudaStream_t s) {
  const int wpb = 8;
  k_cn_edges_seg<<<(n + wpb - 1) / wpb, 32 * wpb, 0, s>>>(n, n_edges, ei.st_s, ei.ord_s, pos, species, src, dst,
                                                          shift, tab, mask_r2, ei.bad, cn);
  FD3_LAUNCHED();
  return FD3_OK;
}

// dE/dshift of every edge, g_e = dE/dCN_i f'(r) v / r (zero for an edge out of range).
__global__ void __launch_bounds__(256) k_edge_grad(int64_t ne, int n, const double* __restrict__ x,
                                                  const int32_t* __restrict__ species, const int64_t* __restrict__ src,
                                                  const int64_t* __restrict__ dst, const double* __restrict__ sh,
                                                  const Tables* __restrict__ tab, double mask_r2,
                                                  const double* __restrict__ gcn, double* __restrict__ gshift) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int64_t i = src[e], j = dst[e];
  double g0 = 0, g1 = 0, g2 = 0;
  if (i >= 0 && i < n && j >= 0 && j < n) {
    const double v0 = x[3 * j] - x[3 * i] + sh[3 * e];
    const double v1 = x[3 * j + 1] - x[3 * i + 1] + sh[3 * e + 1];
    const double v2 = x[3 * j + 2] - x[3 * i + 2] + sh[3 * e + 2];
    const double r2 = v0 * v0 + v1 * v1 + v2 * v2;
    const double r = sqrt(r2);
    double f, df;
    cn_edge(r, tab->rcov[species[i]] + tab->rcov[species[j]], tab->r_cut, f, df);
    if (r > 1e-6 && r2 < mask_r2) {
      const double a = gcn[i] * df / r;
      g0 = a * v0;
      g1 = a * v1;
      g2 = a * v2;
    }
  }
  gshift[3 * e] = g0;
  gshift[3 * e + 1] = g1;
  gshift[3 * e + 2] = g2;
}

// dE/dpos_a += sum over edges into a of g_e - sum over edges out of a of g_e, each in edge order.
__global__ void __launch_bounds__(256) k_edge_grad_atoms(int n, const int* __restrict__ st_s,
                                                        const int* __restrict__ ord_s, const int* __restrict__ st_d,
                                                        const int* __restrict__ ord_d,
                                                        const double* __restrict__ gshift, double* __restrict__ gpos) {
  const int lane = threadIdx.x & 31;
  const int a = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (a >= n) return;
  double g[3] = {0.0, 0.0, 0.0};
  for (int p = st_d[a] + lane; p < st_d[a + 1]; p += 32) {
    const int64_t e = ord_d[p];
#pragma unroll
    for (int c = 0; c < 3; ++c) g[c] += gshift[3 * e + c];
  }
  for (int p = st_s[a] + lane; p < st_s[a + 1]; p += 32) {
    const int64_t e = ord_s[p];
#pragma unroll
    for (int c = 0; c < 3; ++c) g[c] -= gshift[3 * e + c];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) g[c] = warp_sum(g[c]);
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c) gpos[3 * (int64_t)a + c] += g[c];
  }
}

int launch_cn_adjoint_edges_seg(int64_t n_edges, int n, const double* pos, const int32_t* species,
                                const int64_t* src, const int64_t* dst, const double* shift, const Tables* tab,
                                double mask_r2, const double* gcn, const EdgeIndex& ei, double* gpos,
                                double* gshift, cudaStream_t s) {
  if (n_edges > 0) {
    const int tb = 256;
    k_edge_grad<<<(unsigned)((n_edges + tb - 1) / tb), tb, 0, s>>>(n_edges, n, pos, species, src, dst, shift, tab,
                                                                   mask_r2, gcn, gshift);
    FD3_LAUNCHED();
  }
  const int wpb = 8;
  k_edge_grad_atoms<<<(n + wpb - 1) / wpb, 32 * wpb, 0, s>>>(n, ei.st_s, ei.ord_s, ei.st_d, ei.ord_d, gshift, gpos);
  FD3_LAUNCHED();
  return FD3_OK;
}


// Softmax interpolation over the 7 reference CNs and the rank-r factors
// c_r = sum_p w_p V[s, p, r] (core.py:449-478, 525-532), their CN derivative (times the
// cncorr slope) and the self term sum_r lambda_r c_r^2 phi_ss(0) (core.py:545-550). One thread
// per atom; cn holds the raw CN on entry and the corrected CN on exit.
__global__ void __launch_bounds__(256) k_c6_atoms(int n, const int32_t* __restrict__ species,
                                                 const Tables* __restrict__ tab, const double* __restrict__ V, int R,
                                                 double* __restrict__ cn, double* __restrict__ c6,
                                                 double* __restrict__ dc6, RankOut ro,
                                                 double* __restrict__ self_part) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double selfv = 0.0;
  if (i < n) {
    const int s = species[i];
    double cnv = cn[i], slope = 1.0;
    if (tab->has_cncorr) {
      slope = tab->cncorr[2 * s + 1];
      cnv = slope * cnv + tab->cncorr[2 * s + 0];
    }
    double lg[7], dl[7];
    double mx = -INFINITY;
#pragma unroll
    for (int p = 0; p < 7; ++p) {
      const double ref = tab->cnref[7 * s + p];
      const double diff = cnv - ref;
      const bool ok = ref != -1.0;
      lg[p] = ok ? -4.0 * (diff * diff) : -INFINITY;
      dl[p] = ok ? -8.0 * diff : 0.0;
      mx = fmax(mx, lg[p]);
    }
    double sum = 0.0;
#pragma unroll
    for (int p = 0; p < 7; ++p) {
      lg[p] = lg[p] == -INFINITY ? 0.0 : exp(lg[p] - mx);
      sum += lg[p];
    }
    const double inv = 1.0 / sum;
    double dlbar = 0.0;
#pragma unroll
    for (int p = 0; p < 7; ++p) {
      lg[p] *= inv;                   // softmax weight w_p
      dlbar += lg[p] * dl[p];
    }
    for (int r = 0; r < R; ++r) {
      double c = 0.0, d = 0.0;
#pragma unroll
      for (int p = 0; p < 7; ++p) {
        const double v = V[(7 * s + p) * R + r];
        c += lg[p] * v;
        d += lg[p] * (dl[p] - dlbar) * v;
      }
      c6[(size_t)i * R + r] = c;
      dc6[(size_t)i * R + r] = slope * d;
      ro.put(i, r, R, c);
      selfv += tab->eigs[r] * c * c * tab->selfcont[s];
    }
    cn[i] = cnv;
  }
  double v1[1] = {selfv};
  block_sum_store<1>(v1, self_part + blockIdx.x);
}

int launch_c6_atoms(int n, const int32_t* species, const Tables* tab, const double* eigvecs, int R,
                    const double* cn, double* c6, double* dc6, const RankOut& ro, double* self_part,
                    int* n_self_blocks, cudaStream_t s) {
  const int blocks = (n + 255) / 256;
  *n_self_blocks = blocks;
  if (blocks == 0) return FD3_OK;
  k_c6_atoms<<<blocks, 256, 0, s>>>(n, species, tab, eigvecs, R, const_cast<double*>(cn), c6, dc6, ro,
                                     self_part);
  FD3_LAUNCHED();
  return FD3_OK;
}


// ------------------------------------------------------------------ neighbour export
// One warp per atom. The runs of bins around it (two per (dx, dy) at most: a z range that fits the
// grid wraps once) are laid out at once by the lanes, so that the candidates form one numbered
// sequence, in the order of visit_neighbors, and every load of a round is independent of the last
// round's. (Walking the runs one by one waits for bin_start and then for its candidates 18 times per atom.)
// Grids whose runs do not fit the table (cells narrower than the search) take visit_neighbors.
constexpr int kNbrRuns = 64;
struct NbrRuns {
  int pref[kNbrRuns + 1], a0[kNbrRuns], S0[kNbrRuns], S1[kNbrRuns], S2[kNbrRuns];
};
__device__ __forceinline__ bool nbr_runs_fit(const GridDev& g) {
  return 2 * (2 * g.reach[0] + 1) * (2 * g.reach[1] + 1) <= kNbrRuns && 2 * g.reach[2] + 1 <= g.nb[2];
}

// fn as in visit_neighbors, without the candidate slot and the vector.
template <class Fn>
__device__ __forceinline__ void visit_runs(const GridDev& g, const int* __restrict__ bin_start,
                                           const double4* __restrict__ xs, const int4* __restrict__ meta, int i,
                                           double4 xi, int4 offi, NbrRuns& rt, Fn&& fn) {
  const int lane = threadIdx.x & 31;
  const int ny = 2 * g.reach[1] + 1, npair = (2 * g.reach[0] + 1) * ny;
  const int bz = offi.w % g.nb[2], by = (offi.w / g.nb[2]) % g.nb[1], bx = offi.w / (g.nb[2] * g.nb[1]);
  int len0 = 0, len1 = 0;
  if (lane < npair) {
    const int cx = bx + lane / ny - g.reach[0], cy = by + lane % ny - g.reach[1];
    const int sx = floordiv(cx, g.nb[0]), sy = floordiv(cy, g.nb[1]);
    const int row = ((cx - sx * g.nb[0]) * g.nb[1] + (cy - sy * g.nb[1])) * g.nb[2];
    const int zs = bz - g.reach[2], nz = 2 * g.reach[2] + 1;
    const int sz = floordiv(zs, g.nb[2]), wz = zs - sz * g.nb[2];
    const int n0 = g.nb[2] - wz < nz ? g.nb[2] - wz : nz;   // bins before the wrap
    const int a = bin_start[row + wz], b = bin_start[row + wz + n0];
    const int c = n0 < nz ? bin_start[row] : 0, d = n0 < nz ? bin_start[row + nz - n0] : 0;
    len0 = b - a;
    len1 = d - c;
    rt.a0[2 * lane] = a;
    rt.a0[2 * lane + 1] = c;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      rt.S0[2 * lane + u] = sx + offi.x;
      rt.S1[2 * lane + u] = sy + offi.y;
      rt.S2[2 * lane + u] = sz + u + offi.z;
    }
  }
  int incl = len0 + len1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane < npair) {
    rt.pref[2 * lane] = incl - len0 - len1;
    rt.pref[2 * lane + 1] = incl - len1;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  __syncwarp();
  const int last = 2 * npair - 1;
#pragma unroll 2
  for (int c0 = 0; c0 < total; c0 += 32) {
    const int c = c0 + lane;
    bool hit = false;
    int j = 0, S0 = 0, S1 = 0, S2 = 0;
    if (c < total) {
      int lo = 0, hi = last;   // last run with pref <= c
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (rt.pref[mid] <= c) lo = mid; else hi = mid - 1;
      }
      const int u = rt.a0[lo] + (c - rt.pref[lo]);
      const double4 xj = xs[u];
      const int4 mj = meta[u];
      j = mj.w;
      S0 = rt.S0[lo] - mj.x;
      S1 = rt.S1[lo] - mj.y;
      S2 = rt.S2[lo] - mj.z;
      double d0, d1, d2;
      hit = pair_inside(g, xj.x, xj.y, xj.z, xi.x, xi.y, xi.z, S0, S1, S2, d0, d1, d2) &&
            !(j == i && S0 == 0 && S1 == 0 && S2 == 0);
    }
    fn(hit, j, S0, S1, S2);
  }
  __syncwarp();
}

// Number of neighbours of the warp's atom, and the same traversal writing them from row_start[i]; nothing is
// written outside the outputs' `room` pairs, whatever the row starts hold.
template <bool FILL>
__global__ void __launch_bounds__(256) k_nbr(const __grid_constant__ GridDev g, int n,
                                            const int* __restrict__ bin_start, const double4* __restrict__ xs,
                                            const int4* __restrict__ meta, const int4* __restrict__ off,
                                            int* __restrict__ counts, const int* __restrict__ row_start,
                                            int64_t* __restrict__ src, int64_t* __restrict__ dst,
                                            int32_t* __restrict__ shift, unsigned room) {
  __shared__ NbrRuns runs[kWarpsPerBlock];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int t = blockIdx.x * kWarpsPerBlock + wid;
  if (t >= n) return;
  const double4 xi = xs[t];
  const int i = meta[t].w;
  int pos = FILL ? row_start[i] : 0;
  auto take = [&](bool hit, int j, int S0, int S1, int S2) {
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    const int k = pos + __popc(m & ((1u << lane) - 1u));
    if (FILL && hit && (unsigned)k < room) {
      src[k] = i;
      dst[k] = j;
      int32_t* sh = shift + 3 * (size_t)k;
      sh[0] = S0;
      sh[1] = S1;
      sh[2] = S2;
    }
    pos += __popc(m);
  };
  if (nbr_runs_fit(g))
    visit_runs(g, bin_start, xs, meta, i, xi, off[i], runs[wid], take);
  else
    visit_neighbors(g, bin_start, xs, meta, i, xi.x, xi.y, xi.z, off[i],
                    [&](bool hit, int, int j, int S0, int S1, int S2, double, double, double) {
                      take(hit, j, S0, S1, S2);
                    });
  if (!FILL && lane == 0) counts[i] = pos;
}

// ------------------------------------------------------------------ direct pair sum (float64)
// The accuracy oracle's lattice sum on the device: over every image pair (i, j, n) closer than
// the grid's cutoff (r_direct) except i = j at n = 0, with C6_ij = sum_r lambda_r c_ir c_jr
// (the plan's low-rank factors) and the BJ-damped kernel of src/fourierd3/pair_pot.py:64,
//   phi(r) = s6 / (r^6 + R0^6) + 3 s8 qq / (r^8 + R0^8),  E = -1/2 sum C6 phi   (Bohr, Hartree).
// Warp per atom i over the bin-sorted atoms: e_i = sum_j C6 phi, dE/dc_ir = -lambda_r sum_j
// c_jr phi, dE/dx_i = sum_j C6 (phi'/r) d (d = x_j + n - x_i; each pair is seen from both ends),
// and per block e = sum_i e_i and the virial -1/2 sum C6 (phi'/r) d_a d_b (6 components).
__global__ void __launch_bounds__(256) k_direct_pairs(GridDev g, int n, const int* __restrict__ bin_start,
                                                     const double4* __restrict__ xs, const int4* __restrict__ meta,
                                                     const int4* __restrict__ off, const double* __restrict__ c6,
                                                     const Tables* __restrict__ tab, int R, int S,
                                                     const GreenPair* __restrict__ gp, double* __restrict__ dEdc,
                                                     double* __restrict__ grad, double* __restrict__ part) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int t = blockIdx.x * kWarpsPerBlock + wid;
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};   // e, virial xx xy xz yy yz zz
  if (t < n) {
    const double4 xi = xs[t];
    const int i = meta[t].w;
    const int Xi = (int)xi.w;
    const double s6 = tab->s6, s8 = tab->s8;
    double ci[8], gc[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      ci[r] = r < R ? tab->eigs[r] * c6[(size_t)i * R + r] : 0.0;
      gc[r] = 0.0;
    }
    double e = 0.0, g0 = 0.0, g1 = 0.0, g2 = 0.0, v[6] = {0, 0, 0, 0, 0, 0};
    visit_neighbors(g, bin_start, xs, meta, i, xi.x, xi.y, xi.z, off[i],
                    [&](bool hit, int u, int j, int, int, int, double d0, double d1, double d2) {
                      if (!hit) return;
                      const double b0 = d0 * kAngToBohr, b1 = d1 * kAngToBohr, b2 = d2 * kAngToBohr;
                      const double r2 = b0 * b0 + b1 * b1 + b2 * b2;
                      const GreenPair q = gp[Xi * S + (int)xs[u].w];
                      const double R02 = q.R * q.R, R06 = R02 * R02 * R02, R08 = R06 * R02;
                      const double r4 = r2 * r2, r6 = r4 * r2, r8 = r6 * r2;
                      const double den6 = r6 + R06, den8 = r8 + R08;
                      const double phi = s6 / den6 + 3.0 * s8 * q.qq / den8;
                      const double dphi_r = -6.0 * s6 * r4 / (den6 * den6) - 24.0 * s8 * q.qq * r6 / (den8 * den8);
                      double C6 = 0.0;
#pragma unroll
                      for (int r = 0; r < 8; ++r)
                        if (r < R) {
                          const double cj = c6[(size_t)j * R + r];
                          C6 += ci[r] * cj;
                          gc[r] += cj * phi;
                        }
                      e += C6 * phi;
                      const double w = C6 * dphi_r;
                      g0 += w * b0;
                      g1 += w * b1;
                      g2 += w * b2;
                      v[0] += w * b0 * b0;
                      v[1] += w * b0 * b1;
                      v[2] += w * b0 * b2;
                      v[3] += w * b1 * b1;
                      v[4] += w * b1 * b2;
                      v[5] += w * b2 * b2;
                    });
    e = warp_sum(e);
    g0 = warp_sum(g0);
    g1 = warp_sum(g1);
    g2 = warp_sum(g2);
#pragma unroll
    for (int r = 0; r < 8; ++r) gc[r] = warp_sum(gc[r]);
#pragma unroll
    for (int c = 0; c < 6; ++c) v[c] = warp_sum(v[c]);
    if (lane == 0) {
      for (int r = 0; r < R; ++r) dEdc[(size_t)i * R + r] = -tab->eigs[r] * gc[r];
      grad[3 * (size_t)i] = g0;
      grad[3 * (size_t)i + 1] = g1;
      grad[3 * (size_t)i + 2] = g2;
      acc[0] = e;
#pragma unroll
      for (int c = 0; c < 6; ++c) acc[1 + c] = -0.5 * v[c];
    }
  }
  block_sum_store<7>(acc, part + 7 * blockIdx.x);
}

int launch_direct_pairs(const CellGrid& g, int n, const CellList& cl, const double* c6, const Tables* tab, int R,
                        int S, const GreenPair* gp, double* dEdc, double* grad, double* part, int* n_blocks,
                        cudaStream_t s) {
  if (R < 1 || R > 8) {
    set_error("direct sum", "the direct pair sum takes at most 8 ranks");
    return FD3_EINVAL;
  }
  const int blocks = (n + kWarpsPerBlock - 1) / kWarpsPerBlock;
  *n_blocks = blocks;
  if (blocks == 0) return FD3_OK;
  k_direct_pairs<<<blocks, 32 * kWarpsPerBlock, 0, s>>>(to_dev(g), n, cl.bin_start, cl.xs, cl.meta, cl.off, c6, tab,
                                                        R, S, gp, dEdc, grad, part);
  FD3_LAUNCHED();
  return FD3_OK;
}

int launch_nbr_count(const CellGrid& g, int n, const CellList& cl, int* counts, cudaStream_t s) {
  const int blocks = (n + kWarpsPerBlock - 1) / kWarpsPerBlock;
  if (blocks == 0) return FD3_OK;
  k_nbr<false><<<blocks, 32 * kWarpsPerBlock, 0, s>>>(to_dev(g), n, cl.bin_start, cl.xs, cl.meta, cl.off, counts,
                                                      nullptr, nullptr, nullptr, nullptr, 0);
  FD3_LAUNCHED();
  return FD3_OK;
}

// Block 0: row starts; block 1: the total in 64 bits (the row starts hold up to 2^31 - 1 pairs).
__global__ void __launch_bounds__(kScanThreads) k_nbr_rows(const int* __restrict__ counts, int n,
                                                          int* __restrict__ row_start, int64_t* __restrict__ total) {
  if (blockIdx.x == 0) {
    scan_exclusive_block(counts, n, row_start);
    return;
  }
  __shared__ long long part[32];
  long long v = 0;
  for (int i = threadIdx.x; i < n; i += kScanThreads) v += counts[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 32; ++w) v += part[w];
    *total = v;
  }
}

int launch_nbr_rows(const int* counts, int n, int* row_start, int64_t* total, cudaStream_t s) {
  k_nbr_rows<<<2, kScanThreads, 0, s>>>(counts, n, row_start, total);
  FD3_LAUNCHED();
  return FD3_OK;
}

int launch_nbr_fill(const CellGrid& g, int n, const CellList& cl, const int* row_start, int64_t* src, int64_t* dst,
                    int32_t* shift, int64_t room, cudaStream_t s) {
  const int blocks = (n + kWarpsPerBlock - 1) / kWarpsPerBlock;
  if (blocks == 0) return FD3_OK;
  k_nbr<true><<<blocks, 32 * kWarpsPerBlock, 0, s>>>(to_dev(g), n, cl.bin_start, cl.xs, cl.meta, cl.off, nullptr,
                                                     row_start, src, dst, shift, (unsigned)room);
  FD3_LAUNCHED();
  return FD3_OK;
}

}  // namespace fd3
