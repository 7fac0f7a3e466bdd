// SPME / PME spread and gather kernel templates (reference: src/fourierd3/mesh_interpolator_d3.py:74-189,
// src/fourierd3/kspace_filter_d3.py:29-98, src/fourierd3/pair_pot.py:113-228, core.py:553-581).
//
// spread  : one CTA owns one mesh tile (8x8x8 points) and one species; it pulls the atoms whose
//           stencil can reach the tile from the counting-sorted (tile, species) segments, and every
//           thread sums the contributions for its own points. Each mesh value is written exactly
//           once, in a fixed summation order: no global atomics, no zero-fill pass, deterministic.
// filter  : one thread per rfft k-point; evaluates G_XY(|k|) and dG/d|k| in registers, applies the
//           deconvolution window and the Hermitian weight, accumulates the energy and the virial
//           (float64), and overwrites the spectrum with H_X = sum_Y G_XY S_Y for the inverse FFT.
// gather  : one warp per atom (tile-sorted order); sums phi over the p^3 stencil for the C6-factor
//           adjoint and the spline-gradient force.
#include <math.h>

#include <type_traits>

#pragma once
#include "fd3_internal.h"

namespace fd3 {

struct MeshDev {
  int n[3], nzh, t[3], nt[3], ns[3], S, R;
  int qpitch;   // complex values per ky row of the half spectrum (nzh or nzh + 1)
  FastDiv div_nzh, div_ny, div_qpitch;
  const float* win_axes;
};
static inline MeshDev to_dev(const MeshGeom& g) {
  MeshDev d;
  for (int a = 0; a < 3; ++a) {
    d.n[a] = g.n[a];
    d.t[a] = g.t[a];
    d.nt[a] = g.nt[a];
    d.ns[a] = g.ns[a];
  }
  d.nzh = g.nzh;
  d.S = g.S;
  d.R = g.R;
  d.div_nzh = make_fastdiv((uint32_t)g.nzh);
  d.qpitch = g.qpitch > 0 ? g.qpitch : g.nzh;
  d.div_qpitch = make_fastdiv((uint32_t)d.qpitch);
  d.div_ny = make_fastdiv((uint32_t)g.n[1]);
  d.win_axes = g.win_axes;
  return d;
}

// Fractional mesh coordinate of one atom along all axes and its first stencil node.
// MeshInterpolator.compute_weights (core.py:555): u = n * (x @ inv); reference node round(u)
// (odd p) or floor(u) (even p); local x = u - ref (odd) or u - ref - 1/2 (even).
template <typename T>
__device__ __forceinline__ void mesh_locate(const double* __restrict__ pos, int i, double ps, const CellInfo* ci,
                                            int n0, int n1, int n2, int P, int* base, T* xl) {
  const double x0 = pos[3 * i] * ps, x1 = pos[3 * i + 1] * ps, x2 = pos[3 * i + 2] * ps;
  const int n[3] = {n0, n1, n2};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double u = n[a] * (x0 * ci->inv[a] + x1 * ci->inv[3 + a] + x2 * ci->inv[6 + a]);
    double ref, x;
    if (P % 2 == 0) {
      ref = floor(u);
      x = u - (ref + 0.5);
    } else {
      ref = rint(u);
      x = u - ref;
    }
    const long long b = (long long)ref + (1 - (P + 1) / 2);
    long long bm = b % n[a];
    if (bm < 0) bm += n[a];
    base[a] = (int)bm;
    xl[a] = (T)x;
  }
}

template <int P, bool LAG, typename T>
__device__ __forceinline__ void stencil_weights(T x, T* w, T* dw) {
  if (LAG)
    lagrange<P, T>(x, w, dw);
  else
    bspline<P, T>(x, w, dw);
}

// ------------------------------------------------------------------ Green table (mixed form)
// Entry e of the table: pair e / (kGreenKnots + 1) (X <= Y, index X S - X (X - 1) / 2 + (Y - X)) at
// knot e mod (kGreenKnots + 1).
__device__ inline float4 green_table_entry(const MeshDev& g, const double (&rec)[9],
                                           const GreenPair* __restrict__ gp, const Tables* __restrict__ tab, int e) {
  const int S = g.S;
  const int pi = e / (kGreenKnots + 1), j = e - pi * (kGreenKnots + 1);
  int X = 0;
  while ((X + 1) * S - (X + 1) * X / 2 <= pi) ++X;
  const int Y = X + (pi - (X * S - X * (X - 1) / 2));
  const GreenPair& q = gp[X * S + Y];
  const int n[3] = {g.n[0], g.n[1], g.n[2]};
  const double h = green_kmax(rec, n) / kGreenKnots;
  const double k = j * h;
  const double s6 = tab->s6, s8 = tab->s8;
  const double A6 = s6 * q.c6pre, A8 = 3.0 * s8 * q.qq * q.c8pre;
  double G, G1, G2, G3;
  if (k * q.R < 1e-15) {
    // k = 0: the value of the reference's Taylor branch (pair_pot.py:146, G = a), and the
    // derivatives of the closed form G = F(kR) / k there, G^(m)(0) = F^(m+1)(0) R^(m+1) / (m+1)
    // with F'(0) = A6 - sqrt2 sin(pi/8) A8, F''(0) = 0, F'''(0) = -2 A6 + sqrt2 sin(pi/8) A8,
    // F''''(0) = 3 A6. (The reference's k^2 coefficient of the C6 term, pair_pot.py:96, scales as
    // R where the expansion of the closed form gives 2 pi^2 / (9 R); it multiplies k^2 = 0 there,
    // so it never enters its results, but the interpolation between knots needs the true G''.)
    const double a = s6 * q.c6s1 + 3.0 * s8 * q.qq * q.c8s1;
    const double r2s8 = 0.54119610014619698440;   // sqrt(2) sin(pi/8)
    const double R3 = q.R * q.R * q.R;
    G = a;
    G1 = 0.0;
    G2 = (-2.0 * A6 + r2s8 * A8) * R3 / 3.0;
    G3 = 3.0 * A6 * R3 * q.R / 4.0;
  } else {
    double n6[4], n8[4];
    green_n(k * q.R, n6, n8);
    double F[4];
    for (int m = 0; m < 4; ++m) F[m] = A6 * n6[m] + A8 * n8[m];
    G = F[0] / k;
    G1 = (q.R * F[1] - G) / k;
    G2 = (q.R * q.R * F[2] - 2.0 * G1) / k;
    G3 = (q.R * q.R * q.R * F[3] - 3.0 * G2) / k;
  }
  return make_float4((float)G, (float)(h * G1), (float)(h * h * G2), (float)(h * h * h * G3));
}

// The records' rank factors (sorted order) from values per atom.
template <typename T>
__global__ void __launch_bounds__(256) k_rank_factors(int n, int R, const double* __restrict__ c6,
                                                      const int* __restrict__ order, T* __restrict__ rc) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int atom = order[t];
  for (int r = 0; r < R; ++r) rc[(size_t)t * R + r] = (T)c6[(size_t)atom * R + r];
}

// ------------------------------------------------------------------ spread
// Tile-owned spread. A CTA owns one (16 x 16 x 8)-point tile of one species; thread (lx, ly)
// owns the z-row of 8 points at (lx, ly). The atoms whose stencil can reach the tile come from
// the counting-sorted (tile, species) segments of the source tiles; they are examined 256 at a
// time, the overlapping ones are compacted (warp ballots, sorted order kept) into shared memory
// as three tile-local 1D weight rows (zero outside the stencil; stencil nodes that wrap onto
// the same point are summed), and every thread accumulates w_x(lx) w_y(ly) w_z(z) c_r for its
// row. Each mesh value is written exactly once: no atomics, no zero fill, fixed summation order.
constexpr int kSpTX = 16, kSpTY = 16, kSpTZ = 8;
constexpr int kSpThreads = kSpTX * kSpTY;
constexpr int kSpRC = 4;                 // ranks accumulated per pass

template <typename T>
struct SpChunk {
  static constexpr int value = sizeof(T) == 8 ? 64 : 128;
};

template <typename T, int P>
__global__ void __launch_bounds__(kSpThreads, sizeof(T) == 8 ? 2 : 4) k_spread(MeshDev g, const int4* __restrict__ rb,
                                                       const T* __restrict__ rw, const T* __restrict__ rc,
                                                       const int* __restrict__ key_start, T* __restrict__ rho) {
  constexpr int CH = SpChunk<T>::value;
  __shared__ T s_wx[CH][kSpTX];
  __shared__ T s_wy[CH][kSpTY];
  __shared__ T s_wz[CH][kSpTZ];
  __shared__ T s_c[CH][kSpRC];
  __shared__ int s_a0[125], s_pref[126];
  __shared__ int s_wcnt[kSpThreads / 32];

  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int X = blockIdx.y;
  const int tile = blockIdx.x;
  const int tz = tile % g.nt[2];
  const int ty = (tile / g.nt[2]) % g.nt[1];
  const int tx = tile / (g.nt[2] * g.nt[1]);
  const int t0[3] = {tx * g.t[0], ty * g.t[1], tz * g.t[2]};
  const int lx = tid / kSpTY, ly = tid % kSpTY;
  const bool row_ok = lx < g.t[0] && ly < g.t[1];
  const int R = g.R;
  const int nsrc = g.ns[0] * g.ns[1] * g.ns[2];

  if (tid < nsrc) {
    const int sxo = tid / (g.ns[1] * g.ns[2]), syo = (tid / g.ns[2]) % g.ns[1], szo = tid % g.ns[2];
    const int sx = posmod(tx - sxo, g.nt[0]), sy = posmod(ty - syo, g.nt[1]), sz = posmod(tz - szo, g.nt[2]);
    const int key = ((sx * g.nt[1] + sy) * g.nt[2] + sz) * g.S + X;
    const int a0 = key_start[key];
    s_a0[tid] = a0;
    s_pref[tid + 1] = key_start[key + 1] - a0;
  }
  __syncthreads();
  if (tid == 0) {
    s_pref[0] = 0;
    for (int k = 0; k < nsrc; ++k) s_pref[k + 1] += s_pref[k];
  }
  __syncthreads();
  const int total = s_pref[nsrc];
  const size_t M = (size_t)g.n[0] * g.n[1] * g.n[2];

  for (int r0 = 0; r0 < R; r0 += kSpRC) {
    T acc[kSpTZ][kSpRC];
#pragma unroll
    for (int z = 0; z < kSpTZ; ++z)
#pragma unroll
      for (int r = 0; r < kSpRC; ++r) acc[z][r] = T(0);

    for (int c0 = 0; c0 < total; c0 += kSpThreads) {
      // examine one candidate per thread
      const int ca = c0 + tid;
      bool keep = false;
      int u = 0, base[3] = {0, 0, 0};
      if (ca < total) {
        int seg = 0;
        while (s_pref[seg + 1] <= ca) ++seg;
        u = s_a0[seg] + (ca - s_pref[seg]);      // record slot (sorted order)
        const int4 b4 = rb[u];
        base[0] = b4.x;
        base[1] = b4.y;
        base[2] = b4.z;
        keep = true;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          int d = t0[a] - base[a];
          if (d < 0) d += g.n[a];
          // stencil offsets [0, min(P, n)) from base; the tile covers offsets [d, d + t)
          const int pf = P < g.n[a] ? P : g.n[a];
          if (!(d < pf || d + g.t[a] > g.n[a])) keep = false;
        }
      }
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      if (lane == 0) s_wcnt[wid] = __popc(bal);
      __syncthreads();
      int off = 0, tot = 0;
#pragma unroll
      for (int w = 0; w < kSpThreads / 32; ++w) {
        off += w < wid ? s_wcnt[w] : 0;
        tot += s_wcnt[w];
      }
      __syncthreads();   // s_wcnt is rewritten by the next examination pass
      for (int h0 = 0; h0 < tot; h0 += CH) {
        const int slot = off + __popc(bal & ((1u << lane) - 1u)) - h0;
        if (keep && slot >= 0 && slot < CH) {
          T w[3][P];
#pragma unroll
          for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int k = 0; k < P; ++k) w[a][k] = rw[((size_t)u * 3 + a) * P + k];
#pragma unroll
          for (int z = 0; z < kSpTX; ++z) s_wx[slot][z] = T(0);
#pragma unroll
          for (int z = 0; z < kSpTY; ++z) s_wy[slot][z] = T(0);
#pragma unroll
          for (int z = 0; z < kSpTZ; ++z) s_wz[slot][z] = T(0);
#pragma unroll
          for (int k = 0; k < P; ++k) {
            int ix = (base[0] + k - t0[0]) % g.n[0]; if (ix < 0) ix += g.n[0];
            int iy = (base[1] + k - t0[1]) % g.n[1]; if (iy < 0) iy += g.n[1];
            int iz = (base[2] + k - t0[2]) % g.n[2]; if (iz < 0) iz += g.n[2];
            if (ix < g.t[0]) s_wx[slot][ix] += w[0][k];
            if (iy < g.t[1]) s_wy[slot][iy] += w[1][k];
            if (iz < g.t[2]) s_wz[slot][iz] += w[2][k];
          }
#pragma unroll
          for (int r = 0; r < kSpRC; ++r) s_c[slot][r] = r0 + r < R ? rc[(size_t)u * R + r0 + r] : T(0);
        }
        __syncthreads();
        const int nc = min(CH, tot - h0);
        if (row_ok) {
          for (int c = 0; c < nc; ++c) {
            const T wxy = s_wx[c][lx] * s_wy[c][ly];
            if (wxy != T(0)) {
              T cr[kSpRC];
#pragma unroll
              for (int r = 0; r < kSpRC; ++r) cr[r] = wxy * s_c[c][r];
#pragma unroll
              for (int z = 0; z < kSpTZ; ++z) {
                const T wz = s_wz[c][z];
#pragma unroll
                for (int r = 0; r < kSpRC; ++r) acc[z][r] += wz * cr[r];
              }
            }
          }
        }
        __syncthreads();
      }
    }
    if (row_ok) {
      const size_t m0 = ((size_t)(t0[0] + lx) * g.n[1] + (t0[1] + ly)) * g.n[2] + t0[2];
#pragma unroll
      for (int r = 0; r < kSpRC; ++r) {
        if (r0 + r >= R) break;
        T* dst = rho + ((size_t)X * R + r0 + r) * M + m0;
        if (g.t[2] == kSpTZ) {
          // the row starts on an 8-element boundary: two 16-byte stores (float) or four (double)
          if (sizeof(T) == 4) {
            float4* v = reinterpret_cast<float4*>(dst);
            v[0] = make_float4((float)acc[0][r], (float)acc[1][r], (float)acc[2][r], (float)acc[3][r]);
            v[1] = make_float4((float)acc[4][r], (float)acc[5][r], (float)acc[6][r], (float)acc[7][r]);
          } else {
            double2* v = reinterpret_cast<double2*>(dst);
#pragma unroll
            for (int z = 0; z < kSpTZ; z += 2) v[z / 2] = make_double2((double)acc[z][r], (double)acc[z + 1][r]);
          }
        } else {
#pragma unroll
          for (int z = 0; z < kSpTZ; ++z)
            if (z < g.t[2]) dst[z] = acc[z][r];
        }
      }
    }
  }
}

// Column spread. A CTA owns a column of 16 x 16 points in (x, y) and a chunk of ZC z-tiles of one
// species; a thread owns 16 bytes of z of the current z-tile in 2 (float) or 4 (double) rows adjacent in
// y, so that neighbouring lanes store one row's 32 or 64 bytes together. The atoms whose x and
// y stencils reach the column are staged ONCE per chunk, in counting-sorted segment order with the
// source z-tile outermost, as tile-local x and y weight rows, rank factors, and two z rows: the
// part of the z stencil inside the atom's own z-tile and the part spilling into the next one
// (a stencil of P <= t_z + 1 nodes spans at most two tiles). The atoms reaching z-tile T are then
// two contiguous ranges of the staged list, those of source tile T (own rows) and of T - 1 (spill
// rows), so the CTA sweeps its z-tiles from shared memory with no selection and no barrier.
// Global loads and the candidate search happen once per ZC tiles. A chunk whose staged set
// exceeds `cap` falls back, inside the same CTA, to staging per tile in pieces of `cap`. Each
// mesh value is written exactly once in a fixed summation order (no atomics); results are
// independent of ZC up to the summation order.
//
// The load/store pipe bounds it (256^3, 8 channels, float64: its wavefronts at 75 % of their peak, DRAM at 26 %),
// so the layouts are chosen for few wavefronts: the stores above (a thread with a whole row stores 16
// bytes per line), staged rows of 17 or 18 values (a thread stages an atom; rows of 16 put all lanes on
// the same banks), and per atom one z, one or two y and the rank loads for 32 multiply-adds. 139,968 atoms on
// 256^3, 2 x 4 channels: float64 497 -> 348 us, float 283 -> 217 (before: a whole row of 8 per thread); with the
// ranks in the rows' padding (kColPadRanks) 320 and 200.
constexpr int kColMaxSeg = 64;

// what a thread owns of a z-tile: kZL values in each of kRows rows
template <typename T>
struct ColOwn {
  static constexpr int kZL = 16 / sizeof(T);
  static constexpr int kRows = kSpTZ / kZL;
  static constexpr int kWx = 17, kWy = 18;            // staged row lengths
  static constexpr int kWz = sizeof(T) == 4 ? 20 : 18;
};

// The words that pad a row off the bank period hold the atom's first four ranks (float: after wz; double: two after
// wz, two after wy) and its source z-tile (after wx), so that padded rows hold as many atoms as rows of 16 did: 256
// float or 270 double with 4 ranks. (226 and 238 with the ranks in rows of their own: chunks of 8 tiles of 128^3 with
// 30,840 atoms, 2 species, float, took 121 us, 70 with rows of 16 and now 52; all sizes gain by the shared address.)
constexpr int kColPadRanks = 4;

template <typename T>
struct ColSmem {
  T* wz;      // [cap][kWz] z row inside the atom's own z-tile (8), then the part spilling into the next (8)
  T* wy;      // [cap][kWy]
  T* wx;      // [cap][kWx]
  T* cc;      // [cap][max(R - kColPadRanks, 0)] the other ranks
  int* zst;   // [kColMaxSeg + 1] first staged slot of each source z-tile
  // source z-tile (index into the chunk's source range) of a slot; bit 30: spills
  __device__ __forceinline__ int& zi(int a) const {
    return *reinterpret_cast<int*>(wx + a * ColOwn<T>::kWx + 16);
  }
};

__host__ __device__ inline size_t col_round16(size_t b) { return (b + 15) & ~(size_t)15; }
__host__ __device__ inline int col_more_ranks(int R) { return R > kColPadRanks ? R - kColPadRanks : 0; }

template <typename T>
__host__ __device__ inline size_t col_smem_bytes(int cap, int R) {
  using O = ColOwn<T>;
  return col_round16((size_t)cap * O::kWz * sizeof(T)) + col_round16((size_t)cap * O::kWy * sizeof(T)) +
         col_round16((size_t)cap * O::kWx * sizeof(T)) + col_round16((size_t)cap * col_more_ranks(R) * sizeof(T)) +
         col_round16((size_t)(kColMaxSeg + 1) * sizeof(int));
}

template <typename T>
__device__ __forceinline__ ColSmem<T> col_carve(unsigned char* base, int cap, int R) {
  using O = ColOwn<T>;
  ColSmem<T> m;
  m.wz = reinterpret_cast<T*>(base);
  base += col_round16((size_t)cap * O::kWz * sizeof(T));
  m.wy = reinterpret_cast<T*>(base);
  base += col_round16((size_t)cap * O::kWy * sizeof(T));
  m.wx = reinterpret_cast<T*>(base);
  base += col_round16((size_t)cap * O::kWx * sizeof(T));
  m.cc = reinterpret_cast<T*>(base);
  base += col_round16((size_t)cap * col_more_ranks(R) * sizeof(T));
  m.zst = reinterpret_cast<int*>(base);
  return m;
}

// The first four ranks of slot a (FIRST), or ranks r0 .. r0 + 3 of a later group: two at lo(a), two at hi(a).
template <typename T, bool FIRST>
struct ColRanks {
  const ColSmem<T>& m;
  int R, r0;
  __device__ __forceinline__ T* lo(int a) const {
    using O = ColOwn<T>;
    static_assert(O::kWz >= 16 + (sizeof(T) == 4 ? 4 : 2) && O::kWy >= 18);
    return FIRST ? m.wz + a * O::kWz + 16 : m.cc + a * (R - kColPadRanks) + (r0 - kColPadRanks);
  }
  __device__ __forceinline__ T* hi(int a) const {
    return FIRST && sizeof(T) == 8 ? m.wy + a * ColOwn<T>::kWy + 16 : lo(a) + 2;
  }
};

constexpr int kZiSpill = 1 << 30;

// Block-wide ordered compaction of one flag per thread: returns this thread's slot (among the
// set flags, in thread order) and writes the block total to *tot. Two barriers.
__device__ __forceinline__ int block_compact(bool keep, int* s_wcnt, int* tot) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned bal = __ballot_sync(0xffffffffu, keep);
  if (lane == 0) s_wcnt[wid] = __popc(bal);
  __syncthreads();
  int off = 0, t = 0;
#pragma unroll
  for (int w = 0; w < kSpThreads / 32; ++w) {
    off += w < wid ? s_wcnt[w] : 0;
    t += s_wcnt[w];
  }
  __syncthreads();
  *tot = t;
  return off + __popc(bal & ((1u << lane) - 1u));
}

// Stage candidates [from, total) whose stencil reaches the column in x and y (and z-tile tzt when
// tzt >= 0) into slots [0, cap). Segment e covers source z-tile e / seg_per_z of the chunk.
// Returns the number staged; *next is the first candidate not yet examined or staged (== total
// when all were taken).
template <typename T, int P>
__device__ int col_stage(const MeshDev& g, const int* s_a0, const int* s_pref, int nseg, int seg_per_z, int total,
                         int from, const int (&t0)[3], int tzt, int cap, const int4* __restrict__ rb,
                         const T* __restrict__ rw, const T* __restrict__ rc, const ColSmem<T>& m, int* s_wcnt,
                         int* s_next, int* next) {
  const int R = g.R;
  int staged = 0;
  int c0 = from;
  bool full = false;
  if (threadIdx.x == 0) *s_next = total;
  for (; c0 < total; c0 += kSpThreads) {
    const int ca = c0 + threadIdx.x;
    bool keep = false;
    int u = 0, seg = 0;
    int4 b4 = make_int4(0, 0, 0, 0);
    if (ca < total) {
      int lo = 0, hi = nseg - 1;   // last segment with pref <= ca
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_pref[mid] <= ca) lo = mid; else hi = mid - 1;
      }
      seg = lo;
      u = s_a0[lo] + (ca - s_pref[lo]);
      b4 = rb[u];
      keep = true;
      const int base[3] = {b4.x, b4.y, b4.z};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (a == 2 && tzt < 0) break;
        const int ta = a == 2 ? tzt * g.t[2] : t0[a];
        int d = ta - base[a];
        if (d < 0) d += g.n[a];
        const int pf = P < g.n[a] ? P : g.n[a];
        if (!(d < pf || d + g.t[a] > g.n[a])) keep = false;
      }
    }
    int tot;
    const int slot = staged + block_compact(keep, s_wcnt, &tot);
    if (keep && slot < cap) {
      // tile-local x and y rows (stencil nodes that wrap onto the same point are summed)
      T* wxr = m.wx + slot * ColOwn<T>::kWx;
      T* wyr = m.wy + slot * ColOwn<T>::kWy;
      T* zo = m.wz + slot * ColOwn<T>::kWz;
      T* zn = zo + kSpTZ;
#pragma unroll
      for (int z = 0; z < 16; ++z) {
        wxr[z] = T(0);
        wyr[z] = T(0);
      }
#pragma unroll
      for (int z = 0; z < kSpTZ; ++z) {
        zo[z] = T(0);
        zn[z] = T(0);
      }
      const T* w = rw + (size_t)u * 3 * P;
      const int oz = b4.z % g.t[2];   // offset of the base inside its own z-tile
      bool spill = false;
#pragma unroll
      for (int k = 0; k < P; ++k) {
        int ix = b4.x + k - t0[0];
        while (ix < 0) ix += g.n[0];
        while (ix >= g.n[0]) ix -= g.n[0];
        int iy = b4.y + k - t0[1];
        while (iy < 0) iy += g.n[1];
        while (iy >= g.n[1]) iy -= g.n[1];
        if (ix < g.t[0]) wxr[ix] += w[k];
        if (iy < g.t[1]) wyr[iy] += w[P + k];
        const int z = oz + k;
        if (z < g.t[2]) {
          zo[z] = w[2 * P + k];
        } else {
          zn[z - g.t[2]] = w[2 * P + k];
          spill = true;
        }
      }
      m.zi(slot) = seg / seg_per_z + (spill ? kZiSpill : 0);
      const ColRanks<T, true> first{m, R, 0};
#pragma unroll
      for (int r = 0; r < kColPadRanks; ++r)
        (r < 2 ? first.lo(slot) : first.hi(slot))[r & 1] = r < R ? rc[(size_t)u * R + r] : T(0);
      for (int r = kColPadRanks; r < R; ++r)
        m.cc[slot * (R - kColPadRanks) + r - kColPadRanks] = rc[(size_t)u * R + r];
    }
    if (keep && slot >= cap) atomicMin(s_next, ca);
    staged += tot;
    if (staged >= cap) {
      full = true;
      break;
    }
  }
  __syncthreads();
  int nx = *s_next;   // first kept candidate that found no slot, else total
  if (full && c0 + kSpThreads < nx) nx = c0 + kSpThreads;   // the pass filled cap exactly
  *next = nx;
  __syncthreads();
  return staged < cap ? staged : cap;
}

// acc[row][z][r] += w_x(lx) w_y(ly0 + row) w_z(z0 + z) c_{r0+r} over staged atoms [a0, a1), with their
// own-tile z rows (spill = false) or spill rows (spill = true). CHECK: the range may hold atoms of other
// source z-tiles (per-tile staging), skip those whose source tile is not zsrc. Atoms are taken
// four at a time so that their x weight loads are in flight together; an atom with no spill
// has an all-zero spill row and adds exact zeros.
template <typename T>
using ColAcc = T[ColOwn<T>::kRows][ColOwn<T>::kZL][kSpRC];

template <typename T, bool CHECK, bool FIRST>
__device__ __forceinline__ void col_atom(const ColSmem<T>& m, int a, int z0, T wx, int zsrc, int R, int r0, int ly0,
                                         ColAcc<T>& acc) {
  using O = ColOwn<T>;
  const ColRanks<T, FIRST> cr4{m, R, r0};
  if (CHECK && (m.zi(a) & ~kZiSpill) != zsrc) return;
  T c[kSpRC], zr[O::kZL], wxy[O::kRows];
  if (sizeof(T) == 4) {
    const float2 y = *reinterpret_cast<const float2*>(m.wy + a * O::kWy + ly0);
    const float4 z = *reinterpret_cast<const float4*>(m.wz + a * O::kWz + z0);
    const float zz[4] = {z.x, z.y, z.z, z.w};
    wxy[0] = wx * (T)y.x;
    wxy[1] = wx * (T)y.y;
#pragma unroll
    for (int k = 0; k < O::kZL; ++k) zr[k] = (T)zz[k];
  } else {
    const double2 ya = *reinterpret_cast<const double2*>(m.wy + a * O::kWy + ly0);
    const double2 yb = *reinterpret_cast<const double2*>(m.wy + a * O::kWy + ly0 + 2);
    const double2 z = *reinterpret_cast<const double2*>(m.wz + a * O::kWz + z0);
    const double yy[4] = {ya.x, ya.y, yb.x, yb.y};
#pragma unroll
    for (int k = 0; k < O::kRows; ++k) wxy[k] = wx * (T)yy[k];
    zr[0] = (T)z.x;
    zr[1] = (T)z.y;
  }
  static_assert(kSpRC == 4 && kColPadRanks == 4);
  if (FIRST || (R & 3) == 0) {
    // a whole 4-rank group in 16-byte loads (the first four, zero beyond R, and groups of rows of 4 n values)
    if (sizeof(T) == 4) {
      const float4 v = *reinterpret_cast<const float4*>(cr4.lo(a));
      c[0] = (T)v.x;
      c[1] = (T)v.y;
      c[2] = (T)v.z;
      c[3] = (T)v.w;
    } else {
      const double2 v0 = *reinterpret_cast<const double2*>(cr4.lo(a));
      const double2 v1 = *reinterpret_cast<const double2*>(cr4.hi(a));
      c[0] = (T)v0.x;
      c[1] = (T)v0.y;
      c[2] = (T)v1.x;
      c[3] = (T)v1.y;
    }
  } else {
#pragma unroll
    for (int r = 0; r < kSpRC; ++r) c[r] = r0 + r < R ? cr4.lo(a)[r] : T(0);
  }
  if constexpr (sizeof(T) == 4) {
    // two ranks per instruction, rounded as two multiply-adds are (instruction issue bounds the float form: 2.7
    // per cycle and SM, 236 us at the size above, without it)
#pragma unroll
    for (int k = 0; k < O::kRows; ++k) {
#pragma unroll
      for (int r = 0; r < kSpRC; r += 2) {
        const float2 cr = make_float2(wxy[k] * c[r], wxy[k] * c[r + 1]);
#pragma unroll
        for (int z = 0; z < O::kZL; ++z) {
          const float2 q = __ffma2_rn(make_float2(zr[z], zr[z]), cr, make_float2(acc[k][z][r], acc[k][z][r + 1]));
          acc[k][z][r] = q.x;
          acc[k][z][r + 1] = q.y;
        }
      }
    }
  } else {
#pragma unroll
  for (int k = 0; k < O::kRows; ++k) {
#pragma unroll
    for (int r = 0; r < kSpRC; ++r) {
      const T cr = wxy[k] * c[r];
#pragma unroll
      for (int z = 0; z < O::kZL; ++z) acc[k][z][r] += zr[z] * cr;
    }
  }
  }
}

template <typename T, bool CHECK, bool FIRST>
__device__ __forceinline__ void col_range(const ColSmem<T>& m, int a0, int a1, int zsrc, bool spill, int R, int r0,
                                          int lx, int ly0, int zl0, ColAcc<T>& acc) {
  using O = ColOwn<T>;
  const int z0 = zl0 + (spill ? kSpTZ : 0);
  int a = a0;
  for (; a + 4 <= a1; a += 4) {
    T wx[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) wx[u] = m.wx[(a + u) * O::kWx + lx];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (wx[u] != T(0)) col_atom<T, CHECK, FIRST>(m, a + u, z0, wx[u], zsrc, R, r0, ly0, acc);
  }
  for (; a < a1; ++a) {
    const T wx = m.wx[a * O::kWx + lx];
    if (wx != T(0)) col_atom<T, CHECK, FIRST>(m, a, z0, wx, zsrc, R, r0, ly0, acc);
  }
}

template <typename T, bool CHECK>
__device__ __forceinline__ void col_accumulate(const ColSmem<T>& m, int a0, int a1, int zsrc, bool spill, int R,
                                               int r0, int lx, int ly0, int zl0, ColAcc<T>& acc) {
  if (r0 == 0)
    col_range<T, CHECK, true>(m, a0, a1, zsrc, spill, R, r0, lx, ly0, zl0, acc);
  else
    col_range<T, CHECK, false>(m, a0, a1, zsrc, spill, R, r0, lx, ly0, zl0, acc);
}

template <typename T>
__device__ __forceinline__ void col_store(const MeshDev& g, int X, int r0, const int (&t0)[3], int tzt, int lx,
                                          int ly0, int zl0, const ColAcc<T>& acc, T* __restrict__ rho) {
  using O = ColOwn<T>;
  if (lx >= g.t[0]) return;
  const size_t M = (size_t)g.n[0] * g.n[1] * g.n[2];
  const size_t m0 =
      ((size_t)(t0[0] + lx) * g.n[1] + (t0[1] + ly0)) * g.n[2] + (size_t)tzt * g.t[2] + (size_t)zl0;
#pragma unroll
  for (int r = 0; r < kSpRC; ++r) {
    if (r0 + r >= g.R) break;
#pragma unroll
    for (int k = 0; k < O::kRows; ++k) {
      if (ly0 + k >= g.t[1]) break;
      T* dst = rho + ((size_t)X * g.R + r0 + r) * M + m0 + (size_t)k * g.n[2];
      if (g.t[2] == kSpTZ) {
        if (sizeof(T) == 4)
          *reinterpret_cast<float4*>(dst) = make_float4((float)acc[k][0][r], (float)acc[k][1 % O::kZL][r],
                                                        (float)acc[k][2 % O::kZL][r], (float)acc[k][3 % O::kZL][r]);
        else
          *reinterpret_cast<double2*>(dst) = make_double2((double)acc[k][0][r], (double)acc[k][1][r]);
      } else {
#pragma unroll
        for (int z = 0; z < O::kZL; ++z)
          if (zl0 + z < g.t[2]) dst[z] = acc[k][z][r];
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ void col_zero(ColAcc<T>& acc) {
#pragma unroll
  for (int k = 0; k < ColOwn<T>::kRows; ++k)
#pragma unroll
    for (int z = 0; z < ColOwn<T>::kZL; ++z)
#pragma unroll
      for (int r = 0; r < kSpRC; ++r) acc[k][z][r] = T(0);
}

template <typename T, int P>
__global__ void __launch_bounds__(kSpThreads, sizeof(T) == 8 ? 2 : 4) k_spread_col(
    MeshDev g, int zc, int cap, const int4* __restrict__ rb, const T* __restrict__ rw, const T* __restrict__ rc,
    const int* __restrict__ key_start, T* __restrict__ rho) {
  extern __shared__ __align__(16) unsigned char col_raw[];
  __shared__ int s_a0[kColMaxSeg], s_pref[kColMaxSeg + 1];
  __shared__ int s_wcnt[kSpThreads / 32];
  __shared__ int s_next;
  const ColSmem<T> m = col_carve<T>(col_raw, cap, g.R);
  const int tid = threadIdx.x;
  const int X = blockIdx.y;
  const int nzc = (g.nt[2] + zc - 1) / zc;
  const int zch = blockIdx.x % nzc;
  const int cxy = blockIdx.x / nzc;
  const int ty = cxy % g.nt[1], tx = cxy / g.nt[1];
  const int tz0 = zch * zc;
  const int tz1 = tz0 + zc < g.nt[2] ? tz0 + zc : g.nt[2];
  const int t0[3] = {tx * g.t[0], ty * g.t[1], 0};
  // a group of kRows lanes owns kRows rows of its warp's 2 x 16 (x, y) rows; the lane picks the z part
  using O = ColOwn<T>;
  const int row0 = (tid >> 5) * 32 + ((tid & 31) / O::kRows) * O::kRows;
  const int lx = row0 / kSpTY, ly0 = row0 % kSpTY, zl0 = (tid % O::kRows) * O::kZL;
  // source z-tiles of the chunk: tz - 1 and tz for tz in [tz0, tz1), each once
  int nzs = (tz1 - tz0) + 1;
  int zs0 = tz0 - 1;
  if (nzs >= g.nt[2]) {
    nzs = g.nt[2];
    zs0 = 0;
  }
  const int spz = g.ns[0] * g.ns[1];   // segments per source z-tile
  const int nseg = spz * nzs;
  for (int e = tid; e < nseg; e += kSpThreads) {
    const int zi = e / spz, xo = (e % spz) / g.ns[1], yo = e % g.ns[1];
    const int sx = posmod(tx - xo, g.nt[0]), sy = posmod(ty - yo, g.nt[1]), sz = posmod(zs0 + zi, g.nt[2]);
    const int key = ((sx * g.nt[1] + sy) * g.nt[2] + sz) * g.S + X;
    const int a0 = key_start[key];
    s_a0[e] = a0;
    s_pref[e + 1] = key_start[key + 1] - a0;
  }
  __syncthreads();
  if (tid < 32) {   // inclusive warp scan of the segment sizes (nseg <= 64)
    int v0 = tid + 1 <= nseg ? s_pref[tid + 1] : 0;
    int v1 = tid + 33 <= nseg ? s_pref[tid + 33] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, v0, o);
      const int b = __shfl_up_sync(0xffffffffu, v1, o);
      if (tid >= o) {
        v0 += a;
        v1 += b;
      }
    }
    const int carry = __shfl_sync(0xffffffffu, v0, 31);
    if (tid + 1 <= nseg) s_pref[tid + 1] = v0;
    if (tid + 33 <= nseg) s_pref[tid + 33] = v1 + carry;
    if (tid == 0) s_pref[0] = 0;
  }
  __syncthreads();
  const int total = s_pref[nseg];
  int next = 0;
  const int staged = col_stage<T, P>(g, s_a0, s_pref, nseg, spz, total, 0, t0, -1, cap, rb, rw, rc, m, s_wcnt,
                                     &s_next, &next);
  if (next >= total) {
    // first staged slot of each source z-tile (the staged list is ordered by source z-tile)
    for (int zi = tid; zi <= nzs; zi += kSpThreads) {
      int lo = 0, hi = staged;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((m.zi(mid) & ~kZiSpill) < zi) lo = mid + 1; else hi = mid;
      }
      m.zst[zi] = lo;
    }
    __syncthreads();
    for (int tzt = tz0; tzt < tz1; ++tzt) {
      const int zown = nzs == g.nt[2] ? tzt : tzt - zs0;
      const int zprev = nzs == g.nt[2] ? (tzt + g.nt[2] - 1) % g.nt[2] : zown - 1;
      for (int r0 = 0; r0 < g.R; r0 += kSpRC) {
        ColAcc<T> acc;
        col_zero<T>(acc);
        col_accumulate<T, false>(m, m.zst[zprev], m.zst[zprev + 1], zprev, true, g.R, r0, lx, ly0, zl0, acc);
        col_accumulate<T, false>(m, m.zst[zown], m.zst[zown + 1], zown, false, g.R, r0, lx, ly0, zl0, acc);
        col_store<T>(g, X, r0, t0, tzt, lx, ly0, zl0, acc, rho);
      }
    }
    return;
  }
  // dense column: per z-tile, stage the atoms reaching that tile in pieces of `cap`
  for (int tzt = tz0; tzt < tz1; ++tzt) {
    const int zown = nzs == g.nt[2] ? tzt : tzt - zs0;
    const int zprev = nzs == g.nt[2] ? (tzt + g.nt[2] - 1) % g.nt[2] : zown - 1;
    for (int r0 = 0; r0 < g.R; r0 += kSpRC) {
      ColAcc<T> acc;
      col_zero<T>(acc);
      int from = 0;
      while (from < total) {
        const int st = col_stage<T, P>(g, s_a0, s_pref, nseg, spz, total, from, t0, tzt, cap, rb, rw, rc, m,
                                       s_wcnt, &s_next, &from);
        col_accumulate<T, true>(m, 0, st, zprev, true, g.R, r0, lx, ly0, zl0, acc);
        col_accumulate<T, true>(m, 0, st, zown, false, g.R, r0, lx, ly0, zl0, acc);
        __syncthreads();
      }
      col_store<T>(g, X, r0, t0, tzt, lx, ly0, zl0, acc, rho);
    }
  }
}

// Staged atoms per column chunk: as many as let 4 (float) or 2 (double) CTAs share an SM's 228 KB, of which each
// has 1 KB reserved and 560 bytes static.
template <typename T>
inline int spread_col_cap(const MeshGeom& mg) {
  constexpr int per_sm = sizeof(T) == 8 ? 2 : 4;
  const size_t fixed = col_smem_bytes<T>(0, mg.R);
  const size_t per_atom = (col_smem_bytes<T>(64, mg.R) - fixed) / 64;
  int cap = (int)((size_t)(228 * 1024 / per_sm - 1024 - 704 - fixed) / per_atom);
  if (cap > 1024) cap = 1024;
  if (mg.spread_cap > 0 && mg.spread_cap < cap) cap = mg.spread_cap;
  return cap;
}
constexpr int kColMinCap = 128;

// z-tiles per column chunk in effect for this mesh (0: per-tile kernel).
inline int spread_zc(const MeshGeom& mg) {
  // the column form needs stencils that span at most two z-tiles of a mesh with >= 2 z-tiles
  if (mg.spread_zc == 0 || mg.ns[0] > 2 || mg.ns[1] > 2 || mg.nt[2] < 2 || mg.order > mg.t[2] + 1 ||
      mg.t[2] > kSpTZ)
    return 0;
  // By default four z-tiles per CTA, fewer while that leaves the chip short of CTAs: staging the
  // atoms once for longer chunks saves less than an idle SM costs. (With rows of 8 points per thread: 648
  // atoms, 64^3, float64: 8 tiles 37 us, 1 tile 17; 1,500 HCNO atoms, 64^3, float: 47 -> 21; 12,000,
  // 128^3: 117 -> 99; 139,968, 256^3: 309 -> 283 with 4, 358 with 1.)
  int zc = mg.spread_zc;
  if (zc < 0)
    for (zc = 4; zc > 1 && mg.nt[0] * mg.nt[1] * ((mg.nt[2] + zc - 1) / zc) * mg.S < 400;) zc >>= 1;
  const int lim = kColMaxSeg / (mg.ns[0] * mg.ns[1]) - 1;
  if (zc > lim) zc = lim;
  if (zc > mg.nt[2]) zc = mg.nt[2];
  return zc < 1 ? 0 : zc;
}

template <typename T, int P>
static int spread_r(const MeshGeom& mg, dim3 grid, int n, const double* factors, const int* ks, const int* order,
                    const MeshRecords& rec, T* rho, cudaStream_t s) {
  const MeshDev g = to_dev(mg);
  if (n > 0 && factors) {
    k_rank_factors<T><<<(n + 255) / 256, 256, 0, s>>>(n, mg.R, factors, order, (T*)rec.c);
    FD3_LAUNCHED();
  }
  const int zc = spread_zc(mg);
  if (zc > 0) {
    const int cap = spread_col_cap<T>(mg);
    if (cap >= kColMinCap) {
      const size_t smem = col_smem_bytes<T>(cap, mg.R);
      const int rc = allow_dynamic_smem(k_spread_col<T, P>, 200 * 1024);
      if (rc) return rc;
      const int nzc = (mg.nt[2] + zc - 1) / zc;
      const dim3 cgrid(mg.nt[0] * mg.nt[1] * nzc, mg.S);
      k_spread_col<T, P><<<cgrid, kSpThreads, smem, s>>>(g, zc, cap, rec.b, (const T*)rec.w, (const T*)rec.c, ks,
                                                        rho);
      FD3_LAUNCHED();
      return FD3_OK;
    }
  }
  k_spread<T, P><<<grid, kSpThreads, 0, s>>>(g, rec.b, (const T*)rec.w, (const T*)rec.c, ks, rho);
  FD3_LAUNCHED();
  return FD3_OK;
}

template <typename T>
int launch_spread(const MeshGeom& mg, int n, const double* factors, const int* key_start, const int* order,
                  const MeshRecords& rec, T* rho, cudaStream_t s) {
  if (mg.R > FD3_MAX_RANK || mg.order < 1 || mg.order > FD3_MAX_ORDER) return FD3_EINVAL;
  if (mg.t[0] > kSpTX || mg.t[1] > kSpTY || mg.t[2] > kSpTZ || mg.ns[0] * mg.ns[1] * mg.ns[2] > 125)
    return FD3_EINVAL;
  const dim3 grid(mg.nt[0] * mg.nt[1] * mg.nt[2], mg.S);
#define FD3_SPREAD_CASE(PP) \
  case PP:                  \
    return spread_r<T, PP>(mg, grid, n, factors, key_start, order, rec, rho, s);
  switch (mg.order) {
    FD3_SPREAD_CASE(1)
    FD3_SPREAD_CASE(2)
    FD3_SPREAD_CASE(3)
    FD3_SPREAD_CASE(4)
    FD3_SPREAD_CASE(5)
    FD3_SPREAD_CASE(6)
    FD3_SPREAD_CASE(7)
    FD3_SPREAD_CASE(8)
  }
#undef FD3_SPREAD_CASE
  return FD3_EINVAL;
}

// ------------------------------------------------------------------ gather
}  // namespace fd3
#include "fd3_gather_tile.cuh"   // the tile-staged (TMA) gather, on MeshDev / MeshRecords above
namespace fd3 {

constexpr int kGatherWarps = 8;

// Sums of four values over the warp, 12 shuffles (four butterflies take 40): lanes 8 k .. 8 k + 7 return the
// k-th sum.
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool hi = lane & 16;
  double u = hi ? c : a, v = hi ? d : b;
  u += __shfl_xor_sync(kAll, hi ? a : c, 16);
  v += __shfl_xor_sync(kAll, hi ? b : d, 16);
  const bool odd = lane & 8;
  double w = odd ? v : u;
  w += __shfl_xor_sync(kAll, odd ? u : v, 8);
  w += __shfl_xor_sync(kAll, w, 4);
  w += __shfl_xor_sync(kAll, w, 2);
  w += __shfl_xor_sync(kAll, w, 1);
  return w;
}

// Gather, one warp per atom. The P z-values of a stencil column lie in NV aligned 16-byte vectors; a lane
// takes one vector of one column (neighbouring lanes the vectors of one column, so that a load of the warp
// touches 32 / NV lines) for RC rank channels at a time, with the z weights shifted to the vector (zero
// outside the stencil), and forms
//   zr_r = sum_z w_z phi_r,  cp_z = sum_r lambda_r c_r phi_r,  s0 = sum_z w_z cp_z,  s2 = sum_z w'_z cp_z
// in TA, then accumulates P_r = sum W phi_r and the three spline-gradient sums in float64.
// A column that wraps the periodic z edge (or a mesh whose nz is not a multiple of the vector
// width) is read element by element, from the stencil's first value on.
// The load/store pipe bounds it (its wavefronts at 89 % of their peak when a lane read a whole column,
// which is a line per lane and vector, and each rank had a butterfly): 139,968 atoms, p = 5, 4 ranks: float
// 207 -> 166 us, float64 321 -> 246; 12,000 atoms, p = 6, 5 ranks, float 62 -> 54; 20,736 atoms with the cell
// partials 78 -> 51. With the loads and reductions of one pass after the other it was a chain of nine memory
// waits per atom (float 218 us).
// TA: float sums for the orders and ranks of the mixed form that have always had them (launch rule),
// float64 otherwise. MC: the positions-fixed cell partials of the edge-list path too. ONE: all ranks are
// one chunk.
template <typename T, typename TA, int P, int RC, bool MC, bool ONE>
__global__ void __launch_bounds__(32 * kGatherWarps, RC == 8 ? 2 : 3) k_gather_z(
    MeshDev g, int n, const double* __restrict__ pos, double ps, const double* __restrict__ c6,
    const double* __restrict__ dc6, const CellInfo* __restrict__ ci, const Tables* __restrict__ tab,
    const int* __restrict__ order, const int4* __restrict__ rb, const T* __restrict__ rw, const T* __restrict__ rdw,
    const T* __restrict__ phi, double* __restrict__ gcn, double* __restrict__ gpos,
    double* __restrict__ mcell_part) {
  constexpr int VW = 16 / (int)sizeof(T);          // elements per 16-byte vector
  constexpr int NV = (VW - 1 + P + VW - 1) / VW;   // vectors covering a run at any offset
  constexpr int CPP = 32 / NV;                     // columns per pass
  constexpr int U = RC == 4 ? 2 : 1;               // passes whose loads are in flight together
  using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int t = blockIdx.x * kGatherWarps + wid;
  double mc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (t < n) {
    // two memory waits per atom: the record, then mesh, factors and their derivatives together
    const int R = g.R;
    const int i = order[t];
    const int4 b4 = rb[t];
    const T wl = lane < 3 * P ? rw[(size_t)t * 3 * P + lane] : T(0);
    const T dwl = lane < 3 * P ? rdw[(size_t)t * 3 * P + lane] : T(0);
    const int s = b4.w;
    const int n2 = g.n[2];
    const int iz0 = b4.z;
    const bool scalar = iz0 + P > n2 || (n2 % VW) != 0;   // warp-uniform
    const int o = scalar ? 0 : iz0 % VW;
    const int c0 = lane / NV, h = lane - c0 * NV;
    const int k0 = h * VW - o;   // stencil node of the vector's first element
    const bool mine = c0 < CPP && k0 < P;
    const size_t M = (size_t)g.n[0] * g.n[1] * n2;
    const double inv_vol = 1.0 / ci->volume;
    double gu0 = 0.0, gu1 = 0.0, gu2 = 0.0, gsum = 0.0;
    for (int rc0 = 0; rc0 < (ONE ? 1 : R); rc0 += RC) {
      const int nr = ONE || R - rc0 < RC ? R - rc0 : RC;
      // lane r: lambda_r c_r and the weight of P_r in g (below)
      double lc = 0.0, gp = 0.0;
      if (lane < nr) {
        const double lam = tab->eigs[rc0 + lane], dc = dc6[(size_t)i * R + rc0 + lane];
        lc = c6[(size_t)i * R + rc0 + lane] * lam;
        gp = -lam * inv_vol * dc;
        gsum += lc * tab->selfcont[s] * dc;
      }
      double pr[RC];
#pragma unroll
      for (int r = 0; r < RC; ++r) pr[r] = 0.0;
#pragma unroll 1
      for (int q0 = 0; q0 < P * P; q0 += U * CPP) {
        T v[U][RC][VW];
        int kx[U], ky[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          int q = q0 + u * CPP + c0;
          const bool ok = mine && q < P * P;
          if (!ok) q = 0;
          kx[u] = q / P;
          ky[u] = q - kx[u] * P;
          int ix = b4.x + kx[u];
          while (ix >= g.n[0]) ix -= g.n[0];   // a stencil wider than the mesh wraps more than once
          int iy = b4.y + ky[u];
          while (iy >= g.n[1]) iy -= g.n[1];
          const T* col = phi + ((size_t)s * R + rc0) * M + ((size_t)ix * g.n[1] + iy) * n2;
#pragma unroll
          for (int r = 0; r < RC; ++r)
#pragma unroll
            for (int j = 0; j < VW; ++j) v[u][r][j] = T(0);
          if (ok && !scalar) {
            // in the row: iz0 + P <= n2 and n2 is a multiple of VW, so the vector of a node below P is too
#pragma unroll
            for (int r = 0; r < RC; ++r)
              if (r < nr)
                *reinterpret_cast<V*>(v[u][r]) = *reinterpret_cast<const V*>(col + (size_t)r * M + (iz0 + k0));
          } else if (ok) {
#pragma unroll
            for (int j = 0; j < VW; ++j) {
              int iz = iz0 + k0 + j;
              while (iz >= n2) iz -= n2;
#pragma unroll
              for (int r = 0; r < RC; ++r)
                if (r < nr && k0 + j < P) v[u][r][j] = col[(size_t)r * M + iz];
            }
          }
        }
        T wz[VW], dwz[VW];
#pragma unroll
        for (int j = 0; j < VW; ++j) {
          const int k = k0 + j;
          const T w = __shfl_sync(kAll, wl, (2 * P + k) & 31), dw = __shfl_sync(kAll, dwl, (2 * P + k) & 31);
          wz[j] = k >= 0 && k < P ? w : T(0);
          dwz[j] = k >= 0 && k < P ? dw : T(0);
        }
        TA cp[U][VW];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int j = 0; j < VW; ++j) cp[u][j] = TA(0);
        TA wx[U], wy[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          wx[u] = (TA)__shfl_sync(kAll, wl, kx[u]);
          wy[u] = (TA)__shfl_sync(kAll, wl, P + ky[u]);
        }
#pragma unroll
        for (int r = 0; r < RC; ++r) {
          const TA cl = (TA)__shfl_sync(kAll, lc, r);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            TA zr = TA(0);
#pragma unroll
            for (int j = 0; j < VW; ++j) {
              const TA f = (TA)v[u][r][j];
              zr += (TA)wz[j] * f;
              cp[u][j] += cl * f;
            }
            pr[r] += (double)(wx[u] * wy[u] * zr);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          TA s0 = TA(0), s2 = TA(0);
#pragma unroll
          for (int j = 0; j < VW; ++j) {
            s0 += (TA)wz[j] * cp[u][j];
            s2 += (TA)dwz[j] * cp[u][j];
          }
          const TA dwx = (TA)__shfl_sync(kAll, dwl, kx[u]), dwy = (TA)__shfl_sync(kAll, dwl, P + ky[u]);
          gu0 += (double)(dwx * wy[u] * s0);
          gu1 += (double)(wx[u] * dwy * s0);
          gu2 += (double)(wx[u] * wy[u] * s2);
        }
      }
      // dE/dc_r = -(lambda_r / Omega) P_r + lambda_r c_r phi_ss(0); g = sum_r dE/dc_r dc_r/dCN: this lane's part
#pragma unroll
      for (int r = 0; r < RC; ++r) gsum += __shfl_sync(kAll, gp, r) * pr[r];
    }
    const double sum = warp_sum4(gu0, gu1, gu2, gsum);
    gu0 = __shfl_sync(kAll, sum, 0);
    gu1 = __shfl_sync(kAll, sum, 8);
    gu2 = __shfl_sync(kAll, sum, 16);
    if (lane == 24) gcn[i] = sum;
    if (lane == 0) {
      // dE/du_a = -(1/Omega) sum_r lambda_r c_r sum_m phi dW/du_a; dE/dx_b = sum_a dE/du_a n_a inv[b][a]
      const double du[3] = {-inv_vol * gu0, -inv_vol * gu1, -inv_vol * gu2};
      double gx[3];
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        gx[b] = du[0] * g.n[0] * ci->inv[3 * b + 0] + du[1] * g.n[1] * ci->inv[3 * b + 1] +
                du[2] * g.n[2] * ci->inv[3 * b + 2];
        gpos[3 * i + b] = gx[b];
      }
      // mesh part of dE/dcell with positions fixed: -sum_i s_iA g_ia (s = fractional coordinate)
      if constexpr (MC) {
        const double x0 = pos[3 * i] * ps, x1 = pos[3 * i + 1] * ps, x2 = pos[3 * i + 2] * ps;
#pragma unroll
        for (int A = 0; A < 3; ++A) {
          const double sf = x0 * ci->inv[A] + x1 * ci->inv[3 + A] + x2 * ci->inv[6 + A];
#pragma unroll
          for (int a = 0; a < 3; ++a) mc[3 * A + a] = sf * gx[a];
        }
      }
    }
  }
  if constexpr (MC) block_sum_store<9>(mc, mcell_part + 9 * blockIdx.x);
}

template <typename T, int P>
static int gather_r(const MeshGeom& mg, int blocks, int n, const double* pos, double ps, const double* c6,
                    const double* dc6, const CellInfo* ci, const Tables* tab, const int* order,
                    const int* key_start, const MeshRecords& rec, const T* phi, double* gcn, double* gpos,
                    double* mcell, int* n_mcell, cudaStream_t s) {
  // tile-staged gather (one CTA per (tile, species) key, the key's mesh box staged once by TMA)
  // for the fused path where its box fits two CTAs per SM, when asked for
  if (!mcell && mg.gather_tile == 1 && gather_tile_applies(mg, sizeof(T))) {
    *n_mcell = 0;
    return launch_gather_tile<T, P>(mg, n, c6, dc6, ci, tab, order, key_start, rec, phi, gcn, gpos, s);
  }
  const MeshDev g = to_dev(mg);
  *n_mcell = mcell ? blocks : 0;
  auto launch = [&](auto kern) {
    kern<<<blocks, 32 * kGatherWarps, 0, s>>>(g, n, pos, ps, c6, dc6, ci, tab, order, rec.b, (const T*)rec.w,
                                              (const T*)rec.dw, phi, gcn, gpos, mcell);
  };
  // 4 or 8 ranks in flight per lane (vectors of 16 bytes), in one chunk where they all fit
#define FD3_GATHER(TA, MC)                                         \
  (mg.R <= 4   ? launch(k_gather_z<T, TA, P, 4, MC, true>)         \
   : mg.R <= 8 ? launch(k_gather_z<T, TA, P, 8, MC, true>)         \
               : launch(k_gather_z<T, TA, P, 8, MC, false>))
  if (mcell) {
    FD3_GATHER(double, true);
  } else if constexpr (sizeof(T) == 4) {
    // float sums: up to 4 ranks at any order, up to 8 ranks up to order 5
    if (mg.R <= 4 || (mg.R <= 8 && P <= 5))
      FD3_GATHER(float, false);
    else
      FD3_GATHER(double, false);
  } else {
    FD3_GATHER(double, false);
  }
#undef FD3_GATHER
  FD3_LAUNCHED();
  return FD3_OK;
}

template <typename T>
int launch_gather(const MeshGeom& mg, int n, const double* pos, double pos_scale, const double* c6, const double* dc6, const CellInfo* ci, const Tables* tab, const int* order,
                  const int* key_start, const MeshRecords& rec, const T* phi, double* gcn, double* gpos,
                  double* mcell_part, int* n_blocks, cudaStream_t s) {
  const int blocks = (n + kGatherWarps - 1) / kGatherWarps;
  *n_blocks = 0;
  if (blocks == 0) return FD3_OK;
#define FD3_GATHER_CASE(PP)                                                                                      \
  case PP:                                                                                                       \
    return gather_r<T, PP>(mg, blocks, n, pos, pos_scale, c6, dc6, ci, tab, order, key_start, rec, phi, gcn, gpos, \
                           mcell_part, n_blocks, s);
  switch (mg.order) {
    FD3_GATHER_CASE(1)
    FD3_GATHER_CASE(2)
    FD3_GATHER_CASE(3)
    FD3_GATHER_CASE(4)
    FD3_GATHER_CASE(5)
    FD3_GATHER_CASE(6)
    FD3_GATHER_CASE(7)
    FD3_GATHER_CASE(8)
  }
#undef FD3_GATHER_CASE
  return FD3_EINVAL;
}

// instantiated once each, in fd3_spread_*.cu and fd3_gather_*.cu
extern template int launch_spread<float>(const MeshGeom&, int, const double*, const int*, const int*,
                                         const MeshRecords&, float*, cudaStream_t);
extern template int launch_spread<double>(const MeshGeom&, int, const double*, const int*, const int*,
                                          const MeshRecords&, double*, cudaStream_t);
extern template int launch_gather<float>(const MeshGeom&, int, const double*, double, const double*, const double*,
                                         const CellInfo*, const Tables*, const int*, const int*, const MeshRecords&,
                                         const float*, double*, double*, double*, int*, cudaStream_t);
extern template int launch_gather<double>(const MeshGeom&, int, const double*, double, const double*, const double*,
                                          const CellInfo*, const Tables*, const int*, const int*,
                                          const MeshRecords&, const double*, double*, double*, double*, int*,
                                          cudaStream_t);

}  // namespace fd3
