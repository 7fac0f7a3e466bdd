// Direct Ewald k-sum (reference: src/fourierd3/core.py:225-242, 563-577).
//
// k-vectors: the full Miller box of torch-pme's generate_kvectors_for_ewald, m_a in fftfreq order
// on every axis (k = 0 included), k = m0 b0 + m1 b1 + m2 b2. The reference weights rank r by
// sqrt(|lambda_r|) on both structure factors, i.e. the k-space energy uses |lambda_r| (the self
// term keeps the signed lambda_r); this is reproduced as is.
//
// exp(i k.x) factors into one phase per axis, exp(2 pi i m_a s_a) (s = fractional coordinate), so every
// phase the sums need comes from a table of N (n0 + n1 + n2) entries by two complex multiplications;
// a sincospi for each (atom, k) pair, twice per call, was most of the time (240 atoms, 39^3 k, 4
// species, 5 ranks, float64: the three sums 2,450 us before, 318 us now).
//
//   tables : e^{2 pi i m s} per atom (species-sorted) and Miller index of each axis, reduced to a
//            fraction of a turn before sincospi; in two layouts, one for each sum's lanes.
//   sf     : one thread per (m1, m2) and kEwM0 values of m0: S_X^r(k) = sum_{i in X} c_ir e^{i k.x_i},
//            lanes over m2.
//   filter : a CTA takes a tile of k: G_XY(|k|) of every species pair once, shared by the ranks,
//            energy and virial (float64 accumulation), H = G S.
//   gather : one thread per (atom, chunk of (m0, m1) rows), lanes over the atoms; partial sums reduced
//            per atom in a fixed order by one warp.
#include <math.h>

#include "fd3_internal.h"

namespace fd3 {

struct EwaldDev {
  int ns[3];
  int nk;
  int S, R;
};

__device__ __forceinline__ int fftfreq_order(int i, int n) { return i <= (n - 1) / 2 ? i : i - n; }

__device__ __forceinline__ void ewald_miller(const EwaldDev& e, int k, int& m0, int& m1, int& m2) {
  const int i2 = k % e.ns[2];
  const int i1 = (k / e.ns[2]) % e.ns[1];
  const int i0 = k / (e.ns[2] * e.ns[1]);
  m0 = fftfreq_order(i0, e.ns[0]);
  m1 = fftfreq_order(i1, e.ns[1]);
  m2 = fftfreq_order(i2, e.ns[2]);
}

template <typename T> struct Cplx2;
template <> struct Cplx2<double> { using type = double2; };
template <> struct Cplx2<float> { using type = float2; };

// Per sorted slot t: species, fractional coordinates s = x inv(cell) and the axis phases
// e^{2 pi i m s_a} at axis entry q (n0 entries of axis 0, then axis 1, then axis 2, fftfreq order).
// One thread per (slot, entry).
__global__ void __launch_bounds__(256) k_ewald_tables(EwaldDev e, int n, const double* __restrict__ pos, double ps,
                                                     const CellInfo* __restrict__ ci,
                                                     const int* __restrict__ order,
                                                     const int32_t* __restrict__ species, int4* __restrict__ sp_of,
                                                     double* __restrict__ frac, double2* __restrict__ by_atom,
                                                     double2* __restrict__ by_m) {
  const int ne = e.ns[0] + e.ns[1] + e.ns[2];
  const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (int64_t)n * ne) return;
  const int t = (int)(id / ne), q = (int)(id - (int64_t)t * ne);
  const int a = q < e.ns[0] ? 0 : q < e.ns[0] + e.ns[1] ? 1 : 2;
  const int m = fftfreq_order(a == 0 ? q : a == 1 ? q - e.ns[0] : q - e.ns[0] - e.ns[1], e.ns[a]);
  const int i = order[t];
  const double f = pos[3 * i] * ps * ci->inv[a] + pos[3 * i + 1] * ps * ci->inv[3 + a] +
                   pos[3 * i + 2] * ps * ci->inv[6 + a];
  const double turns = m * f;
  double sn, cs;
  sincospi(2.0 * (turns - rint(turns)), &sn, &cs);
  by_atom[id] = make_double2(cs, sn);
  by_m[(size_t)q * n + t] = make_double2(cs, sn);
  if (m == 0) frac[3 * t + a] = f;
  if (q == 0) sp_of[t] = make_int4(species[i], 0, 0, 0);
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

constexpr int kEwSfThreads = 128;
// m0 values per thread: its accumulators are 2 M0 MAXR float64 values
template <int MAXR>
struct EwSf {
  static constexpr int kM0 = MAXR <= 8 ? 4 : MAXR <= 16 ? 2 : 1;
};

template <typename T, int MAXR>
__global__ void __launch_bounds__(kEwSfThreads) k_ewald_sf(EwaldDev e, const double2* __restrict__ ph,
                                                          const int* __restrict__ order,
                                                          const int* __restrict__ sp_start,
                                                          const double* __restrict__ c6,
                                                          typename Cplx2<T>::type* __restrict__ spec) {
  using C2 = typename Cplx2<T>::type;
  constexpr int M0 = EwSf<MAXR>::kM0;
  constexpr int kTile = 32;
  __shared__ double s_c[kTile][MAXR];
  __shared__ double2 s_e0[kTile][M0];
  const int R = e.R, n12 = e.ns[1] * e.ns[2], ne = e.ns[0] + e.ns[1] + e.ns[2];
  const int p = blockIdx.x * kEwSfThreads + threadIdx.x;   // (m1, m2)
  const int i0 = blockIdx.y * M0;
  const bool on = p < n12;
  const int i1 = on ? p / e.ns[2] : 0, i2 = on ? p - i1 * e.ns[2] : 0;
  for (int X = 0; X < e.S; ++X) {
    double are[M0][MAXR], aim[M0][MAXR];
#pragma unroll
    for (int u = 0; u < M0; ++u)
#pragma unroll
      for (int r = 0; r < MAXR; ++r) are[u][r] = aim[u][r] = 0.0;
    const int a0 = sp_start[X], a1 = sp_start[X + 1];
    for (int t0 = a0; t0 < a1; t0 += kTile) {
      const int cnt = min(kTile, a1 - t0);
      __syncthreads();
      for (int q = threadIdx.x; q < cnt * MAXR; q += kEwSfThreads) {
        const int j = q / MAXR, r = q - j * MAXR;
        s_c[j][r] = r < R ? c6[(size_t)order[t0 + j] * R + r] : 0.0;
      }
      for (int q = threadIdx.x; q < cnt * M0; q += kEwSfThreads) {
        const int j = q / M0, u = q - j * M0;
        s_e0[j][u] = ph[(size_t)(t0 + j) * ne + min(i0 + u, e.ns[0] - 1)];
      }
      __syncthreads();
      const double2* row = ph + (size_t)t0 * ne + e.ns[0];
#pragma unroll 2
      for (int j = 0; j < cnt; ++j, row += ne) {
        const double2 e12 = cmul(row[i1], row[e.ns[1] + i2]);
#pragma unroll
        for (int u = 0; u < M0; ++u) {
          const double2 z = cmul(e12, s_e0[j][u]);
#pragma unroll
          for (int r = 0; r < MAXR; ++r) {
            are[u][r] += s_c[j][r] * z.x;
            aim[u][r] += s_c[j][r] * z.y;
          }
        }
      }
    }
    if (on) {
#pragma unroll
      for (int u = 0; u < M0; ++u)
        if (i0 + u < e.ns[0]) {
#pragma unroll
          for (int r = 0; r < MAXR; ++r)
            if (r < R)
              spec[((size_t)X * R + r) * e.nk + (size_t)(i0 + u) * n12 + p] = C2{(T)are[u][r], (T)aim[u][r]};
        }
    }
  }
}

// Tile of KT k-points: phase 1, one thread per (k, species pair): G and dG/d|k| to shared memory;
// phase 2, one thread per (k, channel): H = sum_Y G S_Y, its share of the energy and virial.
constexpr int kEwFilterThreads = 256;
constexpr int kEwFilterSmem = 40 * 1024;

template <typename T>
__global__ void __launch_bounds__(kEwFilterThreads) k_ewald_filter(EwaldDev e, int KT,
                                                     const CellInfo* __restrict__ ci,
                                                     const GreenPair* __restrict__ gp, const Tables* __restrict__ tab,
                                                     const typename Cplx2<T>::type* __restrict__ spec,
                                                     typename Cplx2<T>::type* __restrict__ hout,
                                                     double* __restrict__ part) {
  using C2 = typename Cplx2<T>::type;
  extern __shared__ __align__(16) unsigned char ewf_raw[];
  T* g = reinterpret_cast<T*>(ewf_raw);             // [pairs][KT]
  const int S = e.S, R = e.R, NP = S * (S + 1) / 2;
  T* dg = g + (size_t)NP * KT;
  const int kk = threadIdx.x % KT, slot = threadIdx.x / KT, nslot = kEwFilterThreads / KT;
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  const T s6 = (T)tab->s6, s8 = (T)tab->s8;
  for (int k0 = blockIdx.x * KT; k0 < e.nk; k0 += gridDim.x * KT) {
    const int k = k0 + kk;
    const bool on = k < e.nk;
    int m0, m1, m2;
    ewald_miller(e, on ? k : 0, m0, m1, m2);
    double kv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) kv[c] = m0 * ci->recip[c] + m1 * ci->recip[3 + c] + m2 * ci->recip[6 + c];
    const double knorm = sqrt(kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2]);
    __syncthreads();   // the previous tile has been read
    for (int pr = slot; pr < NP; pr += nslot) {
      int X = 0, base = 0;   // pair pr: X <= Y, row X starts at X S - X (X - 1) / 2
      while (base + S - X <= pr) base += S - X++;
      T gv, dv;
      green_eval<T>(gp[X * S + X + (pr - base)], (T)knorm, s6, s8, gv, dv);
      g[pr * KT + kk] = gv;
      dg[pr * KT + kk] = dv;
    }
    __syncthreads();
    double qq = 0.0, dq = 0.0;
    for (int c = slot; on && c < S * R; c += nslot) {
      const int X = c / R, r = c - X * R;
      T hre = T(0), him = T(0), dre = T(0), dim = T(0);
      int pr = X;   // pair (Y, X) for Y < X, then (X, Y)
      for (int Y = 0; Y < S; ++Y) {
        const C2 sy = spec[((size_t)Y * R + r) * e.nk + k];
        const T gv = g[pr * KT + kk], dv = dg[pr * KT + kk];
        pr += Y < X ? S - Y - 1 : 1;
        hre += gv * sy.x;
        him += gv * sy.y;
        dre += dv * sy.x;
        dim += dv * sy.y;
      }
      const C2 sx = spec[(size_t)c * e.nk + k];
      const double lam = fabs(tab->eigs[r]);
      qq += lam * ((double)sx.x * hre + (double)sx.y * him);
      dq += lam * ((double)sx.x * dre + (double)sx.y * dim);
      hout[(size_t)c * e.nk + k] = C2{hre, him};
    }
    acc[0] += qq;
    if (on && knorm > 0.0) {
      const double f = dq / knorm;
      acc[1] += f * kv[0] * kv[0];
      acc[2] += f * kv[1] * kv[1];
      acc[3] += f * kv[2] * kv[2];
      acc[4] += f * kv[0] * kv[1];
      acc[5] += f * kv[0] * kv[2];
      acc[6] += f * kv[1] * kv[2];
    }
  }
  block_sum_store<7>(acc, part + 7 * blockIdx.x);
}

constexpr int kEwGatherThreads = 128;

// Partial sums of one atom over the (m0, m1) rows of one chunk: P_r = sum_k Re(e^{i phi} conj H_r) and
// U = sum_k k sum_r |lambda_r| c_r (-sin phi H_r.re + cos phi H_r.im)  (phi = k.x).
template <typename T, int MAXR>
__global__ void __launch_bounds__(kEwGatherThreads) k_ewald_gather(EwaldDev e, int n, int rows,
                                                     const double2* __restrict__ ph,
                                                     const int* __restrict__ order, const int4* __restrict__ sp_of,
                                                     const double* __restrict__ c6, const Tables* __restrict__ tab,
                                                     const typename Cplx2<T>::type* __restrict__ h,
                                                     double* __restrict__ gpart, int nchunk) {
  using C2 = typename Cplx2<T>::type;
  const int t = blockIdx.x * kEwGatherThreads + threadIdx.x;    // atom slot (species-sorted)
  const int chunk = blockIdx.y;
  const int R = e.R;
  if (t >= n) return;
  const int i = order[t];
  const int X = sp_of[t].x;
  double cl[MAXR];
#pragma unroll
  for (int r = 0; r < MAXR; ++r) cl[r] = r < R ? c6[(size_t)i * R + r] * fabs(tab->eigs[r]) : 0.0;
  double pr[MAXR];
#pragma unroll
  for (int r = 0; r < MAXR; ++r) pr[r] = 0.0;
  double u0 = 0, u1 = 0, u2 = 0;
  const int nrow = e.ns[0] * e.ns[1];
  const int r0 = chunk * rows, r1 = min(nrow, r0 + rows);
  for (int row = r0; row < r1; ++row) {
    const int i0 = row / e.ns[1], i1 = row - i0 * e.ns[1];
    const double2 e01 = cmul(ph[(size_t)i0 * n + t], ph[(size_t)(e.ns[0] + i1) * n + t]);
    const double2* p2 = ph + (size_t)(e.ns[0] + e.ns[1]) * n + t;
    const C2* hr = h + (size_t)X * R * e.nk + (size_t)row * e.ns[2];
    double ur = 0.0;
    for (int i2 = 0; i2 < e.ns[2]; ++i2) {
      const double2 z = cmul(e01, p2[(size_t)i2 * n]);
      double u = 0.0;
#pragma unroll
      for (int r = 0; r < MAXR; ++r) {
        if (r < R) {
          const C2 hv = hr[(size_t)r * e.nk + i2];
          pr[r] += z.x * (double)hv.x + z.y * (double)hv.y;
          u += cl[r] * (z.x * (double)hv.y - z.y * (double)hv.x);
        }
      }
      // u multiplies the Cartesian k = m0 b0 + m1 b1 + m2 b2; accumulate per Miller axis
      ur += u;
      u2 += u * fftfreq_order(i2, e.ns[2]);
    }
    u0 += ur * fftfreq_order(i0, e.ns[0]);
    u1 += ur * fftfreq_order(i1, e.ns[1]);
  }
  double* out = gpart + ((size_t)t * nchunk + chunk) * (R + 3);
#pragma unroll
  for (int r = 0; r < MAXR; ++r)
    if (r < R) out[r] = pr[r];
  out[R] = u0;
  out[R + 1] = u1;
  out[R + 2] = u2;
}

// Per atom (one warp): the chunks summed lane by lane in a fixed order, then dE/dc -> dE/dCN, the
// force and the cell term.
__global__ void __launch_bounds__(256) k_ewald_finish(EwaldDev e, int n, const double* __restrict__ frac,
                                                     const int* __restrict__ order, const int4* __restrict__ sp_of,
                                                     const double* __restrict__ c6, const double* __restrict__ dc6,
                                                     const CellInfo* __restrict__ ci, const Tables* __restrict__ tab,
                                                     const double* __restrict__ gpart, int nchunk,
                                                     double* __restrict__ gcn, double* __restrict__ gpos,
                                                     double* __restrict__ mcell_part) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int R = e.R;
  double mc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (t < n) {
    const int i = order[t];
    const int X = sp_of[t].x;
    const double* src = gpart + (size_t)t * nchunk * (R + 3);
    const double inv_vol = 1.0 / ci->volume;
    double gsum = 0.0, u[3] = {0, 0, 0};
    for (int q = 0; q < R + 3; ++q) {
      double v = 0.0;
      for (int c = lane; c < nchunk; c += 32) v += src[(size_t)c * (R + 3) + q];
      v = warp_sum(v);
      if (q < R) {
        const double lam = tab->eigs[q];
        gsum += (-fabs(lam) * inv_vol * v + lam * c6[(size_t)i * R + q] * tab->selfcont[X]) * dc6[(size_t)i * R + q];
      } else {
        u[q - R] = v;
      }
    }
    // dE/dx = -(1/Omega) sum_k k (...) with k = sum_a m_a b_a  ->  -(1/Omega) sum_a U_a b_a
    if (lane == 0) {
      double gx[3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
        gx[c] = -inv_vol * (u[0] * ci->recip[c] + u[1] * ci->recip[3 + c] + u[2] * ci->recip[6 + c]);
      gcn[i] = gsum;
      gpos[3 * i] = gx[0];
      gpos[3 * i + 1] = gx[1];
      gpos[3 * i + 2] = gx[2];
      if (mcell_part) {
#pragma unroll
        for (int A = 0; A < 3; ++A)
#pragma unroll
          for (int a = 0; a < 3; ++a) mc[3 * A + a] = frac[3 * t + A] * gx[a];
      }
    }
  }
  if (mcell_part) block_sum_store<9>(mc, mcell_part + 9 * blockIdx.x);
}

__global__ void __launch_bounds__(256) k_species_keys(int n, const int32_t* __restrict__ species,
                                                     int* __restrict__ keys) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) keys[i] = species[i];
}

// Gather chunks of (m0, m1) rows per atom: enough (atom, chunk) threads to fill the chip, at least
// four rows each.
int ewald_chunks(int64_t n, const int* ns) {
  const int64_t nrow = (int64_t)ns[0] * ns[1];
  int64_t want = (148 * 1024 + n - 1) / n;
  if (want > (nrow + 3) / 4) want = (nrow + 3) / 4;
  if (want > 65535) want = 65535;
  const int64_t rows = (nrow + want - 1) / want;
  return (int)((nrow + rows - 1) / rows);
}

// (atom, chunk) pairs that the workspace holds for n atoms: no fewer than n ewald_chunks(n), and no fewer
// than for any smaller n, so that a workspace made for more atoms serves fewer.
int64_t ewald_gather_slots(int64_t n, const int* ns) {
  const int64_t by_rows = n * (((int64_t)ns[0] * ns[1] + 3) / 4), by_chip = 148 * 1024 + n;
  return by_rows < by_chip ? by_rows : by_chip;
}

template <typename T>
int launch_ewald(const EwaldGeom& eg, int n, const double* pos, double ps, const int32_t* species,
                 const double* c6, const double* dc6, const CellInfo* ci, const GreenPair* gp, const Tables* tab,
                 const EwaldWork& w, bool need_grad, double* gcn, double* gpos, double* mcell_part, int* n_kspc,
                 int* n_mcell, cudaStream_t s) {
  using C2 = typename Cplx2<T>::type;
  EwaldDev e;
  for (int a = 0; a < 3; ++a) e.ns[a] = eg.ns[a];
  e.nk = eg.ns[0] * eg.ns[1] * eg.ns[2];
  e.S = eg.S;
  e.R = eg.R;
  if (e.R > FD3_MAX_RANK) return FD3_EINVAL;
  const int tb = 256;
  // species-sorted atom order
  k_species_keys<<<(n + tb - 1) / tb, tb, 0, s>>>(n, species, w.keys);
  FD3_LAUNCHED();
  int rc = counting_sort(w.keys, n, e.S, w.counts, w.sp_start, w.order, reinterpret_cast<int*>(w.sp_of), s);
  if (rc) return rc;
  const int64_t entries = (int64_t)n * (e.ns[0] + e.ns[1] + e.ns[2]);
  k_ewald_tables<<<(unsigned)((entries + tb - 1) / tb), tb, 0, s>>>(e, n, pos, ps, ci, w.order, species, w.sp_of,
                                                                    w.frac, w.ph_atom, w.ph_m);
  FD3_LAUNCHED();
  C2* spec = reinterpret_cast<C2*>(w.spec);
  C2* hsp = reinterpret_cast<C2*>(w.hspec);
  const int n12 = e.ns[1] * e.ns[2];
#define FD3_EW_SF(RR)                                                                                            \
  k_ewald_sf<T, RR><<<dim3((n12 + kEwSfThreads - 1) / kEwSfThreads, (e.ns[0] + EwSf<RR>::kM0 - 1) / EwSf<RR>::kM0), \
                      kEwSfThreads, 0, s>>>(e, w.ph_atom, w.order, w.sp_start, c6, spec)
  if (e.R <= 4)
    FD3_EW_SF(4);
  else if (e.R <= 6)
    FD3_EW_SF(6);
  else if (e.R <= 8)
    FD3_EW_SF(8);
  else if (e.R <= 16)
    FD3_EW_SF(16);
  else
    FD3_EW_SF(32);
#undef FD3_EW_SF
  FD3_LAUNCHED();
  // k-points per filter tile: as many, up to a warp, as the pairs leave shared memory for
  const size_t per_k = (size_t)e.S * (e.S + 1) * sizeof(T);
  int KT = 32;
  while (KT > 1 && KT * per_k > kEwFilterSmem) KT >>= 1;
  const int tiles = (e.nk + KT - 1) / KT;
  const int fb = tiles < 148 * 8 ? tiles : 148 * 8;
  k_ewald_filter<T><<<fb, kEwFilterThreads, KT * per_k, s>>>(e, KT, ci, gp, tab, spec, hsp, w.kpart);
  FD3_LAUNCHED();
  *n_kspc = fb;
  *n_mcell = 0;
  if (!need_grad) return FD3_OK;
  const int nchunk = ewald_chunks(n, e.ns);
  const int rows = (e.ns[0] * e.ns[1] + nchunk - 1) / nchunk;
  const dim3 gg((n + kEwGatherThreads - 1) / kEwGatherThreads, nchunk);
#define FD3_EW_GATHER(RR)                                                                                      \
  k_ewald_gather<T, RR><<<gg, kEwGatherThreads, 0, s>>>(e, n, rows, w.ph_m, w.order, w.sp_of, c6, tab, hsp, w.gpart, \
                                                        nchunk)
  if (e.R <= 4)
    FD3_EW_GATHER(4);
  else if (e.R <= 8)
    FD3_EW_GATHER(8);
  else if (e.R <= 16)
    FD3_EW_GATHER(16);
  else
    FD3_EW_GATHER(32);
#undef FD3_EW_GATHER
  FD3_LAUNCHED();
  const int ab = (n + 7) / 8;
  k_ewald_finish<<<ab, tb, 0, s>>>(e, n, w.frac, w.order, w.sp_of, c6, dc6, ci, tab, w.gpart, nchunk, gcn, gpos,
                                   mcell_part);
  FD3_LAUNCHED();
  *n_mcell = mcell_part ? ab : 0;
  return FD3_OK;
}

template int launch_ewald<double>(const EwaldGeom&, int, const double*, double, const int32_t*, const double*,
                                  const double*, const CellInfo*, const GreenPair*, const Tables*, const EwaldWork&,
                                  bool, double*, double*, double*, int*, int*, cudaStream_t);
template int launch_ewald<float>(const EwaldGeom&, int, const double*, double, const int32_t*, const double*,
                                 const double*, const CellInfo*, const GreenPair*, const Tables*, const EwaldWork&,
                                 bool, double*, double*, double*, int*, int*, cudaStream_t);

}  // namespace fd3
