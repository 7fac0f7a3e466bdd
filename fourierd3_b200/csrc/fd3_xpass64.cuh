// Float64 x-pass: forward FFT along x, the reciprocal-space filter, inverse FFT along x, on pencils of
// the (y, z)-transformed spectrum (layout and register passes as in fd3_xfilter.cuh: one y, KZ
// consecutive kz, every x, every channel in shared memory, transformed, filtered and written in place).
// (reference: src/fourierd3/kspace_filter_d3.py:29-70, src/fourierd3/pair_pot.py:113-228)
//
// In float64 the Green function is the work: three exponentials and three sine-cosine pairs per
// species pair and k-point, about 300 instructions with CUDA's functions, half with TabTrig's. A thread that
// evaluates all pairs of its k-point holds 3 S (S + 1) / 2 values through long chains (255 registers, 8 warps
// per SM; and on a small mesh the chain is the kernel's time). Here a chunk of kPts points is filtered
// at a time: geometry once per point, then one (point, pair) evaluation per thread, G, dG and the
// Hermitian-averaged Gh to shared memory, then one (point, rank) per thread for H = Gh S, the energy and the
// virial. Two CTAs of 256 threads per SM wherever two pencils fit, so that one loads and stores while the
// other computes. (One thread for all pairs of a point, one CTA of 256 threads: 128^3, 4 species, 5 ranks
// 728 us, 64^3 128 us; with a pair per thread 600 and 87; with TabTrig too 557 and 76. 16^3 and 32^3, which had
// 3D cuFFT around the separate filter: 64 and 45 us, then 33 and 32 with the plane transforms.)
#pragma once
#include "fd3_xfilter.cuh"

namespace fd3 {

constexpr size_t kX64Smem = 224 * 1024;   // of the 227 KB that a CTA may have, 2 KB being static

struct X64Shape {
  int LKZ, two;   // pencil width 2^LKZ; two CTAs of 256 threads per SM, else one of 512
};

template <int MAXS>
struct X64Chunk {
  static constexpr int kPts = MAXS <= 2 ? 128 : 64;
  static constexpr int kPairs = MAXS * (MAXS + 1) / 2;
  static constexpr int kDoubles = kPts * (3 + 3 * kPairs);   // |k|, 1/window, partner |k| | G | dG | Gh
};

template <int N1, int N2>
__host__ __device__ constexpr size_t x64_smem(int C, int LKZ, int MAXS) {
  using L = XLayout<N1, N2>;
  return ((size_t)L::TW + ((size_t)C * L::PC << LKZ)) * sizeof(double2) +
         ((MAXS <= 2 ? X64Chunk<2>::kDoubles : X64Chunk<4>::kDoubles) + TabTrig::kDoubles) * sizeof(double);
}

template <int N1, int N2, int LKZ, int MAXS, int NT>
__global__ void __launch_bounds__(NT, 512 / NT)
    k_xpass64(MeshDev g, int P, int spme, const CellInfo* __restrict__ ci, const GreenPair* __restrict__ gp,
              const Tables* __restrict__ tab, const float* __restrict__ deconv, double2* __restrict__ spec,
              double* __restrict__ part) {
  using L = XLayout<N1, N2>;
  constexpr int NX = L::NX, KZ = 1 << LKZ;
  constexpr int kPts = X64Chunk<MAXS>::kPts, kPairs = X64Chunk<MAXS>::kPairs;
  extern __shared__ __align__(16) unsigned char xd_raw[];
  double2* tw = reinterpret_cast<double2*>(xd_raw);   // [n2][k1] exp(-2 pi i n2 k1 / NX), rows of N1 + 1
  double2* buf = tw + L::TW;
  const int S = g.S, R = g.R, C = S * R, NP = S * (S + 1) / 2;
  constexpr int CSC = L::PC << LKZ;
  double* trig = reinterpret_cast<double*>(buf + (size_t)C * CSC);
  for (int i = threadIdx.x; i < TabTrig::kDoubles / 2; i += NT)   // waited for with the first pencil
    copy_async16(trig + 2 * i, tab->trig + 2 * i);
  double* kn = trig + TabTrig::kDoubles;   // [kPts] each
  double* isc = kn + kPts;
  double* kpart = isc + kPts;          // partner |k|, or -1
  double* sG = kpart + kPts;           // [kPairs][kPts]
  double* sdG = sG + kPairs * kPts;
  double* sGh = sdG + kPairs * kPts;
  const int n1 = g.n[1], nzh = g.nzh;
  const size_t xrow = (size_t)n1 * nzh;
  for (int m = threadIdx.x; m < L::TW; m += NT) {
    const int a = m / (N1 + 1), b = m % (N1 + 1);
    double sn, cs;
    sincospi(-2.0 * ((a * b) % NX) / NX, &sn, &cs);
    tw[m] = make_double2(cs, sn);
  }
  const int ngz = (nzh + KZ - 1) >> LKZ;
  const int ngroups = n1 * ngz;
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  const double s6 = tab->s6, s8 = tab->s8;
  for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    const int y = grp / ngz, kz0 = (grp - y * ngz) << LKZ;
    double2* src = spec + (size_t)y * nzh + kz0;
    __syncthreads();   // twiddles written; the previous pencil has been stored
    for (int i = threadIdx.x; i < (C * NX) << LKZ; i += NT) {
      const int j = i & (KZ - 1), cx = i >> LKZ, c = cx >> L::LNX, x = cx & (NX - 1);
      double2* d = buf + c * CSC + (((x >> L::LN2) * L::ROW + (x & (N2 - 1))) << LKZ) + j;
      if (kz0 + j < nzh)
        copy_async(d, src + (size_t)cx * xrow + j);
      else
        *d = make_double2(0.0, 0.0);
    }
    copy_async_wait_all();
    __syncthreads();
    xfft_forward<double, N1, N2>(buf, tw, C, LKZ);
    for (int p0 = 0; p0 < NX << LKZ; p0 += kPts) {
      const int npt = (NX << LKZ) - p0 < kPts ? (NX << LKZ) - p0 : kPts;
      // geometry
      for (int q = threadIdx.x; q < npt; q += NT) {
        const int pt = p0 + q, j = pt & (KZ - 1), pos = pt >> LKZ;
        const int iz = kz0 + j, ix = (pos >> L::LN2) + N1 * (pos & (N2 - 1));
        double k = -1.0, w = 0.0, kp = -1.0;
        if (iz < nzh) {
          double rc[9];
          load_recip<double>(ci, rc);
          const KPoint<double> kpt =
              kpoint_idx<double>(g, ix, y, iz, ((size_t)ix * n1 + y) * nzh + iz, rc, deconv, spme, P);
          k = kpt.knorm;
          w = kpt.inv_sc;
          if (kpt.partner) kp = kpt.kpart;
        }
        kn[q] = k;
        isc[q] = w;
        kpart[q] = kp;
      }
      __syncthreads();
      // Green function: one (pair, point) per thread
      for (int it = threadIdx.x; it < NP * kPts; it += NT) {
        const int pr = it / kPts, q = it & (kPts - 1);
        if (q >= npt || kn[q] < 0.0) continue;   // kz beyond the half spectrum
        int X = 0, base = 0;   // pair pr: X <= Y, row X starts at X S - X (X - 1) / 2
        while (base + S - X <= pr) base += S - X++;
        const GreenPair& pair = gp[X * S + X + (pr - base)];
        double gv, dv;
        green_eval<double>(pair, kn[q], s6, s8, gv, dv, TabTrig{trig});
        const double w = isc[q];
        gv *= w;
        double gh = gv;
        if (kpart[q] >= 0.0) {
          double g2, d2;
          green_eval<double>(pair, kpart[q], s6, s8, g2, d2, TabTrig{trig});
          gh = 0.5 * (gv + g2 * w);
        }
        sG[it] = gv;
        sdG[it] = dv * w;
        sGh[it] = gh;
      }
      __syncthreads();
      // H = Gh S, energy and virial: one (rank, point) per thread
      for (int it = threadIdx.x; it < R * kPts; it += NT) {
        const int r = it / kPts, q = it & (kPts - 1);
        if (q >= npt || kn[q] < 0.0) continue;
        const int pt = p0 + q, j = pt & (KZ - 1), pos = pt >> LKZ;
        const int iz = kz0 + j, i1 = pos >> L::LN2, i2 = pos & (N2 - 1), ix = i1 + N1 * i2;
        double2* v = buf + r * CSC + ((i1 * L::ROW + i2) << LKZ) + j;
        const int xs = R * CSC;   // channel stride between species
        double2 s[MAXS], h[MAXS];
#pragma unroll
        for (int X = 0; X < MAXS; ++X) {
          s[X] = X < S ? v[X * xs] : make_double2(0.0, 0.0);
          h[X] = make_double2(0.0, 0.0);
        }
        double qr = 0.0, dqr = 0.0;
        int pr = 0;
#pragma unroll
        for (int X = 0; X < MAXS; ++X)
#pragma unroll
          for (int Y = X; Y < MAXS; ++Y)
            if (Y < S) {   // pairs in the order of the table
              const double gv = sG[pr * kPts + q], dv = sdG[pr * kPts + q], gh = sGh[pr * kPts + q];
              ++pr;
              const double re = (X == Y ? 1.0 : 2.0) * (s[X].x * s[Y].x + s[X].y * s[Y].y);
              qr += gv * re;
              dqr += dv * re;
              h[X].x += gh * s[Y].x;
              h[X].y += gh * s[Y].y;
              if (X != Y) {
                h[Y].x += gh * s[X].x;
                h[Y].y += gh * s[X].y;
              }
            }
#pragma unroll
        for (int X = 0; X < MAXS; ++X)
          if (X < S) v[X * xs] = h[X];
        const double lw = tab->eigs[r] * ((iz == 0 || iz == nzh - 1) ? 1.0 : 2.0);   // lambda, Hermitian weight
        acc[0] += lw * qr;
        const double k = kn[q];
        if (k > 0.0) {
          const int mx = ix <= (NX - 1) / 2 ? ix : ix - NX, my = y <= (n1 - 1) / 2 ? y : y - n1;
          const double f = lw * dqr / k;
          double kv[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) kv[c] = mx * ci->recip[c] + my * ci->recip[3 + c] + iz * ci->recip[6 + c];
          acc[1] += f * kv[0] * kv[0];
          acc[2] += f * kv[1] * kv[1];
          acc[3] += f * kv[2] * kv[2];
          acc[4] += f * kv[0] * kv[1];
          acc[5] += f * kv[0] * kv[2];
          acc[6] += f * kv[1] * kv[2];
        }
      }
      __syncthreads();   // the chunk's tables may be overwritten
    }
    xfft_inverse<double, N1, N2>(buf, tw, C, LKZ);
    for (int i = threadIdx.x; i < (C * NX) << LKZ; i += NT) {
      const int j = i & (KZ - 1), cx = i >> LKZ, c = cx >> L::LNX, x = cx & (NX - 1);
      if (kz0 + j < nzh)
        src[(size_t)cx * xrow + j] = buf[c * CSC + (((x >> L::LN2) * L::ROW + (x & (N2 - 1))) << LKZ) + j];
    }
  }
  block_sum_store<7>(acc, part + 7 * blockIdx.x);
}

// ------------------------------------------------------------------ launch
struct X64Args {
  const MeshGeom* mg;
  const CellInfo* ci;
  const GreenPair* gp;
  const Tables* tab;
  const float* deconv;
  int spme;
  double2* spec;
  double* part;
  int* n_blocks;
  cudaStream_t s;
};

template <int N1, int N2, int LKZ, int MAXS, int NT>
static int launch_x64_t(const X64Args& a) {
  const MeshGeom& mg = *a.mg;
  const size_t smem = x64_smem<N1, N2>(mg.S * mg.R, LKZ, MAXS);
  auto kern = k_xpass64<N1, N2, LKZ, MAXS, NT>;
  if (smem > 40 * 1024) {   // (a few KB are static)
    const int rc = allow_dynamic_smem(kern, kX64Smem);
    if (rc) return rc;
  }
  const long long ngroups = (long long)mg.n[1] * ((mg.nzh + (1 << LKZ) - 1) >> LKZ);
  long long blocks = 148LL * (512 / NT);
  if (blocks > ngroups) blocks = ngroups;
  *a.n_blocks = (int)blocks;
  kern<<<(int)blocks, NT, smem, a.s>>>(to_dev(mg), mg.order, a.spme, a.ci, a.gp, a.tab, a.deconv, a.spec, a.part);
  FD3_LAUNCHED();
  return FD3_OK;
}

template <int N1, int N2, int LKZ>
static int launch_x64_kz(const X64Args& a, bool two) {
  if (a.mg->S <= 2)
    return two ? launch_x64_t<N1, N2, LKZ, 2, 256>(a) : launch_x64_t<N1, N2, LKZ, 2, 512>(a);
  return two ? launch_x64_t<N1, N2, LKZ, 4, 256>(a) : launch_x64_t<N1, N2, LKZ, 4, 512>(a);
}

template <int N1, int N2>
int launch_x64(const X64Args& a, X64Shape sh) {
  if (sh.LKZ == 2) return launch_x64_kz<N1, N2, 2>(a, sh.two != 0);
  if (sh.LKZ == 1) return launch_x64_kz<N1, N2, 1>(a, sh.two != 0);
  return launch_x64_kz<N1, N2, 0>(a, sh.two != 0);
}

// Pencil width and CTA shape for this mesh, LKZ = -1 where the x-pass does not apply: the widest pencil
// of 2 or 4 values that fits twice per SM beside its chunk tables, else the widest that fits once
// (128^3, 4 species, 5 ranks, with CUDA's functions: 2 values twice 600 us, 4 values once 728; with TabTrig
// 64^3: 4 values twice 76, 2 values twice 82); from there on the width that makes the rounds of the chip the
// shortest: a pencil costs its kz values and about 1200 / (C nx) of one more. (A narrower one only below 148
// pencils left half of the chip idle: whole calls of 64 atoms, 4 species, 5 ranks, 64 x 64 x 32 128 -> 111 us,
// 128 x 64 x 16 134 -> 116; 2 species, 4 ranks, 256 x 32 x 16 85 -> 73.)
template <int N1, int N2>
inline X64Shape x64_shape_t(const MeshGeom& mg) {
  const int C = mg.S * mg.R, most = mg.xpencil == 1 ? 0 : mg.xpencil == 2 ? 1 : 2;
  X64Shape sh{-1, 0};
  for (int pass = 0; pass < 2 && sh.LKZ < 0; ++pass)
    for (int l = most; l >= (pass == 0 && most > 0 ? 1 : 0); --l)
      if (x64_smem<N1, N2>(C, l, mg.S) + 2048 <= (pass == 0 ? (size_t)113 * 1024 : kX64Smem)) {
        sh = X64Shape{l, pass == 0 ? 1 : 0};
        break;
      }
  if (mg.xpencil < 0) {
    const long long slots = sh.two ? 2 * 148 : 148;
    double least = 0.0;
    for (int l = sh.LKZ, widest = sh.LKZ; l >= 0; --l) {
      const long long pencils = (long long)mg.n[1] * ((mg.nzh + (1 << l) - 1) >> l);
      const double cost = (double)((pencils + slots - 1) / slots) * ((1 << l) + 1200.0 / (C * mg.n[0]));
      if (l == widest || cost < least) {
        least = cost;
        sh.LKZ = l;
      }
    }
  }
  return sh;
}

inline X64Shape x64_shape(const MeshGeom& mg) {
  if (mg.S > 4 || mg.R > 8) return X64Shape{-1, 0};
  switch (mg.n[0]) {
    case 16: return x64_shape_t<4, 4>(mg);
    case 32: return x64_shape_t<4, 8>(mg);
    case 64: return x64_shape_t<8, 8>(mg);
    case 128: return x64_shape_t<8, 16>(mg);
    case 256: return x64_shape_t<16, 16>(mg);
  }
  return X64Shape{-1, 0};
}

}  // namespace fd3
