// Many-species filter of the mixed form (16 to 64 species, at most 8 ranks): per k-point
// H_X = sum_Y G_XY S_Y over S x S species pairs and the ranks, with the energy and the virial.
// (reference: src/fourierd3/kspace_filter_d3.py:29-70, src/fourierd3/pair_pot.py:113-228)
//
// A CTA takes KT consecutive k-points at a time, as k_filter_tiled does: spectrum tile and the pairs'
// Gh in shared memory, phase B over the pairs X <= Y (Green function, energy, virial), phase C over the
// species (H in place). At 54 species and 8 ranks a k-point takes 1,485 pair functions, 23,760 multiply-adds
// for the pair sums and 46,656 for H; instruction issue and shared-memory loads bound it (16 warps per SM). So
//   * phase B works on blocks of 4 x 4 species: 8 rows loaded serve 16 pairs;
//   * a row keeps a (species, k)'s ranks side by side, so one 16-byte load brings two of them (rows
//     RP + 2 values apart: eight lanes' 16-byte loads fall on distinct banks);
//   * multiply-adds are packed (fma.rn.f32x2), real and imaginary part in one instruction.
// 64^3, 8 ranks: 54 species 1,705 us against 1,856 for k_filter_tiled, which loads a row per pair; 26 species 528
// against 715; 32^3, 16 species, 5 ranks 48 against 63. k_filter_tiled stays for float64, more ranks and
// fewer species (10 species: 4 x 4 blocks leave most slots idle). Interpolating G across the pairs from
// per-k nodes in sqrt(qq) instead of reading each pair's table over |k| was slower (2,027 us: more
// shared-memory loads, and the table's 32 bytes per pair and k are not what bounds the kernel).
#include "fd3_filter.cuh"

namespace fd3 {

namespace {

using u64 = unsigned long long;

__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 pack2(float x, float y) {
  u64 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(u64 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

constexpr int kManyThreads = 256;
constexpr int kManyWide = 40;   // species up to which two CTAs' tiles of 16 k-points fit an SM; tiles of 8 beyond

template <int KT, int RP>
struct Many {
  static constexpr int kRow = RP + 2;          // complex values from one (species, k) to the next
  static constexpr int kSlots = kManyThreads / KT;
  static size_t smem(int S) {
    const size_t S4 = (size_t)(S + 3) / 4 * 4, np = (size_t)S * (S + 1) / 2, nt = S4 / 4;
    return S4 * KT * kRow * sizeof(float2) + np * KT * sizeof(float) + nt * (nt + 1) / 2 * sizeof(int);
  }
};

template <int KT, int RP>
__global__ void __launch_bounds__(kManyThreads, 2)
    k_filter_many(MeshDev g, int P, int spme, const CellInfo* __restrict__ ci, const float4* __restrict__ gtab,
                  const Tables* __restrict__ tab, const float* __restrict__ deconv, float2* __restrict__ spec,
                  double* __restrict__ part) {
  using M = Many<KT, RP>;
  extern __shared__ __align__(16) unsigned char many_raw[];
  const int S = g.S, R = g.R, S4 = (S + 3) / 4 * 4, nt = S4 / 4, NP = S * (S + 1) / 2, nu = nt * (nt + 1) / 2;
  float2* ss = reinterpret_cast<float2*>(many_raw);               // [S4][KT][kRow]
  float* gs = reinterpret_cast<float*>(ss + (size_t)S4 * KT * M::kRow);   // [NP][KT]
  int* units = reinterpret_cast<int*>(gs + (size_t)NP * KT);      // block a | block b << 16, a <= b
  for (int u = threadIdx.x; u < nu; u += kManyThreads) {
    int a = 0, base = 0;
    while (base + nt - a <= u) base += nt - a++;
    units[u] = a | ((a + u - base) << 16);
  }
  // zero rows and ranks beyond S and R: they enter the blocks and contribute nothing
  for (int e = threadIdx.x; e < S4 * KT * M::kRow; e += kManyThreads) ss[e] = make_float2(0.f, 0.f);
  const size_t Mh = (size_t)g.n[0] * g.n[1] * g.nzh;
  const size_t ntile = (Mh + KT - 1) / KT;
  const int kk = threadIdx.x % KT, slot = threadIdx.x / KT;
  u64 lam[RP];
#pragma unroll
  for (int r = 0; r < RP; ++r) {
    const float l = r < R ? (float)tab->eigs[r] : 0.f;
    lam[r] = pack2(l, l);
  }
  float rc[9];
  load_recip<float>(ci, rc);
  const float inv_h = green_inv_h(g, ci);
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  auto row0 = [&](int X) { return X * S - X * (X - 1) / 2; };
  for (size_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const size_t k0 = tile * KT;
    __syncthreads();   // the previous tile's phase C has finished with ss and gs
    for (int e = threadIdx.x; e < S * R * KT; e += kManyThreads) {
      const int c = e / KT, j = e % KT, X = c / R, r = c - X * R;
      const size_t k = k0 + j;
      ss[(X * KT + j) * M::kRow + r] = k < Mh ? spec[(size_t)c * Mh + k] : make_float2(0.f, 0.f);
    }
    const size_t k = k0 + kk;
    const bool valid = k < Mh;
    const KPoint<float> q = kpoint<float>(g, valid ? k : 0, rc, deconv, spme, P);
    int tj = 0, pj = 0;
    HermiteF hb{}, pb{};
    table_pos(q.knorm, inv_h, tj, hb);
    table_pos(q.kpart, inv_h, pj, pb);
    __syncthreads();
    float qq = 0.f, dq = 0.f;
    for (int u = slot; u < nu; u += M::kSlots) {
      const int xa = (units[u] & 0xffff) * 4, yb = (units[u] >> 16) * 4;
      const float2* sx = ss + (xa * KT + kk) * M::kRow;
      const float2* sy = ss + (yb * KT + kk) * M::kRow;
      u64 pr[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) pr[i][j] = 0ull;
#pragma unroll
      for (int r = 0; r < RP; r += 2) {
        ulonglong2 x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[i] = *reinterpret_cast<const ulonglong2*>(sx + i * KT * M::kRow + r);
          y[i] = *reinterpret_cast<const ulonglong2*>(sy + i * KT * M::kRow + r);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[i].x = mul2(x[i].x, lam[r]);
          x[i].y = mul2(x[i].y, lam[r + 1]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) pr[i][j] = fma2(x[i].y, y[j].y, fma2(x[i].x, y[j].x, pr[i][j]));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int X = xa + i;
        float4 ta[4], tb[4];
        const int p0 = row0(X) - X + yb;   // pair (X, yb + j) at p0 + j
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (X <= yb + j && yb + j < S) {
            const float4* row = gtab + (size_t)(p0 + j) * (kGreenKnots + 1) + tj;
            ta[j] = row[0];
            tb[j] = row[1];
          } else {
            ta[j] = tb[j] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (X <= yb + j && yb + j < S) {
            const float2 p2 = unpack2(pr[i][j]);
            const float w = X == yb + j ? p2.x + p2.y : 2.f * (p2.x + p2.y);
            const float gv = herm_value(hb, ta[j], tb[j]) * q.inv_sc;
            const float dv = herm_slope(hb, ta[j], tb[j]) * inv_h * q.inv_sc;
            float gh = gv;
            if (q.partner) {
              float gpv, dpv;
              green_lookup(gtab + (size_t)(p0 + j) * (kGreenKnots + 1), pj, pb, inv_h, gpv, dpv);
              gh = 0.5f * (gv + gpv * q.inv_sc);
            }
            qq += gv * w;
            dq += dv * w;
            gs[(p0 + j) * KT + kk] = gh;
          }
      }
    }
    if (valid) {
      acc[0] += (double)(q.wk * qq);
      virial_acc<float>(q, dq, acc);
    }
    __syncthreads();
    // two species per thread (X and X + kSlots): every staged row serves both
    for (int X = slot; X < S; X += 2 * M::kSlots) {
      const int X2 = X + M::kSlots;
      const bool two = X2 < S;
      u64 h[RP], h2[RP];
#pragma unroll
      for (int r = 0; r < RP; ++r) h[r] = h2[r] = 0ull;
      // pair index of (X, Y): row0(Y) + (X - Y) for Y < X, row0(X) + (Y - X) for Y >= X
      int pa = X, pc = two ? X2 : 0;
      const float2* sy = ss + kk * M::kRow;
      for (int Y = 0; Y < S; ++Y, sy += KT * M::kRow) {
        const float g1 = gs[pa * KT + kk], g2 = two ? gs[pc * KT + kk] : 0.f;
        const u64 gg = pack2(g1, g1), gg2 = pack2(g2, g2);
        pa += Y < X ? S - Y - 1 : 1;
        pc += Y < X2 ? S - Y - 1 : 1;
#pragma unroll
        for (int r = 0; r < RP; r += 2) {
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(sy + r);
          h[r] = fma2(gg, y.x, h[r]);
          h[r + 1] = fma2(gg, y.y, h[r + 1]);
          h2[r] = fma2(gg2, y.x, h2[r]);
          h2[r + 1] = fma2(gg2, y.y, h2[r + 1]);
        }
      }
      if (valid) {
#pragma unroll
        for (int r = 0; r < RP; ++r)
          if (r < R) {
            spec[((size_t)X * R + r) * Mh + k] = unpack2(h[r]);
            if (two) spec[((size_t)X2 * R + r) * Mh + k] = unpack2(h2[r]);
          }
      }
    }
  }
  block_sum_store<7>(acc, part + 7 * blockIdx.x);
}

template <int KT, int RP>
int launch_many_t(const MeshGeom& mg, const CellInfo* ci, const float4* gtab, const Tables* tab, const float* deconv,
                  int spme, float2* spec, double* part, int* n_blocks, cudaStream_t s) {
  const size_t smem = Many<KT, RP>::smem(mg.S);
  const int rc = allow_dynamic_smem(k_filter_many<KT, RP>, Many<KT, RP>::smem(KT == 16 ? kManyWide : FD3_MAX_SPECIES));
  if (rc) return rc;
  const size_t Mh = (size_t)mg.n[0] * mg.n[1] * mg.nzh, ntile = (Mh + KT - 1) / KT;
  const size_t most = 148 * 2;   // two CTAs per SM, persistent over the tiles
  const int blocks = (int)(ntile < most ? ntile : most);
  *n_blocks = blocks;
  k_filter_many<KT, RP><<<blocks, kManyThreads, smem, s>>>(to_dev(mg), mg.order, spme, ci, gtab, tab, deconv, spec,
                                                          part);
  FD3_LAUNCHED();
  return FD3_OK;
}

}  // namespace

bool filter_many_applies(const MeshGeom& mg) {
  return mg.S >= 16 && mg.S <= FD3_MAX_SPECIES && mg.R <= 8 && mg.filter_kt < 0;
}

int launch_filter_many(const MeshGeom& mg, const CellInfo* ci, const float4* gtab, const Tables* tab,
                       const float* deconv, int spme, void* spec, double* part, int* n_blocks, cudaStream_t s) {
  float2* sp = reinterpret_cast<float2*>(spec);
#define FD3_MANY(KT, RP) launch_many_t<KT, RP>(mg, ci, gtab, tab, deconv, spme, sp, part, n_blocks, s)
  if (mg.S <= kManyWide) return mg.R <= 4 ? FD3_MANY(16, 4) : FD3_MANY(16, 8);
  return mg.R <= 4 ? FD3_MANY(8, 4) : FD3_MANY(8, 8);
#undef FD3_MANY
}

}  // namespace fd3
