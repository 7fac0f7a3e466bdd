// Arguments of a call's preparation (kernels in fd3_prep.cuh).
#pragma once
#include "fd3_mesh_impl.cuh"
#include "fd3_sort.cuh"

namespace fd3 {

struct PrepDev {
  int n;
  const double* pos;
  double ps;                  // positions to Bohr (the bins take them as they are)
  const int32_t* species;     // null: bins alone, no species
  // bins
  GridDev g;
  int K;                      // number of bins, 0: no cell list
  double4* xs;
  int4 *meta, *off;
  int *bin_start, *bslot, *btmp;
  // mesh
  MeshDev m;
  int P, Km;                  // Km: number of (tile, species) keys, 0: no mesh
  int *mkeys, *mslot, *mtmp, *mstart, *morder;   // mslot ends as the sorted slot of each atom
  int4* rb;
  void *rw, *rdw;
  int* counts;                // [K + Km], zeroed (k_prep_small: unused)
  // cell: the caller's (use_host), copied into *ci, or the one that *ci holds already
  int use_host;
  CellInfo host;
  const double* d_cell;       // the same cell on the device, compared with host_cell (null: not compared)
  double host_cell[9];
  CellInfo* ci;
  // Green table (null: none)
  const GreenPair* gp;
  const Tables* tab;
  float4* gtab;
};

}  // namespace fd3
