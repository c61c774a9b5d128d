// mg_rb.h -- the FP64 red-black cycle on x/y-periodic levels with one
// coefficient per direction in x and y (mg_rb.cu).
#pragma once

#include "mg_launch.h"

namespace anel {

// A level whose half-sweeps write their own ghosts: nx, ny even (a cell's
// periodic images are then read by the other colour only), z walls.
struct RBLevel {
  int nx, ny, nz, X;
  int64_t XY;
  double* phi;
  const double* src;
  double a1, a2, a3, a4;
  const double* zc;   // a5[Z], a6[Z], diagonal[Z]
  int n1, nZ;         // z-min / z-max Neumann (else Dirichlet: ghosts constant)
  double add1, addZ;  // the Neumann additions (value * spacing)
};
void launch_rb_march(const RBLevel& L, int color, cudaStream_t s);

// Levels 1..lc of the cycle in one block, phi and f in shared memory.
constexpr int kRBSharedLevels = 10;
constexpr size_t kRBSharedBytes = 220 << 10;
struct RBShared {
  int lc;
  DevLevel<double> L[kRBSharedLevels + 1];   // [1..lc]
  int pre[kRBSharedLevels + 1], post[kRBSharedLevels + 1];
  int cd[kRBSharedLevels + 1];               // directions coarsened from l + 1 to l
  unsigned mh[kRBSharedLevels + 1], mx[kRBSharedLevels + 1], my[kRBSharedLevels + 1];  // dividers of cell indices
  int coef[kRBSharedLevels + 1], ghost[kRBSharedLevels + 1], phi[kRBSharedLevels + 1]; // shared-memory offsets
  int nblob, res;
  size_t bytes;
  // the levels' coefficients and homogeneous ghost tables (ghost cell << 16
  // | interior cell it copies, or 0xffff for zero), as they lie in shared
  // memory
  const double* blob;
};
// phi += the interpolated correction of the coarse level, ghosts included
void launch_rb_prolong(const RBLevel& L, const DevLevel<double>& F, const DevLevel<double>& C, int cdir,
                       cudaStream_t s);
// whether levels 1..l fit (their L, cd filled in), and their layout
bool rb_shared_fits(RBShared& S, int l);
void rb_shared_prepare();
// level lc's f from global memory, its corrected phi (ghosts too) to it
void launch_rb_shared(const RBShared& S, cudaStream_t s);

// max|phin|, max|phin - phio| over the interior and phio <- phin on the whole array
void launch_relmax_copy(const DevLevel<double>& L, const double* phin, double* phio, unsigned long long* out,
                        cudaStream_t s);

}  // namespace anel
