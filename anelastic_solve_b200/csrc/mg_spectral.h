// mg_spectral.h -- host side of the direct fine-level solve (mg_spectral.cuh).
#pragma once

#include <vector>

#include "mg_spectral.cuh"

namespace anel {

struct SpecHost {
  SpecDev d{};
  double* d_tab = nullptr;    // twiddles, eigenvalues, z tables
  double* d_buf = nullptr;    // states, arrival counters, partial sums
  SpecState* h_st = nullptr;  // the states' mirror, mapped
  SpecState* h_one = nullptr; // the caller's mapped memory for one member
  int cap = 0;                // members the buffers above have room for
  bool ok = false;
};

// whether the passes handle the extents
bool spec_supported(int nx, int ny, int nz);
// Tables of a fine level with line coefficients a1 (x), a3 (y), z
// coefficients indexed k-1 and homogeneous z-ghosts z1/zZ (1: copy of the
// adjacent row, 0: zero).  coef: the level's device cz5[Z] cz6[Z] dz5[Z] dz6[Z].
// h_one: mapped host memory for one member's state.
int spec_build(SpecHost& H, SpecState* h_one, int nx, int ny, int nz, double a1, double a3, const double* cz5, const double* cz6,
               const double* dz5, const double* dz6, int z1, int zZ, const double* coef);
void spec_free(SpecHost& H);
// buffers for n members
int spec_reserve(SpecHost& H, int n);
// doubles of spectral work space of one member
inline int64_t spec_work_doubles(int nx, int ny, int nz) { return (int64_t)nx * ny * nz; }

// residual and x transform; test: fold the norms and set the states
void launch_spec_forward(const SpecDev& D, int nm, bool test, cudaStream_t s);
// y transform, z-systems, inverse y transform, inverse x transform and
// phi += e, for the active members
void launch_spec_y(const SpecDev& D, int nm, bool inverse, cudaStream_t s);
void launch_spec_z(const SpecDev& D, int nm, cudaStream_t s);
void launch_spec_update(const SpecDev& D, int nm, cudaStream_t s);
// residual norm of the corrected phi and the next states
void launch_spec_check(const SpecDev& D, int nm, cudaStream_t s);

}  // namespace anel
