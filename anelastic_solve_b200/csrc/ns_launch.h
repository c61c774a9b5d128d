// ns_launch.h -- host launchers of the RK3 sub-step kernels.
#pragma once

#include "anel_internal.h"
#include "ns_device.cuh"

namespace anel {

// Device pointers of the column-independent CN factors of one variable.
// Column-independent CN data per row k = 1..nz+2 (index k-1): eliminated
// sub-diagonal ap and diagonal bp, super-diagonal c, explicit weights t1,
// t2, wall-row right-hand side rb and flag isbc, and the raw sub-diagonal
// and diagonal (the LES solve adds its eddy terms to these).
struct CNFacHost {
  const double *ap, *bp, *c, *t1, *t2, *rb, *isbc, *sub, *diag;
};

// The sub-step launchers below that take Ds[0..n) work on n members of one
// grid, models and boundary setup at once (an ensemble cohort; n = 1: a
// context of its own), with the members' own time steps.
void launch_rhs_accum(const NSDev* const* Ds, const double* dts, int n, double a1, double a2, bool first,
                      cudaStream_t s);
// One member's Crank-Nicolson factors: the destination (3 slots x 5
// variables x 9 arrays x Z), rkdt of each slot and the z wall types and
// values of u, v, w, rho, scal1; slots slot0 .. slot0 + nslots - 1 are made
struct CNFactorSet {
  double* dst;
  double rkdt[3];
  int type[5][2];
  double val[5][2];
};
void launch_cn_factors(const NSDev* const* Ds, const CNFactorSet* set, int n, int slot0, int nslots, cudaStream_t s);
// One variable's column solve (var_advance_CN_PL): var 1 u, 2 v, 3 w, 5 rho,
// 8 scal1; LES also its eddy coefficient kT (nuT for u, v, w, kappaT for
// rho, nappaT for scal1) and scratch b of its own for the eliminated
// diagonal (G values).
struct CNSet {
  int var;
  double* fld;
  const double* q;
  CNFacHost F;
  ZRule R;
  const double* kT;
  double* b;
};
// The column solves of nset <= 5 variables of each member (member m's at
// set[m * nset]) in one launch, then the periodic images of their fields.  variant: rows per load batch and columns per
// block (0: 8 rows, 256; 1: 16, 128; 2: 16, 256; 3: 32, 128; 4: 16, 32),
// chosen by the autotuner; every variant computes the same bits
constexpr int kCNVariants = 5;
void launch_cn(const NSDev* const* Ds, const CNSet* set, int nset, const double* rkdts, int n, double a3, int variant,
               cudaStream_t s);
// the same with the eddy terms (Vmodel = SSM): per-column elimination (the
// super-diagonal is formed again from kT in the back substitution).
// variant: 0: 8 rows, 256 columns; 1: 4, 128; 2: 8, 128; 3: 16, 128; 4: 8, 32
constexpr int kCNLesVariants = 5;
void launch_cn_les(const NSDev& D, const CNSet* set, int n, double a3, double rkdt, int variant, cudaStream_t s);
// SGSdiff (straincal.F90:339-414): modS, nuT, kappaT, nappaT on the
// interior from the model profiles, then their ghosts ('cfluc').
void launch_sgs(const NSDev& D, const ZRule& cfluc, cudaStream_t s);
void launch_psource(const NSDev* const* Ds, const double* dts, int n, cudaStream_t s);
// shear-layer initial state (NSSolver::init_shear): prof = tanh(zc)[Z],
// |zc|[Z]; noise from the Park-Miller sequence of seed, element q*G + c
// for u (q = 0), v (1), w (2) at Fortran linear index c.
void launch_init_shear(const NSDev& D, const double* prof, uint32_t seed, double amp, double zmax,
                       cudaStream_t s);
// hist (one member only; may be null): a copy of p's interior (pressure
// guess history)
void launch_pgrad(const NSDev* const* Ds, const double* dts, int n, const ZRule& Ru, const ZRule& Rv,
                  const ZRule& Rw, cudaStream_t s, double* hist = nullptr);
// p = 2 h1 - h2 on the interior (the extrapolated pressure guess)
void launch_extrap(const NSDev& D, double* p, const double* h1, const double* h2, cudaStream_t s);
void launch_ghost_field(const NSDev& D, double* a, const ZRule& R, cudaStream_t s);
void launch_ghost_fields2(const NSDev& D, double* a, double* b, const ZRule& R, cudaStream_t s);
// clipVS (Routines.F90:301-380) of a cell-centred field's interior
void launch_clip(const NSDev& D, double* a, double vmin, double vmax, cudaStream_t s);
void launch_cfl_max(const NSDev& D, unsigned long long* out, cudaStream_t s);
// plane statistics (NSsolver.F90:288-395): center_velocity of one
// component, squared fluctuations, weighted x-y plane averages of every
// plane (part: plane_part_doubles scratch) and the profile update
void launch_center(const NSDev& D, const double* in, double* out, int dir, int stretched, int corrected,
                   const double* e, const double* c, cudaStream_t s);
void launch_fluct_sq(const NSDev& D, const double* a, const double* mean, double* out, cudaStream_t s);
int64_t plane_part_doubles(const NSDev& D);
// the partial sums alone; returns their number per plane
int launch_plane_part(const NSDev& D, const double* a, const double* wx, const double* wy, double* part,
                      cudaStream_t s);
void launch_plane_avg(const NSDev& D, const double* a, const double* wx, const double* wy, double area,
                      double* part, double* out, cudaStream_t s);
void launch_diag_update(int Z, double dtt, const double* m, double* dg, cudaStream_t s);
// One member's divergence pass: partial sums (divergence_part_doubles), an
// arrival counter (zero), and the results sum |div| vol, sum vol, max |div|
// and, with cfl, calcdt's CFL maximum, in mapped host memory
struct DivSet {
  double* part;
  unsigned* count;
  double* host;
};
int64_t divergence_part_doubles(const NSDev& D);
void launch_divergence(const NSDev* const* Ds, const DivSet* set, int n, bool cfl, cudaStream_t s);

}  // namespace anel
