// mg_rb.cu -- the FP64 red-black point smoother's cycle on x/y-periodic
// levels.  Compiled with -fmad=false: every value is rounded as in
// k_rb_sweep, k_restrict and k_prolong, whose expressions these are.
#include "mg_rb.h"
#include "pdl.cuh"

namespace anel {

// v at interior cell (i, j, k), offset c, and at the ghosts that copy it
__device__ __forceinline__ void rb_put(const RBLevel& L, int64_t c, int i, int64_t oy, int k, double v) {
  const int ox = i == 2 ? L.nx : (i == L.nx + 1 ? -L.nx : 0);
  auto put = [&](int64_t at, double x) {
    L.phi[at] = x;
    if (ox) L.phi[at + ox] = x;
    if (oy) L.phi[at + oy] = x;
    if (ox && oy) L.phi[at + ox + oy] = x;
  };
  put(c, v);
  if (k == 2 && L.n1) put(c - L.XY, v - L.add1);
  if (k == L.nz + 1 && L.nZ) put(c + L.XY, v + L.addZ);
}
// the y shift to the image of row j (0: none)
__device__ __forceinline__ int64_t rb_yshift(const RBLevel& L, int j) {
  return j == 2 ? (int64_t)L.ny * L.X : (j == L.ny + 1 ? -(int64_t)L.ny * L.X : 0);
}

// One half-sweep of mg_relaxRB (mg_relax.F90:146-168) and the boundary pass
// after it.  The boundary pass rewrites every ghost from the interior cell
// it copies; here the thread that updates such a cell writes its images, so
// a half-sweep is one launch.  A thread takes U planes of one pair of
// columns, loads before stores: the planes' cells are of one colour and
// read the other one only.  256x128x128: 31 us and 5 us for the two
// launches before.
template <int U>
__global__ void __launch_bounds__(128) k_rb_march(RBLevel L, int color) {
  chain_enter();
  const int hx = L.nx >> 1;
  const int col = blockIdx.x * 128 + threadIdx.x;
  if (col >= hx * L.ny) return;
  const int j = 2 + col / hx, q = col - (j - 2) * hx;
  const int k0 = 2 + blockIdx.y * U;
  const int Z = L.nz + 2, X = L.X;
  const int64_t XY = L.XY;
  const int64_t row = (int64_t)X * (j - 1) + XY * (k0 - 1);
  double v[U];
  int64_t c[U];
  int ii[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int k = k0 + u;
    ii[u] = 2 + 2 * q + ((color + j + k) & 1);
    c[u] = row + u * XY + (ii[u] - 1);
    if (k <= L.nz + 1) {
      const double* p = L.phi + c[u];
      double acc = L.a1 * p[-1];
      acc = acc + L.a2 * p[1];
      acc = acc + L.a3 * p[-X];
      acc = acc + L.a4 * p[X];
      acc = acc + L.zc[k - 1] * p[-XY];
      acc = acc + L.zc[Z + k - 1] * p[XY];
      v[u] = (L.src[c[u]] - acc) / L.zc[2 * Z + k - 1];
    }
  }
  const int64_t oy = rb_yshift(L, j);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (k0 + u <= L.nz + 1) rb_put(L, c[u], ii[u], oy, k0 + u, v[u]);
}

void launch_rb_march(const RBLevel& L, int color, cudaStream_t s) {
  const int cols = ((L.nx / 2) * L.ny + 127) / 128;
  // four planes per thread where that still gives two blocks per SM
  if ((int64_t)cols * ((L.nz + 3) / 4) >= 2 * 148)
    launch_chained(k_rb_march<4>, dim3((unsigned)cols, (unsigned)((L.nz + 3) / 4)), 128, 0, s, L, color);
  else
    launch_chained(k_rb_march<1>, dim3((unsigned)cols, (unsigned)L.nz), 128, 0, s, L, color);
  count_launch();
}

// mg_cor.F90:102-290 (k_prolong) with the boundary pass after it.
constexpr int kRBProlongK = 4;
template <int CD>
__global__ void __launch_bounds__(128) k_rb_prolong(RBLevel L, DevLevel<double> F, DevLevel<double> C) {
  chain_enter();
  const int col = blockIdx.x * 128 + threadIdx.x;
  if (col >= L.nx * L.ny) return;
  const int j = 2 + col / L.nx, i = 2 + col - (j - 2) * L.nx;
  const int k0 = 2 + blockIdx.y * kRBProlongK;
  const int64_t c0 = cidx(i, j, k0, L.X, L.XY), oy = rb_yshift(L, j);
  double v[kRBProlongK];
#pragma unroll
  for (int u = 0; u < kRBProlongK; ++u)
    if (k0 + u <= L.nz + 1) v[u] = L.phi[c0 + u * L.XY] + prolong_corr<double, CD>(C, i, j, k0 + u);
#pragma unroll
  for (int u = 0; u < kRBProlongK; ++u)
    if (k0 + u <= L.nz + 1) rb_put(L, c0 + u * L.XY, i, oy, k0 + u, v[u]);
}

void launch_rb_prolong(const RBLevel& L, const DevLevel<double>& F, const DevLevel<double>& C, int cdir,
                       cudaStream_t s) {
  const dim3 g((unsigned)((L.nx * L.ny + 127) / 128), (unsigned)((L.nz + kRBProlongK - 1) / kRBProlongK));
  switch (cdir & 7) {
    case 0: launch_chained(k_rb_prolong<0>, g, 128, 0, s, L, F, C); break;
    case 1: launch_chained(k_rb_prolong<1>, g, 128, 0, s, L, F, C); break;
    case 2: launch_chained(k_rb_prolong<2>, g, 128, 0, s, L, F, C); break;
    case 3: launch_chained(k_rb_prolong<3>, g, 128, 0, s, L, F, C); break;
    case 4: launch_chained(k_rb_prolong<4>, g, 128, 0, s, L, F, C); break;
    case 5: launch_chained(k_rb_prolong<5>, g, 128, 0, s, L, F, C); break;
    case 6: launch_chained(k_rb_prolong<6>, g, 128, 0, s, L, F, C); break;
    default: launch_chained(k_rb_prolong<7>, g, 128, 0, s, L, F, C); break;
  }
  count_launch();
}

// ---------------------------------------------------- coarse levels
// The levels of at most kRBSharedCells cells and everything below them in
// one block: their half-sweeps are 1000 to 4 cells long and as separate
// launches cost 6 us each, about 60 of them per cycle.  phi and f stay in
// shared memory; boundary passes go by the ghost tables.  An 8192-cell
// level fits too, but one SM takes longer over it than its launches
// (256x128x128 solve: 39.1 ms with it, 34.3 without; 128x64x128 step with
// the 2048-cell level 20.0, without 20.2).
constexpr int kRBThreads = 512;

__device__ __forceinline__ unsigned rb_magic(int d) { return (unsigned)((0x100000000ull + d - 1) / (unsigned)d); }
__device__ __forceinline__ int rb_div(int u, int d, unsigned m) { return d == 1 ? u : (int)__umulhi((unsigned)u, m); }

__device__ __forceinline__ int rb_ghosts(const DevLevel<double>& L) { return (int)L.G - L.nx * L.ny * L.nz; }

__device__ __forceinline__ void rb_bdry(const DevLevel<double> L, const int2* __restrict__ gt) {
  const int n = rb_ghosts(L);
  for (int g = threadIdx.x; g < n; g += kRBThreads) {
    const int2 e = gt[g];
    L.phi[e.x] = e.y >= 0 ? L.phi[e.y] : 0.0;
  }
  __syncthreads();
}

__device__ __forceinline__ void rb_relax(const DevLevel<double> L, const int2* __restrict__ gt, int iters) {
  const int hx = (L.nx + 1) >> 1, n = hx * L.ny * L.nz;
  const unsigned mx = rb_magic(hx), my = rb_magic(L.ny);
  for (int it = 0; it < 2 * iters; ++it) {
    const int color = it & 1;
    for (int t = threadIdx.x; t < n; t += kRBThreads) {
      const int r = rb_div(t, hx, mx), q = t - r * hx;
      const int kk = rb_div(r, L.ny, my);
      const int k = 2 + kk, j = 2 + r - kk * L.ny;
      const int i = 2 + ((color + j + k) & 1) + 2 * q;
      if (i > L.nx + 1) continue;
      const int64_t c = cidx(i, j, k, L.X, L.XY);
      L.phi[c] = stencil_update(L, (const double*)L.phi, L.src[c], c, i, j, k);
    }
    __syncthreads();
    rb_bdry(L, gt);
  }
}

template <int CD>
__device__ __forceinline__ void rb_restrict(const DevLevel<double> F, const DevLevel<double> C) {
  const int n = C.nx * C.ny * C.nz;
  for (int t = threadIdx.x; t < (int)C.G; t += kRBThreads) C.phi[t] = 0.0;
  for (int t = threadIdx.x; t < n; t += kRBThreads) {
    const int i = 2 + t % C.nx, r = t / C.nx, j = 2 + r % C.ny, k = 2 + r / C.ny;
    C.src[cidx(i, j, k, C.X, C.XY)] = restrict_value<double, CD>(F, i, j, k);
  }
  __syncthreads();
}

template <int CD>
__device__ __forceinline__ void rb_prolong(const DevLevel<double> F, const DevLevel<double> C) {
  const int n = F.nx * F.ny * F.nz;
  for (int t = threadIdx.x; t < n; t += kRBThreads) {
    const int i = 2 + t % F.nx, r = t / F.nx, j = 2 + r % F.ny, k = 2 + r / F.ny;
    const int64_t c = cidx(i, j, k, F.X, F.XY);
    F.phi[c] = F.phi[c] + prolong_corr<double, CD>(C, i, j, k);
  }
  __syncthreads();
}

#define RB_BY_CD(cd, call)        \
  switch ((cd) & 7) {             \
    case 0: call<0>(F, C); break; \
    case 1: call<1>(F, C); break; \
    case 2: call<2>(F, C); break; \
    case 3: call<3>(F, C); break; \
    case 4: call<4>(F, C); break; \
    case 5: call<5>(F, C); break; \
    case 6: call<6>(F, C); break; \
    default: call<7>(F, C); break; \
  }

__host__ __device__ inline int rb_coefs(int X, int Y, int Z) { return 2 * X + 2 * Y + 4 * Z; }

__global__ void __launch_bounds__(kRBThreads) k_rb_shared(const __grid_constant__ RBShared S) {
  chain_enter();
  extern __shared__ double rsm[];
  __shared__ DevLevel<double> lv[kRBSharedLevels + 1];
  if (threadIdx.x == 0) {
    double* at = rsm;
    for (int l = 1; l <= S.lc; ++l) {
      DevLevel<double> L = S.L[l];
      L.phi = at;
      L.src = at + L.G;
      L.coef = at + 2 * L.G;
      at += 2 * L.G + rb_coefs(L.X, L.Y, L.Z);
      lv[l] = L;
    }
  }
  __syncthreads();
  for (int l = 1; l <= S.lc; ++l) {
    const DevLevel<double>& L = lv[l];
    const int n = rb_coefs(L.X, L.Y, L.Z);
    for (int t = threadIdx.x; t < n; t += kRBThreads) const_cast<double*>(L.coef)[t] = S.L[l].coef[t];
  }
  const int G = (int)lv[S.lc].G;
  for (int t = threadIdx.x; t < G; t += kRBThreads) {
    lv[S.lc].phi[t] = 0.0;
    lv[S.lc].src[t] = S.L[S.lc].src[t];
  }
  __syncthreads();
  // the schedule of mg_cycle.F90:186-325 between the restriction to level
  // lc and the prolongation from it
  for (int l = S.lc; l >= 2; --l) {
    rb_relax(lv[l], S.gt[l], S.pre[l]);
    const DevLevel<double>&F = lv[l], &C = lv[l - 1];
    RB_BY_CD(S.cd[l - 1], rb_restrict);
  }
  rb_relax(lv[1], S.gt[1], S.pre[1]);
  for (int l = 1; l < S.lc; ++l) {
    rb_relax(lv[l], S.gt[l], S.post[l]);
    const DevLevel<double>&F = lv[l + 1], &C = lv[l];
    RB_BY_CD(S.cd[l], rb_prolong);
    rb_bdry(lv[l + 1], S.gt[l + 1]);
  }
  rb_relax(lv[S.lc], S.gt[S.lc], S.post[S.lc]);
  for (int t = threadIdx.x; t < G; t += kRBThreads) S.L[S.lc].phi[t] = lv[S.lc].phi[t];
}

size_t rb_shared_bytes(const RBShared& S) {
  size_t n = 0;
  for (int l = 1; l <= S.lc; ++l) n += 2 * (size_t)S.L[l].G + rb_coefs(S.L[l].X, S.L[l].Y, S.L[l].Z);
  return n * sizeof(double);
}

void rb_shared_prepare() { set_smem_limit_once((const void*)k_rb_shared, (int)kRBSharedBytes); }

void launch_rb_shared(const RBShared& S, cudaStream_t s) {
  launch_chained(k_rb_shared, 1, kRBThreads, rb_shared_bytes(S), s, S);
  count_launch();
}

// ---------------------------------------------------------- stop test
// mg_residual.F90:60-105 over the whole ghosted array, four values per
// thread loaded before the first is stored (ghosts are copied only); the
// maxima of non-negative doubles by their bit patterns, exact in any order,
// one atomic pair per block.  256x128x128: 66 us with one value at a time.
constexpr int kMaxU = 4;
__global__ void __launch_bounds__(256) k_relmax_copy(DevLevel<double> L, const double* __restrict__ phin,
                                                     double* __restrict__ phio, unsigned long long* out) {
  chain_enter();
  __shared__ unsigned long long sh[2][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long m1 = 0, m2 = 0;
  for (int64_t t0 = (int64_t)blockIdx.x * 256 * kMaxU + threadIdx.x; t0 < L.G; t0 += (int64_t)gridDim.x * 256 * kMaxU) {
    double n[kMaxU], o[kMaxU];
#pragma unroll
    for (int u = 0; u < kMaxU; ++u) {
      const int64_t t = t0 + u * 256;
      n[u] = t < L.G ? phin[t] : 0.0;
      o[u] = t < L.G ? phio[t] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kMaxU; ++u) {
      const int64_t t = t0 + u * 256;
      if (t >= L.G) break;
      phio[t] = n[u];
      const int k = (int)(t / L.XY), r = (int)(t - k * L.XY), j = r / L.X, i = r - j * L.X;
      if (i >= 1 && i <= L.nx && j >= 1 && j <= L.ny && k >= 1 && k <= L.nz) {
        const unsigned long long a = __double_as_longlong(fabs(n[u]));
        const unsigned long long d = __double_as_longlong(fabs(n[u] - o[u]));
        m1 = a > m1 ? a : m1;
        m2 = d > m2 ? d : m2;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, m1, o), b = __shfl_xor_sync(0xffffffffu, m2, o);
    m1 = a > m1 ? a : m1;
    m2 = b > m2 ? b : m2;
  }
  if (lane == 0) {
    sh[0][wid] = m1;
    sh[1][wid] = m2;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned long long m = 0;
    for (int q = 0; q < 8; ++q) m = sh[threadIdx.x][q] > m ? sh[threadIdx.x][q] : m;
    atomicMax(out + threadIdx.x, m);
  }
}

void launch_relmax_copy(const DevLevel<double>& L, const double* phin, double* phio, unsigned long long* out,
                        cudaStream_t s) {
  const int64_t b = (L.G + 256 * kMaxU - 1) / (256 * kMaxU);
  launch_chained(k_relmax_copy, (unsigned)(b < 148 * 8 ? b : 148 * 8), 256, 0, s, L, phin, phio, out);
  count_launch();
}

}  // namespace anel
