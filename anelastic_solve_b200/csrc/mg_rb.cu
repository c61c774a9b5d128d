// mg_rb.cu -- the FP64 red-black point smoother's cycle on x/y-periodic
// levels.  Compiled with -fmad=false: every value is rounded as in
// k_rb_sweep, k_restrict and k_prolong, whose expressions these are.
#include "mg_rb.h"
#include "pdl.cuh"

namespace anel {

// x at interior cell or z ghost `at` of column (i, j) and at the x and y
// ghosts that copy it
__device__ __forceinline__ void rb_images(const RBLevel& L, double* phi, int64_t at, int i, int64_t oy, double x) {
  const int ox = i == 2 ? L.nx : (i == L.nx + 1 ? -L.nx : 0);
  phi[at] = x;
  if (ox) phi[at + ox] = x;
  if (oy) phi[at + oy] = x;
  if (ox && oy) phi[at + ox + oy] = x;
}
// v at interior cell (i, j, k), offset c, and at the ghosts that copy it
__device__ __forceinline__ void rb_put(const RBLevel& L, int64_t c, int i, int64_t oy, int k, double v) {
  rb_images(L, L.phi, c, i, oy, v);
  if (k == 2 && L.n1) rb_images(L, L.phi, c - L.XY, i, oy, v - L.add1);
  if (k == L.nz + 1 && L.nZ) rb_images(L, L.phi, c + L.XY, i, oy, v + L.addZ);
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
// The levels of at most 2 kRBThreads cells of a colour and everything below
// them in one block: their half-sweeps are 1024 to 4 cells long and as
// separate launches cost 6 us each, about 60 of them per cycle.  phi and f
// stay in shared memory.  What bounds the block is latency: a thread holds
// its cells' coefficients and f in registers for the sweeps and the residual
// of a visit, its ghosts as packed words, and the schedule is one loop, so
// the code is fetched once.  An 8192-cell level fits too, but one SM takes
// longer over it than its launches (256x128x128 solve: 39.1 ms with it, 34.3
// without).
constexpr int kRBThreads = 512;
constexpr int kRBGhosts = 4;  // ghosts of a thread held in registers
constexpr unsigned kNoGhost = 0xffffffffu;

static unsigned rb_magic(int d) { return (unsigned)((0x100000000ull + d - 1) / (unsigned)d); }
__device__ __forceinline__ int rb_div(int u, int d, unsigned m) { return d == 1 ? u : (int)__umulhi((unsigned)u, m); }

// a colour's cell: offset (negative: none), coefficients, diagonal, f
struct RBCell {
  int c;
  double a1, a2, a3, a4, a5, a6, d, f;
};

__device__ __forceinline__ RBCell rb_cell(const RBShared& S, int l, const double* sm, const double* src, int color,
                                          int t) {
  const DevLevel<double>& L = S.L[l];
  const int hx = (L.nx + 1) >> 1;
  RBCell q;
  q.c = -1;
  if (t >= hx * L.ny * L.nz) return q;
  const int r = rb_div(t, hx, S.mh[l]), kk = rb_div(r, L.ny, S.my[l]);
  const int k = 2 + kk, j = 2 + r - kk * L.ny, i = 2 + ((color + j + k) & 1) + 2 * (t - r * hx);
  if (i > L.nx + 1) return q;
  q.c = (int)cidx(i, j, k, L.X, L.XY);
  const double *cx = sm + S.coef[l] + i - 1, *cy = sm + S.coef[l] + 2 * L.X + j - 1,
               *cz = sm + S.coef[l] + 2 * L.X + 2 * L.Y + k - 1;
  q.a1 = cx[0];
  q.a2 = cx[L.X];
  q.a3 = cy[0];
  q.a4 = cy[L.Y];
  q.a5 = cz[0];
  q.a6 = cz[L.Z];
  q.d = -(q.a1 + q.a2 + q.a3 + q.a4 + cz[2 * L.Z] + cz[3 * L.Z]);
  q.f = src[q.c];
  return q;
}

// the six neighbours' terms in stencil_update's order
__device__ __forceinline__ double rb_terms(const RBCell& q, const double* phi, int X, int XY) {
  const double* p = phi + q.c;
  double acc = q.a1 * p[-1];
  acc = acc + q.a2 * p[1];
  acc = acc + q.a3 * p[-X];
  acc = acc + q.a4 * p[X];
  acc = acc + q.a5 * p[-XY];
  acc = acc + q.a6 * p[XY];
  return acc;
}

__device__ __forceinline__ void rb_ghost(double* phi, unsigned w) {
  if (w != kNoGhost) phi[w >> 16] = (w & 0xffffu) == 0xffffu ? 0.0 : phi[w & 0xffffu];
}

template <int CD>
__device__ __forceinline__ void rb_prolong(const RBShared& S, int l, double* phi, const DevLevel<double>& C) {
  const DevLevel<double>& F = S.L[l];
  const int n = F.nx * F.ny * F.nz;
  for (int t = threadIdx.x; t < n; t += kRBThreads) {
    const int r = rb_div(t, F.nx, S.mx[l]), kk = rb_div(r, F.ny, S.my[l]);
    const int i = 2 + t - r * F.nx, j = 2 + r - kk * F.ny, k = 2 + kk;
    const int c = (int)cidx(i, j, k, F.X, F.XY);
    phi[c] = phi[c] + prolong_corr<double, CD>(C, i, j, k);
  }
}

__global__ void __launch_bounds__(kRBThreads) k_rb_shared(const __grid_constant__ RBShared S) {
  chain_enter();
  extern __shared__ double sm[];
  const int tid = threadIdx.x, lc = S.lc;
  for (int t = tid; t < S.nblob; t += kRBThreads) sm[t] = S.blob[t];
  const int G = (int)S.L[lc].G;
  for (int t = tid; t < G; t += kRBThreads) {
    sm[S.phi[lc] + t] = 0.0;
    sm[S.phi[lc] + G + t] = S.L[lc].src[t];
  }
  __syncthreads();
  double* const res = sm + S.res;
  // the schedule of mg_cycle.F90:186-325 between the restriction to level
  // lc and the prolongation from it
#pragma unroll 1
  for (int v = 0; v < 2 * lc; ++v) {
    const bool down = v < lc;
    const int l = down ? lc - v : v - lc + 1;
    const DevLevel<double>& L = S.L[l];
    const int X = L.X, XY = (int)L.XY, GL = (int)L.G, iters = down ? S.pre[l] : S.post[l];
    double* const phi = sm + S.phi[l];
    const unsigned* const gw = reinterpret_cast<const unsigned*>(sm + S.ghost[l]);
    const int ng = GL - L.nx * L.ny * L.nz;
    RBCell q[2][2];
    unsigned w[kRBGhosts];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int r = 0; r < 2; ++r) q[h][r] = rb_cell(S, l, sm, phi + GL, h, tid + r * kRBThreads);
#pragma unroll
    for (int g = 0; g < kRBGhosts; ++g) w[g] = tid + g * kRBThreads < ng ? gw[tid + g * kRBThreads] : kNoGhost;
    auto ghosts = [&]() {
      __syncthreads();
#pragma unroll
      for (int g = 0; g < kRBGhosts; ++g) rb_ghost(phi, w[g]);
      for (int g = tid + kRBGhosts * kRBThreads; g < ng; g += kRBThreads) rb_ghost(phi, gw[g]);
      __syncthreads();
    };
#pragma unroll 1
    for (int it = 0; it < iters; ++it)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
          if (q[h][r].c >= 0) phi[q[h][r].c] = (q[h][r].f - rb_terms(q[h][r], phi, X, XY)) / q[h][r].d;
        ghosts();
      }
    if (v < lc - 1) {
      // the children's residuals (fine_resid), then their sums in the order
      // of restrict_value: a nibble per child, bits x, y, z
      const DevLevel<double>& C = S.L[l - 1];
      double* const cphi = sm + S.phi[l - 1];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < 2; ++r)
          if (q[h][r].c >= 0) {
            double acc = rb_terms(q[h][r], phi, X, XY);
            acc = acc + q[h][r].d * phi[q[h][r].c];
            res[q[h][r].c] = q[h][r].f - acc;
          }
      for (int t = tid; t < (int)C.G; t += kRBThreads) cphi[t] = 0.0;
      __syncthreads();
      const int cd = S.cd[l - 1], m = 1 << __popc(cd), n = C.nx * C.ny * C.nz;
      const unsigned seq = cd == 7 ? 0x53716420u : cd == 6 ? 0x6420u : cd == 5 ? 0x5140u : cd == 3 ? 0x3210u : cd << 4;
      const double wgt = 1.0 / m;
      for (int t = tid; t < n; t += kRBThreads) {
        const int r = rb_div(t, C.nx, S.mx[l - 1]), kk = rb_div(r, C.ny, S.my[l - 1]);
        const int i = 2 + t - r * C.nx, j = 2 + r - kk * C.ny, k = 2 + kk;
        const double* p =
            res + cidx(cd & 1 ? 2 * i - 2 : i, cd & 2 ? 2 * j - 2 : j, cd & 4 ? 2 * k - 2 : k, X, XY);
        double s = p[0];
        for (int e = 1; e < m; ++e) {
          const unsigned b = seq >> (4 * e);
          s = s + p[(b & 1) + ((b >> 1) & 1) * X + ((b >> 2) & 1) * XY];
        }
        cphi[C.G + cidx(i, j, k, C.X, C.XY)] = wgt * s;
      }
      __syncthreads();
    } else if (v >= lc && l < lc) {
      DevLevel<double> C = L;
      C.phi = phi;
      double* const fphi = sm + S.phi[l + 1];
      switch (S.cd[l]) {
        case 1: rb_prolong<1>(S, l + 1, fphi, C); break;
        case 2: rb_prolong<2>(S, l + 1, fphi, C); break;
        case 3: rb_prolong<3>(S, l + 1, fphi, C); break;
        case 4: rb_prolong<4>(S, l + 1, fphi, C); break;
        case 5: rb_prolong<5>(S, l + 1, fphi, C); break;
        case 6: rb_prolong<6>(S, l + 1, fphi, C); break;
        default: rb_prolong<7>(S, l + 1, fphi, C); break;
      }
      __syncthreads();
      const unsigned* const fw = reinterpret_cast<const unsigned*>(sm + S.ghost[l + 1]);
      const DevLevel<double>& F = S.L[l + 1];
      const int nf = (int)F.G - F.nx * F.ny * F.nz;
      for (int g = tid; g < nf; g += kRBThreads) rb_ghost(fphi, fw[g]);
      __syncthreads();
    }
  }
  for (int t = tid; t < G; t += kRBThreads) S.L[lc].phi[t] = sm[S.phi[lc] + t];
}

bool rb_shared_fits(RBShared& S, int l) {
  // offsets in doubles: coefficients and ghost words (the blob), the
  // residuals of a visit, phi and f of each level
  int at = 0;
  for (int m = 1; m <= l; ++m) {
    const DevLevel<double>& L = S.L[m];
    const int64_t hx = (L.nx + 1) / 2, ng = L.G - (int64_t)L.nx * L.ny * L.nz;
    if (hx * L.ny * L.nz > 2 * kRBThreads || L.G >= 0xffff || (m < l && S.cd[m] == 0)) return false;
    S.mh[m] = rb_magic((int)hx);
    S.mx[m] = rb_magic(L.nx);
    S.my[m] = rb_magic(L.ny);
    S.coef[m] = at;
    at += 2 * L.X + 2 * L.Y + 4 * L.Z;
    S.ghost[m] = at;
    at += (int)((ng + 1) / 2);
  }
  S.nblob = S.res = at;
  at += (int)S.L[l].G;
  for (int m = 1; m <= l; ++m) {
    S.phi[m] = at;
    at += 2 * (int)S.L[m].G;
  }
  S.bytes = (size_t)at * sizeof(double);
  return S.bytes <= kRBSharedBytes;
}

void rb_shared_prepare() { set_smem_limit_once((const void*)k_rb_shared, (int)kRBSharedBytes); }

void launch_rb_shared(const RBShared& S, cudaStream_t s) {
  launch_chained(k_rb_shared, 1, kRBThreads, S.bytes, s, S);
  count_launch();
}

// ---------------------------------------------------------- stop test
// mg_residual.F90:60-105 over the whole ghosted array, four values per
// thread loaded before the first is stored (ghosts are copied only); the
// maxima of non-negative doubles by their bit patterns, exact in any order,
// one atomic pair per block.  256x128x128: 66 us with one value at a time.
constexpr int kMaxU = 4;
__global__ void __launch_bounds__(256) k_relmax_copy(DevLevel<double> L, const double* phin, double* phio,
                                                     unsigned long long* out) {
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
