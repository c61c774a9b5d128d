// mg_spectral.cu -- the passes of the direct fine-level solve
// (mg_spectral.cuh) and their host side.
#include "mg_spectral.h"

#include <algorithm>
#include <cmath>

#include "fp64_div.h"
#include "mg_launch.h"
#include "pdl.cuh"

namespace anel {

// The end of a norm pass in two halves.  spec_norm_arrive: the block's sums
// to its slot of the member's partials and its arrival; spec_norm_finish:
// the member's last block to arrive adds all partials in slot order (fixed
// for a launch shape, so the sums are deterministic) and sets the member's
// state.  Work between the two hides the arrival's round trip.  corrected:
// the pass follows a correction.
struct SpecNorm {
  double sh[2][8];
  int last;
};

__device__ __forceinline__ void spec_norm_arrive(SpecNorm& N, const SpecDev& D, int b, int slot, int nslots, double rr,
                                                 double ff) {
  for (int o = 16; o > 0; o >>= 1) {
    rr += __shfl_xor_sync(0xffffffffu, rr, o);
    ff += __shfl_xor_sync(0xffffffffu, ff, o);
  }
  if ((threadIdx.x & 31) == 0) {
    N.sh[0][threadIdx.x >> 5] = rr;
    N.sh[1][threadIdx.x >> 5] = ff;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
      rr += N.sh[0][q];
      ff += N.sh[1][q];
    }
    double* part = D.part + (int64_t)b * D.pstride;
    part[2 * slot] = rr;
    part[2 * slot + 1] = ff;
    __threadfence();
    N.last = atomicAdd(D.count + b, 1u) == (unsigned)nslots - 1;
  }
}

__device__ __forceinline__ void spec_norm_finish(SpecNorm& N, const SpecDev& D, int b, int nslots, bool corrected) {
  __syncthreads();
  if (!N.last) return;
  __threadfence();
  const double* part = D.part + (int64_t)b * D.pstride;
  double a = 0.0, c = 0.0;
  for (int q = threadIdx.x; q < nslots; q += blockDim.x) {
    a += __ldcg(part + 2 * q);
    c += __ldcg(part + 2 * q + 1);
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) {
    N.sh[0][threadIdx.x >> 5] = a;
    N.sh[1][threadIdx.x >> 5] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
      a += N.sh[0][q];
      c += N.sh[1][q];
    }
    D.count[b] = 0;
    SpecState s = D.st[b];
    s.ff = c;
    s.rel = c > 0.0 ? sqrt(a / c) : sqrt(a);
    s.iter = corrected ? s.iter + 1 : 0;
    s.conv = s.rel <= D.tol;
    s.act = !s.conv && s.iter < D.maxcy;
    D.st[b] = s;
    D.hst[b] = s;
  }
}

// The passes wait for DRAM with 16 to 24 warps per SM (the transforms' stages
// fill the registers), so each block asks L2 for what the block that will
// take its place reads: the block `resident` further on, in launch order.
// 512x256x512: forward 539 -> 515 us, y 260 -> 219, z 350 -> 365, update
// 411 -> 361, check 326 -> 314 (ncu, cold); a solve with its caller's gauge
// (0.46 ms) 2.79 -> 2.58 ms, 2.60 without the z pass's; twice the distance
// gives nothing.
__device__ __forceinline__ void spec_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ bool spec_next_block(int resident, int& bx, int& by) {
  const int at = blockIdx.x + gridDim.x * blockIdx.y + resident;
  by = at / gridDim.x;
  bx = at - by * gridDim.x;
  return by < (int)gridDim.y;
}
// rows of n elements of esize bytes, `stride` elements apart, by lines
__device__ __forceinline__ void spec_prefetch_rows(const void* p, int rows, int n, int64_t stride, int esize) {
  const int per = 128 / esize, lines = (n + per - 1) / per;
  for (int t = threadIdx.x; t < rows * lines; t += blockDim.x) {
    const int r = t / lines;
    spec_prefetch(static_cast<const char*>(p) + (r * stride + (int64_t)(t - r * lines) * per) * esize);
  }
}

// f - A phi at interior cell offset c of plane k (1-based), whose
// coefficients are (c5, c6, dg)
__device__ __forceinline__ double spec_resid(const SpecDev& D, const double* p, int64_t c, double f,
                                             double c5, double c6, double dg) {
  double acc = D.a1 * (p[c - 1] + p[c + 1]);
  acc += D.a3 * (p[c - D.X] + p[c + D.X]);
  acc += c5 * p[c - D.XY];
  acc += c6 * p[c + D.XY];
  acc += dg * p[c];
  return f - acc;
}

// Residual of row pairs (j, j+1) of plane k, the two rows as the real and
// imaginary part of one transform of length nx, then the rows' own modes.
__global__ void __launch_bounds__(256, 2) k_spec_forward(SpecDev D, int test) {
  chain_enter();
  extern __shared__ double2 xsm[];
  const int b = blockIdx.z;
  if (!test && !D.st[b].act) return;  // the whole block
  const double* phi = D.mt ? D.mt[b].phi : D.phi;
  const double* rhs = D.mt ? D.mt[b].rhs : D.rhs;
  const int n = D.nx, row = spec_row(n), k = 2 + blockIdx.y;
  const int pair0 = blockIdx.x * D.pairs;
  const int nb = min(D.pairs, D.ny / 2 - pair0);
  const double c5 = D.coef[k - 1], c6 = D.coef[D.Z + k - 1];
  const double dg = -(2.0 * D.a1 + 2.0 * D.a3 + D.coef[2 * D.Z + k - 1] + D.coef[3 * D.Z + k - 1]);
  const int64_t base = cidx(2, 2 + 2 * pair0, k, D.X, D.XY);
  int bx, by;
  if (spec_next_block(148 * 2, bx, by)) {
    const int64_t c = cidx(2, 2 + 2 * bx * D.pairs, 2 + by, D.X, D.XY);
    const int rows = min(2 * D.pairs, D.ny - 2 * bx * D.pairs);
    spec_prefetch_rows(phi + c, rows, n, D.X, 8);
    spec_prefetch_rows(rhs + c, rows, n, D.X, 8);
  }
  double rr = 0.0, ff = 0.0;
  auto in = [&](int q, int i) {
    const int64_t c = base + (int64_t)(2 * q) * D.X + i;
    const double f0 = rhs[c], f1 = rhs[c + D.X];
    const double r0 = spec_resid(D, phi, c, f0, c5, c6, dg);
    const double r1 = spec_resid(D, phi, c + D.X, f1, c5, c6, dg);
    rr += r0 * r0 + r1 * r1;
    ff += f0 * f0 + f1 * f1;
    return make_double2(r0, r1);
  };
  auto at = [&](int q, int i) { return q * row + spec_pad(i); };
  auto none = [](int, int, double2) {};
  double2* z = spec_fft<0, true>(D.px, nb, xsm, xsm + D.pairs * row, in, none, at);
  __shared__ SpecNorm norm;
  if (test) spec_norm_arrive(norm, D, b, blockIdx.x + gridDim.x * blockIdx.y, gridDim.x * gridDim.y, rr, ff);
  const int h = D.nxh;
  double2* w = D.work + (int64_t)b * D.nz * D.nu + (int64_t)(k - 2) * D.nu + (int64_t)(2 * pair0) * h;
  for (int it = threadIdx.x; it < nb * h; it += blockDim.x) {
    const int q = spec_div(it, D.dnh), c = it - q * h;
    const double2 u = z[at(q, c)];
    double2 A, B;
    if (c == 0) {
      const double2 v = z[at(q, h)];
      A = make_double2(u.x, v.x);
      B = make_double2(u.y, v.y);
    } else {
      const double2 v = z[at(q, n - c)];
      A = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
      B = make_double2(0.5 * (u.y + v.y), 0.5 * (v.x - u.x));
    }
    w[(int64_t)(2 * q) * h + c] = A;
    w[(int64_t)(2 * q + 1) * h + c] = B;
  }
  if (test) spec_norm_finish(norm, D, b, gridDim.x * gridDim.y, false);
}

// Inverse x transform of row pairs and phi += e.  The inverse transform is
// the forward one with real and imaginary parts exchanged before and after.
__global__ void __launch_bounds__(256, 3) k_spec_update(SpecDev D) {
  chain_enter();
  extern __shared__ double2 xsm[];
  const int b = blockIdx.z;
  if (!D.st[b].act) return;
  double* phi = D.mt ? D.mt[b].phi : D.phi;
  const int n = D.nx, row = spec_row(n), k = 2 + blockIdx.y, h = D.nxh;
  const int pair0 = blockIdx.x * D.pairs;
  const int nb = min(D.pairs, D.ny / 2 - pair0);
  const int64_t base = cidx(2, 2 + 2 * pair0, k, D.X, D.XY);
  const double2* w =
      D.work + (int64_t)b * D.nz * D.nu + (int64_t)(k - 2) * D.nu + (int64_t)(2 * pair0) * h;
  spec_prefetch_rows(phi + base, 2 * nb, n, D.X, 8);
  int bx, by;
  if (spec_next_block(148 * 3, bx, by))
    spec_prefetch_rows(D.work + ((int64_t)b * D.nz + by) * D.nu + (int64_t)(2 * bx * D.pairs) * h,
                       min(2 * D.pairs, D.ny - 2 * bx * D.pairs), h, h, 16);
  auto in = [&](int q, int i) {
    const bool up = i > h;
    const int c = i == h ? 0 : (up ? n - i : i);
    const double2 A = w[(int64_t)(2 * q) * h + c], B = w[(int64_t)(2 * q + 1) * h + c];
    double2 z;  // (re, im)
    if (c == 0) z = i == 0 ? make_double2(A.x, B.x) : make_double2(A.y, B.y);
    else if (up) z = make_double2(A.x + B.y, B.x - A.y);
    else z = make_double2(A.x - B.y, A.y + B.x);
    return make_double2(z.y, z.x);
  };
  auto none = [](int, int, double2) {};
  auto at = [&](int q, int i) { return q * row + spec_pad(i); };
  const double2* z = spec_fft<0, true>(D.px, nb, xsm, xsm + D.pairs * row, in, none, at);
  // a thread's loads of phi before its stores: as a last-stage accessor
  // each phi += e waited for the one before it (833 us at 512x256x512)
  constexpr int U = 4;
  const int total = nb * n;
  for (int it = threadIdx.x; it < total; it += U * blockDim.x) {
    double p0[U], p1[U];
    int64_t c[U];
    int o[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = it + u * blockDim.x;
      if (t >= total) break;
      const int q = spec_div(t, D.dnx), i = t - q * n;
      c[u] = base + (int64_t)(2 * q) * D.X + i;
      o[u] = at(q, i);
      p0[u] = phi[c[u]];
      p1[u] = phi[c[u] + D.X];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (it + u * (int)blockDim.x >= total) break;
      const double2 v = z[o[u]];
      phi[c[u]] = p0[u] + D.scale * v.y;
      phi[c[u] + D.X] = p1[u] + D.scale * v.x;
    }
  }
}

// y transform of W columns of a plane, in place.
template <bool kInv, int W>
__global__ void __launch_bounds__(256, 3) k_spec_y(SpecDev D) {
  chain_enter();
  extern __shared__ double2 xsm[];
  const int b = blockIdx.z;
  if (!D.st[b].act) return;
  const int n = D.ny, h = D.nxh, hy = n / 2;
  const int c0 = blockIdx.x * W;
  const int nb = min(W, h - c0);
  double2* w = D.work + (int64_t)b * D.nz * D.nu + (int64_t)blockIdx.y * D.nu + c0;
  double2* col = xsm + 2 * W * n;  // column 0 of the forward transform
  int bx, by;
  if (spec_next_block(148 * 3, bx, by))
    spec_prefetch_rows(D.work + ((int64_t)b * D.nz + by) * D.nu + bx * W, n, min(W, h - bx * W), h, 16);
  const bool zero = c0 == 0;
  auto in = [&](int q, int i) {
    if (kInv) {
      double2 z;
      if (zero && q == 0 && i != 0 && i != hy) {
        const int l = i < hy ? i : n - i;
        const double2 e = w[(int64_t)l * h], m = w[(int64_t)(n - l) * h];
        z = i < hy ? make_double2(e.x - m.y, e.y + m.x) : make_double2(e.x + m.y, m.x - e.y);
      } else {
        z = w[(int64_t)i * h + q];
      }
      return make_double2(z.y, z.x);
    }
    return w[(int64_t)i * h + q];
  };
  auto out = [&](int q, int i, double2 v) {
    if (kInv) v = make_double2(v.y, v.x);
    if (!kInv && zero && q == 0) col[i] = v;
    else w[(int64_t)i * h + q] = v;
  };
  auto at = [&](int q, int i) { return i * W + q; };
  spec_fft<W, false>(D.py, nb, xsm, xsm + W * n, in, out, at);
  if (!kInv && zero) {
    for (int l = threadIdx.x; l <= hy; l += blockDim.x) {
      const double2 u = col[l];
      if (l == 0 || l == hy) {
        w[(int64_t)l * h] = u;
      } else {
        const double2 v = col[n - l];
        w[(int64_t)l * h] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
        w[(int64_t)(n - l) * h] = make_double2(0.5 * (u.y + v.y), 0.5 * (v.x - u.x));
      }
    }
  }
}

// 1 / x for a normal x from the hardware's approximation (its top 20
// mantissa bits).  A division branches to its special cases, which a chain of
// them waits for.
__device__ __forceinline__ double spec_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return rcp_newton(x, y);
}

// The z-systems of eight modes at a time.  Thread (mode w, segment g) holds
// M consecutive rows in registers: the first M-1 are eliminated against the
// segment's neighbours (their values are v + L x(last row of the previous
// segment) - cp x(next row)), the last rows of the S segments are solved
// for by cyclic reduction through shared memory, and the inner rows follow
// by substitution.  The reciprocals of the eliminated diagonal are kept, L
// is formed again.  A tile's rows are read and written once, 128 bytes at a
// time.  The last tile holds the four real systems of column 0's rows 0 and
// ny/2: one component each.
template <int M>
__global__ void __launch_bounds__(512) k_spec_z(SpecDev D, int ntiles) {
  chain_enter();
  extern __shared__ double zsm[];
  const int b = blockIdx.y;
  if (!D.st[b].act) return;
  const int S = D.S, w = threadIdx.x & 7, g = threadIdx.x >> 3;
  double* t_sub = zsm;
  double* t_dia = t_sub + M * S;
  double* t_sup = t_dia + M * S;
  double* x0 = t_sup + M * S;          // exchange buffers: S*8 x 4 doubles each
  double* x1 = x0 + 32 * S;
  for (int q = threadIdx.x; q < 3 * M * S; q += blockDim.x) zsm[q] = D.zt[q];
  __syncthreads();
  double2* work = D.work + (int64_t)b * D.nz * D.nu;
  const int r0 = g * M;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const bool special = tile == ntiles - 1;
    int64_t u;
    double sh;
    bool live;
    int comp = 0;  // special: 0 real, 1 imaginary part
    bool pin = false;
    if (special) {
      const int l = (w & 2) ? D.ny / 2 : 0;
      comp = w & 1;
      u = (int64_t)l * D.nxh;
      sh = D.lx[comp ? D.nxh : 0] + D.ly[l];
      live = w < 4;
      pin = w == 0 && D.singular;
    } else {
      u = (int64_t)tile * 8 + w;
      live = u < D.nu;
      const int l = live ? (int)(u / D.nxh) : 0, c = live ? (int)(u - (int64_t)l * D.nxh) : 1;
      sh = c == 0 ? D.l0[l] : D.lx[c] + D.ly[l];
      if (c == 0 && (l == 0 || l == D.ny / 2)) live = false;
    }
    if (tile + (int)gridDim.x < ntiles - 1)
      for (int q = w; q < M; q += 8)
        if (r0 + q < D.nz) spec_prefetch(work + (int64_t)(r0 + q) * D.nu + (int64_t)(tile + gridDim.x) * 8);
    double2 v[M];
#pragma unroll
    for (int q = 0; q < M; ++q)
      v[q] = (live && r0 + q < D.nz) ? __ldcg(work + (int64_t)(r0 + q) * D.nu + u) : make_double2(0.0, 0.0);
    if (special) {
#pragma unroll
      for (int q = 0; q < M; ++q) {
        if (comp) v[q].x = v[q].y;
        v[q].y = 0.0;
        if (pin && r0 + q == D.nz - 1) v[q].x = 0.0;
      }
    }
    // row q of this segment; the pinned row is x = 0
    auto sub = [&](int q) { return pin && r0 + q == D.nz - 1 ? 0.0 : t_sub[q * S + g]; };
    auto dia = [&](int q) { return pin && r0 + q == D.nz - 1 ? 1.0 : t_dia[q * S + g] - (r0 + q < D.nz ? sh : 0.0); };
    double inv[M - 1];
    inv[0] = spec_rcp(dia(0));
    v[0].x *= inv[0];
    v[0].y *= inv[0];
    double L = -sub(0) * inv[0];
    // first inner row's value, Y + L0 x(previous) + P x(this segment's last)
    double P = 1.0, L0 = L;
    double2 Y = v[0];
#pragma unroll
    for (int q = 1; q < M - 1; ++q) {
      const double cp = t_sup[(q - 1) * S + g] * inv[q - 1], sb = sub(q);
      inv[q] = spec_rcp(dia(q) - sb * cp);
      v[q].x = (v[q].x - sb * v[q - 1].x) * inv[q];
      v[q].y = (v[q].y - sb * v[q - 1].y) * inv[q];
      L = -sb * L * inv[q];
      P = -P * cp;
      Y.x += P * v[q].x;
      Y.y += P * v[q].y;
      L0 += P * L;
    }
    const double cl = t_sup[(M - 2) * S + g] * inv[M - 2];
    P = -P * cl;
    double4* e0 = reinterpret_cast<double4*>(x0);
    double4* e1 = reinterpret_cast<double4*>(x1);
    __syncthreads();  // the previous tile's reads are done
    e0[threadIdx.x] = make_double4(Y.x, Y.y, L0, P);
    __syncthreads();
    double A, C;
    double2 F;
    {
      const double4 nx = g + 1 < S ? e0[threadIdx.x + 8] : make_double4(0.0, 0.0, 0.0, 0.0);
      const double sb = sub(M - 1), sp = t_sup[(M - 1) * S + g];
      const double spn = pin && r0 + M - 1 == D.nz - 1 ? 0.0 : sp;
      const double ib = spec_rcp(dia(M - 1) - sb * cl + spn * nx.z);
      A = sb * L * ib;
      C = spn * nx.w * ib;
      F.x = (v[M - 1].x - sb * v[M - 2].x - spn * nx.x) * ib;
      F.y = (v[M - 1].y - sb * v[M - 2].y - spn * nx.y) * ib;
    }
    for (int d = 1; d < S; d *= 2) {
      double4* e = (e0 == reinterpret_cast<double4*>(x0)) ? e1 : reinterpret_cast<double4*>(x0);
      e[threadIdx.x] = make_double4(A, C, F.x, F.y);
      __syncthreads();
      const double4 z4 = make_double4(0.0, 0.0, 0.0, 0.0);
      const double4 um = g >= d ? e[threadIdx.x - 8 * d] : z4;
      const double4 up = g + d < S ? e[threadIdx.x + 8 * d] : z4;
      const double kk = spec_rcp(1.0 - A * um.y - C * up.x);
      F.x = (F.x - A * um.z - C * up.z) * kk;
      F.y = (F.y - A * um.w - C * up.w) * kk;
      A = -A * um.x * kk;
      C = -C * up.y * kk;
      e0 = e;
    }
    double4* e = (e0 == reinterpret_cast<double4*>(x0)) ? e1 : reinterpret_cast<double4*>(x0);
    e[threadIdx.x] = make_double4(F.x, F.y, 0.0, 0.0);
    __syncthreads();
    const double4 xp = g > 0 ? e[threadIdx.x - 8] : make_double4(0.0, 0.0, 0.0, 0.0);
    L = 1.0;
#pragma unroll
    for (int q = 0; q < M - 1; ++q) {
      L = -sub(q) * L * inv[q];
      v[q].x += L * xp.x;
      v[q].y += L * xp.y;
    }
    v[M - 1] = F;
#pragma unroll
    for (int q = M - 2; q >= 0; --q) {
      const double cp = t_sup[q * S + g] * inv[q];
      v[q].x -= cp * v[q + 1].x;
      v[q].y -= cp * v[q + 1].y;
    }
    if (special) {
      // mode (0, 0) is fixed up to its null vector: return it with zero sum,
      // so that corrections leave the mean of the solution alone
      if (D.singular) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < M; ++q)
          if (w == 0 && r0 + q < D.nz) s += v[q].x;
        double* ms = reinterpret_cast<double*>(e == reinterpret_cast<double4*>(x0) ? x1 : x0);
        __syncthreads();
        if (w == 0) ms[g] = s;
        __syncthreads();
        if (w == 0) {
          double m = 0.0;
          for (int q = 0; q < S; ++q) m += ms[q];
#pragma unroll
          for (int q = 0; q < M; ++q) v[q].x -= m * D.zt[3 * M * S + q * S + g];
        }
      }
      double* wd = reinterpret_cast<double*>(work);
#pragma unroll
      for (int q = 0; q < M; ++q)
        if (live && r0 + q < D.nz) wd[2 * ((int64_t)(r0 + q) * D.nu + u) + comp] = v[q].x;
    } else {
#pragma unroll
      for (int q = 0; q < M; ++q)
        if (live && r0 + q < D.nz) work[(int64_t)(r0 + q) * D.nu + u] = v[q];
    }
  }
}

// |f - A phi|: a block owns 32 x 8 columns (a row's y neighbours come from
// L1 then) and marches `per` planes, the z neighbours kept in registers;
// grid (ceil(nx/32), ceil(ny/8), ceil(nz/per) * members).  per = 32, fewer
// where that leaves less than two blocks per SM: a block ends in two sums
// and an arrival, as long as about four planes (337 us with 8 planes and
// flat columns at 512x256x512).
constexpr int kCheckK = 4;
__global__ void __launch_bounds__(256) k_spec_check(SpecDev D, int per, int nzb) {
  chain_enter();
  const int b = blockIdx.z / nzb;
  if (!D.st[b].act) return;
  const double* phi = D.mt ? D.mt[b].phi : D.phi;
  const double* rhs = D.mt ? D.mt[b].rhs : D.rhs;
  const int i = 2 + blockIdx.x * 32 + (threadIdx.x & 31), j = 2 + blockIdx.y * 8 + (threadIdx.x >> 5);
  const int zb = blockIdx.z - b * nzb;
  const int k0 = 2 + zb * per, kend = min(k0 + per, D.nz + 2);  // exclusive
  double rr = 0.0, ff = 0.0;
  if (i <= D.nx + 1 && j <= D.ny + 1) {
    int64_t c = cidx(i, j, k0, D.X, D.XY);
    double pm = phi[c - D.XY], pc = phi[c];
    const double a0 = 2.0 * D.a1 + 2.0 * D.a3;
    auto cell = [&](int k, double pp, double f, double pw, double pe, double ps, double pn) {
      const double dg = -(a0 + D.coef[2 * D.Z + k - 1] + D.coef[3 * D.Z + k - 1]);
      double acc = D.a1 * (pw + pe);
      acc += D.a3 * (ps + pn);
      acc += D.coef[k - 1] * pm;
      acc += D.coef[D.Z + k - 1] * pp;
      acc += dg * pc;
      const double r = f - acc;
      rr += r * r;
      ff += f * f;
      pm = pc;
      pc = pp;
    };
    int k = k0;
    const int lane = threadIdx.x & 31;
    const bool ahead = lane == 0 || lane == 16 || lane == 31;
    for (; k + kCheckK <= kend; k += kCheckK) {
      if (ahead) {
#pragma unroll
        for (int q = 0; q < kCheckK; ++q)
          if (k + 2 * kCheckK + q < kend) {
            spec_prefetch(rhs + c + (2 * kCheckK + q) * D.XY);
            spec_prefetch(phi + c + (2 * kCheckK + q + 1) * D.XY);
          }
      }
      double v[kCheckK][6];
#pragma unroll
      for (int q = 0; q < kCheckK; ++q) {
        const int64_t o = c + q * D.XY;
        v[q][0] = phi[o + D.XY];
        v[q][1] = rhs[o];
        v[q][2] = phi[o - 1];
        v[q][3] = phi[o + 1];
        v[q][4] = phi[o - D.X];
        v[q][5] = phi[o + D.X];
      }
#pragma unroll
      for (int q = 0; q < kCheckK; ++q) cell(k + q, v[q][0], v[q][1], v[q][2], v[q][3], v[q][4], v[q][5]);
      c += kCheckK * D.XY;
    }
    for (; k < kend; ++k, c += D.XY)
      cell(k, phi[c + D.XY], rhs[c], phi[c - 1], phi[c + 1], phi[c - D.X], phi[c + D.X]);
  }
  __shared__ SpecNorm norm;
  const int nslots = gridDim.x * gridDim.y * nzb;
  spec_norm_arrive(norm, D, b, blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * zb), nslots, rr, ff);
  spec_norm_finish(norm, D, b, nslots, true);
}

// ------------------------------------------------------------------ host
static bool plan_radices(int n, std::vector<int>& rad) {
  rad.clear();
  if (n < 2 || n % 2 || n > kSpecMaxN) return false;
  int two = 0;
  while (n % 2 == 0) {
    n /= 2;
    ++two;
  }
  // powers of two as radix 8, with one or two radix-4 stages for the rest
  while (two > 4 || two == 3) {
    rad.push_back(8);
    two -= 3;
  }
  if (two == 4) {
    rad.push_back(4);
    rad.push_back(4);
  } else if (two == 2) {
    rad.push_back(4);
  } else if (two == 1) {
    rad.push_back(2);
  }
  for (int p = 3; n > 1; p += 2)
    while (n % p == 0) {
      if (p > kSpecMaxPrime) return false;
      rad.push_back(p);
      n /= p;
    }
  return (int)rad.size() <= kSpecMaxStages;
}

static void segment(int nz, int* S, int* M) {
  *S = nz <= 512 ? 32 : 64;
  for (int m : {2, 3, 4, 6, 8, 12, 16}) {
    *M = m;
    if (*S * m >= nz) return;
  }
}

bool spec_supported(int nx, int ny, int nz) {
  std::vector<int> r;
  return plan_radices(nx, r) && plan_radices(ny, r) && nz >= 2 && nz <= kSpecMaxNz;
}

constexpr int kFillBlocks = 2 * 148;
static int check_cols(const SpecDev& D) { return ((D.nx + 31) / 32) * ((D.ny + 7) / 8); }
static int check_planes(const SpecDev& D) {
  int per = 32;
  while (per > 2 && check_cols(D) * ((D.nz + per - 1) / per) < kFillBlocks) per /= 2;
  return per;
}
static int check_zblocks(const SpecDev& D) { return (D.nz + check_planes(D) - 1) / check_planes(D); }
static size_t x_smem(const SpecDev& D) { return (size_t)2 * D.pairs * spec_row(D.nx) * sizeof(double2); }
// columns per block of the y passes: eight fill a 128-byte line; fewer
// where the two buffers of a longer transform would not fit
static int y_cols(const SpecDev& D) { return D.ny <= 768 ? 8 : (D.ny <= 1536 ? 4 : 2); }
static size_t y_smem(const SpecDev& D) { return (size_t)(2 * y_cols(D) + 1) * D.ny * sizeof(double2); }
static size_t z_smem(const SpecDev& D) { return ((size_t)3 * D.M * D.S + 64 * (size_t)D.S) * sizeof(double); }

template <class F>
static void y_kernel(bool inverse, int cols, F f) {
  switch (cols) {
    case 8: inverse ? f(k_spec_y<true, 8>) : f(k_spec_y<false, 8>); break;
    case 4: inverse ? f(k_spec_y<true, 4>) : f(k_spec_y<false, 4>); break;
    default: inverse ? f(k_spec_y<true, 2>) : f(k_spec_y<false, 2>); break;
  }
}

template <class F>
static void z_kernel(int M, F f) {
  switch (M) {
    case 2: f(k_spec_z<2>); break;
    case 3: f(k_spec_z<3>); break;
    case 4: f(k_spec_z<4>); break;
    case 6: f(k_spec_z<6>); break;
    case 8: f(k_spec_z<8>); break;
    case 12: f(k_spec_z<12>); break;
    default: f(k_spec_z<16>); break;
  }
}

int spec_build(SpecHost& H, SpecState* h_one, int nx, int ny, int nz, double a1, double a3, const double* cz5, const double* cz6,
               const double* dz5, const double* dz6, int z1, int zZ, const double* coef) {
  SpecDev& D = H.d;
  H.ok = false;
  if (!spec_supported(nx, ny, nz)) return ANEL_OK;
  D.nx = nx;
  D.ny = ny;
  D.nz = nz;
  D.nxh = nx / 2;
  D.X = nx + 2;
  D.XY = (int64_t)(nx + 2) * (ny + 2);
  D.Z = nz + 2;
  D.nu = (int64_t)D.nxh * ny;
  D.dnx = spec_div_magic(nx);
  D.dnh = spec_div_magic(D.nxh);
  D.a1 = a1;
  D.a3 = a3;
  D.scale = 1.0 / ((double)nx * ny);
  D.coef = coef;
  segment(nz, &D.S, &D.M);
  // row pairs per block: about 256 butterflies of radix 8, fewer (down to a
  // warp's) where that leaves the GPU with less than two blocks per SM
  D.pairs = std::max(1, std::min(ny / 2, 2048 / nx));
  while (D.pairs * nx > 256 && D.pairs > 1 && (int64_t)nz * ((ny / 2 + D.pairs - 1) / D.pairs) < kFillBlocks)
    D.pairs = (D.pairs + 1) / 2;
  const double pi = 3.14159265358979323846;
  // tables: twiddles of x and y, eigenvalues, z coefficients
  std::vector<double> tab;
  auto twiddles = [&](int n) {
    const size_t at = tab.size();
    for (int t = 0; t < n; ++t) {
      tab.push_back(std::cos(2.0 * pi * t / n));
      tab.push_back(-std::sin(2.0 * pi * t / n));
    }
    return at;
  };
  const size_t otx = twiddles(nx), oty = twiddles(ny);
  auto eig = [&](double a, int p, int n) {
    const double s = std::sin(pi * p / n);
    return 4.0 * a * s * s;
  };
  const size_t olx = tab.size();
  for (int p = 0; p <= D.nxh; ++p) tab.push_back(eig(a1, p, nx));
  const size_t oly = tab.size();
  for (int q = 0; q < ny; ++q) tab.push_back(eig(a3, q, ny));
  const size_t ol0 = tab.size();
  for (int l = 0; l < ny; ++l) tab.push_back(l <= ny / 2 ? eig(a3, l, ny) : eig(a1, D.nxh, nx) + eig(a3, l, ny));
  const size_t ozt = tab.size();
  std::vector<double> sub(nz), dia(nz), sup(nz);
  for (int r = 0; r < nz; ++r) {
    sub[r] = cz5[r + 1];
    sup[r] = cz6[r + 1];
    dia[r] = -(dz5[r + 1] + dz6[r + 1]);
  }
  if (z1 == 1) dia[0] += sub[0];
  if (zZ == 1) dia[nz - 1] += sup[nz - 1];
  sub[0] = sup[nz - 1] = 0.0;
  // mode (0, 0) is singular when its last pivot vanishes (zero flux through
  // both walls); the null vector is r(z)
  double piv = dia[0];
  for (int r = 1; r < nz; ++r) piv = dia[r] - sub[r] * sup[r - 1] / piv;
  D.singular = std::fabs(piv) <= 1e-10 * std::fabs(dia[nz - 1]);
  std::vector<double> nul(nz, 1.0);
  double nsum = 0.0;
  for (int r = 0; r + 1 < nz && D.singular; ++r)
    nul[r + 1] = -(dia[r] * nul[r] + (r > 0 ? sub[r] * nul[r - 1] : 0.0)) / sup[r];
  for (double v : nul) nsum += v;
  for (double& v : nul) v /= nsum;
  for (int which = 0; which < 4; ++which)
    for (int q = 0; q < D.M; ++q)
      for (int g = 0; g < D.S; ++g) {
        const int r = g * D.M + q;
        const double pad = which == 1 ? 1.0 : 0.0;  // rows past the end: x = 0
        tab.push_back(r < nz ? (which == 0 ? sub[r] : which == 1 ? dia[r] : which == 2 ? sup[r] : nul[r]) : pad);
      }
  if (!H.d_tab) ANEL_CUDA_TRY(cudaMalloc(&H.d_tab, tab.size() * sizeof(double)));
  ANEL_CUDA_TRY(cudaMemcpy(H.d_tab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice));
  auto plan = [&](int n, size_t off) {
    SpecPlan P{};
    P.n = n;
    std::vector<int> rad;
    plan_radices(n, rad);
    P.nst = (int)rad.size();
    int s = 1;
    for (int t = 0; t < P.nst; ++t) {
      P.rad[t] = rad[t];
      P.str[t] = s;
      P.dn[t] = spec_div_magic(n / rad[t]);
      P.ds[t] = spec_div_magic(s);
      s *= rad[t];
    }
    P.tw = reinterpret_cast<const double2*>(H.d_tab + off);
    return P;
  };
  D.px = plan(nx, otx);
  D.py = plan(ny, oty);
  D.lx = H.d_tab + olx;
  D.ly = H.d_tab + oly;
  D.l0 = H.d_tab + ol0;
  D.zt = H.d_tab + ozt;
  // launch attributes, outside any capture
  set_smem_limit_once((const void*)k_spec_forward, (int)x_smem(D));
  set_smem_limit_once((const void*)k_spec_update, (int)x_smem(D));
  for (bool inv : {false, true})
    y_kernel(inv, y_cols(D), [&](auto* k) { set_smem_limit_once((const void*)k, (int)y_smem(D)); });
  z_kernel(D.M, [&](auto* k) { set_smem_limit_once((const void*)k, (int)z_smem(D)); });
  ANEL_CUDA_TRY(cudaGetLastError());
  H.h_one = h_one;
  const int st = spec_reserve(H, 1);
  if (st != ANEL_OK) return st;
  H.ok = true;
  return ANEL_OK;
}

int spec_reserve(SpecHost& H, int n) {
  SpecDev& D = H.d;
  if (n <= H.cap) return ANEL_OK;
  const int64_t fwd = (int64_t)((D.ny / 2 + D.pairs - 1) / D.pairs) * D.nz;
  const int64_t pstride = 2 * std::max<int64_t>(fwd, (int64_t)check_cols(D) * check_zblocks(D));
  const size_t st = (size_t)n * sizeof(SpecState), cnt = ((size_t)n * sizeof(unsigned) + 15) / 16 * 16;
  // the new buffers first: where one of them cannot be had, the old ones
  // stay and solves within their room go on
  double* buf = nullptr;
  SpecState* host = H.h_one;
  cudaError_t e = cudaMalloc(&buf, st + cnt + (size_t)n * pstride * sizeof(double));
  if (e == cudaSuccess) e = cudaMemset(buf, 0, st + cnt);
  // the kernels count on counters that start at zero
  if (e == cudaSuccess) e = setup_wait();
  if (e == cudaSuccess && n > 1) e = cudaHostAlloc(&host, (size_t)n * sizeof(SpecState), cudaHostAllocMapped);
  if (e != cudaSuccess) {
    cudaFree(buf);
    cudaGetLastError();
    set_error("direct solve: no memory for %d members: %s", n, cudaGetErrorString(e));
    return ANEL_ERR_CUDA;
  }
  cudaFree(H.d_buf);
  if (H.h_st && H.h_st != H.h_one) cudaFreeHost(H.h_st);
  H.d_buf = buf;
  H.h_st = host;
  H.cap = n;
  char* p = reinterpret_cast<char*>(buf);
  D.pstride = pstride;
  D.hst = host;
  D.st = reinterpret_cast<SpecState*>(p);
  D.count = reinterpret_cast<unsigned*>(p + st);
  D.part = reinterpret_cast<double*>(p + st + cnt);
  return ANEL_OK;
}

void spec_free(SpecHost& H) {
  cudaFree(H.d_tab);
  cudaFree(H.d_buf);
  if (H.h_st && H.h_st != H.h_one) cudaFreeHost(H.h_st);
  H = SpecHost{};
}

static int x_threads(const SpecDev& D) {
  const int t = (D.pairs * D.nx / 8 + 31) / 32 * 32;
  return std::max(32, std::min(256, t));
}
static int y_threads(const SpecDev& D) {
  return std::max(32, std::min(256, (y_cols(D) * D.ny / 8 + 31) / 32 * 32));
}

void launch_spec_forward(const SpecDev& D, int nm, bool test, cudaStream_t s) {
  const dim3 g((unsigned)((D.ny / 2 + D.pairs - 1) / D.pairs), (unsigned)D.nz, (unsigned)nm);
  launch_chained(k_spec_forward, g, x_threads(D), x_smem(D), s, D, test ? 1 : 0);
  count_launch();
}

void launch_spec_y(const SpecDev& D, int nm, bool inverse, cudaStream_t s) {
  const int cols = y_cols(D);
  const dim3 g((unsigned)((D.nxh + cols - 1) / cols), (unsigned)D.nz, (unsigned)nm);
  y_kernel(inverse, cols, [&](auto* k) { launch_chained(k, g, y_threads(D), y_smem(D), s, D); });
  count_launch();
}

void launch_spec_z(const SpecDev& D, int nm, cudaStream_t s) {
  const int ntiles = (int)((D.nu + 7) / 8) + 1;
  z_kernel(D.M, [&](auto* k) {
    launch_chained(k, dim3((unsigned)std::min(ntiles, 148 * 2), (unsigned)nm), 8 * D.S, z_smem(D), s, D, ntiles);
  });
  count_launch();
}

void launch_spec_update(const SpecDev& D, int nm, cudaStream_t s) {
  const dim3 g((unsigned)((D.ny / 2 + D.pairs - 1) / D.pairs), (unsigned)D.nz, (unsigned)nm);
  launch_chained(k_spec_update, g, x_threads(D), x_smem(D), s, D);
  count_launch();
}

void launch_spec_check(const SpecDev& D, int nm, cudaStream_t s) {
  // member and z-block share blockIdx.z, 65535 at most: more members take
  // more launches (two z-planes per block of a 16x16x64 member: 2047 fit)
  const int nzb = check_zblocks(D), most = 65535 / nzb;
  for (int b = 0; b < nm; b += most) {
    const int m = std::min(most, nm - b);
    SpecDev P = D;
    if (P.mt) P.mt += b;
    P.st += b;
    P.hst += b;
    P.count += b;
    P.part += b * P.pstride;
    const dim3 g((unsigned)((D.nx + 31) / 32), (unsigned)((D.ny + 7) / 8), (unsigned)(nzb * m));
    launch_chained(k_spec_check, g, 256, 0, s, P, check_planes(D), nzb);
    count_launch();
  }
}

}  // namespace anel
