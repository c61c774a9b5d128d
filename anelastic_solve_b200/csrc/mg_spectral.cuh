// mg_spectral.cuh -- FP64 direct solve of the fine level: Fourier in the
// periodic x and y, one tridiagonal z-system per mode.
//
// With x and y periodic and x/y-uniform symmetric coefficients the fine
// operator is diagonal in the Fourier modes of x and y: mode (p, q) leaves
//   cz5(k) e(k-1) + (-(dz5(k) + dz6(k)) - s(p, q)) e(k) + cz6(k) e(k+1) = r(k),
//   s(p, q) = 4 a1 sin^2(pi p / nx) + 4 a3 sin^2(pi q / ny),
// with the z-ghost rule folded into the end rows.  So one step of the
// mixed-precision solve's defect correction, phi += A^-1 (f - A phi), is
// six passes over memory: residual and x transform, y transform, z-systems,
// inverse y transform, inverse x transform and update, and the residual norm
// of the result.  All of it is FP64.
//
// Spectral array of one member: [k][j][c] complex, nxh = nx/2 per row, in
// the space of nx*ny*nz doubles.  nx is even (the level rule), so a real
// row has the modes 0..nx/2; the two real ones share column 0 (real part
// mode 0, imaginary part mode nx/2).  After the y transform column 0 is
// taken apart: rows l < ny/2 hold mode (0, l), row ny-l holds mode
// (nx/2, l), and rows 0 and ny/2 hold the two real values of both.
#pragma once

#include "mg_col.cuh"

namespace anel {

// transform lengths: even, prime factors up to kSpecMaxPrime, at most
// kSpecMaxN points; z-systems of up to kSpecMaxNz rows
constexpr int kSpecMaxPrime = 31;
constexpr int kSpecMaxN = 2048;
constexpr int kSpecMaxNz = 1024;
constexpr int kSpecMaxStages = 12;

// A mixed-radix Stockham transform: stage t of radix rad[t] has stride
// s = rad[0]*...*rad[t-1]; dn / ds are the reciprocals of n/rad and s for
// the index splits (spec_div).
struct SpecPlan {
  int n, nst;
  int rad[kSpecMaxStages], str[kSpecMaxStages];
  unsigned dn[kSpecMaxStages], ds[kSpecMaxStages];
  const double2* tw;  // exp(-2 pi i t / n), t < n
};

// convergence state of one member, mirrored in mapped host memory
struct SpecState {
  double rel;  // |r| / |f| (|r| when f is zero)
  double ff;   // |f|^2
  int iter;    // direct corrections done
  int conv;    // rel <= tol
  int act;     // another correction is wanted
  int pad;
};

struct SpecDev {
  int nx, ny, nz, nxh;
  int X;
  int64_t XY;
  int64_t nu;          // nxh * ny complex values of a plane
  unsigned dnx, dnh;   // reciprocals of nx and nxh (spec_div)
  double a1, a3;       // x and y coefficients
  double scale;        // 1 / (nx * ny)
  const double* coef;  // the fine level's cz5[Z] cz6[Z] dz5[Z] dz6[Z]
  int Z;
  SpecPlan px, py;
  const double* lx;    // [nxh + 1] 4 a1 sin^2
  const double* ly;    // [ny] 4 a3 sin^2
  const double* l0;    // [ny] shift of column 0 (see above)
  const double* zt;    // z tables: sub, dia, sup, null vector (sum 1), each [M][S]
  int S, M;            // segments of a z-system and rows per segment
  int singular;        // mode (0, 0) has a null vector
  int pairs;           // row pairs per block of the x passes
  // members: pointers from mt, or phi / rhs of the only one
  const MemberIO* mt;
  double* phi;
  const double* rhs;
  double2* work;       // member b at b * nz * nu
  SpecState* st;       // device states
  SpecState* hst;      // their mirrors (mapped host memory)
  double* part;        // partial sums, member b at b * pstride
  int64_t pstride;
  unsigned* count;     // arrival counters, one per member
  double tol;
  int maxcy;
};

__host__ __device__ __forceinline__ unsigned spec_div_magic(int d) {
  return d == 1 ? 0u : (unsigned)((0x100000000ull + (unsigned)d - 1) / (unsigned)d);
}
// u / d for u < 2^16, d < 2^16 (magic 0: d = 1)
__device__ __forceinline__ int spec_div(int u, unsigned magic) {
  return magic ? (int)__umulhi((unsigned)u, magic) : u;
}

__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }  // -i a

// a <- sum_r a[r] exp(-2 pi i r t / R) for t = 0..R-1
template <int R>
__device__ __forceinline__ void dft(double2 (&a)[R]);
template <>
__device__ __forceinline__ void dft<2>(double2 (&a)[2]) {
  const double2 t = a[0];
  a[0] = t + a[1];
  a[1] = t - a[1];
}
template <>
__device__ __forceinline__ void dft<3>(double2 (&a)[3]) {
  constexpr double S3 = 0.86602540378443864676;  // sin(2 pi / 3)
  const double2 t = a[1] + a[2], d = mul_mi(a[1] - a[2]);
  const double2 m = make_double2(a[0].x - 0.5 * t.x, a[0].y - 0.5 * t.y);
  a[0] = a[0] + t;
  a[1] = make_double2(m.x + S3 * d.x, m.y + S3 * d.y);
  a[2] = make_double2(m.x - S3 * d.x, m.y - S3 * d.y);
}
__device__ __forceinline__ void dft4(double2& a0, double2& a1, double2& a2, double2& a3) {
  const double2 t0 = a0 + a2, t1 = a0 - a2, t2 = a1 + a3, t3 = mul_mi(a1 - a3);
  a0 = t0 + t2;
  a1 = t1 + t3;
  a2 = t0 - t2;
  a3 = t1 - t3;
}
template <>
__device__ __forceinline__ void dft<4>(double2 (&a)[4]) {
  dft4(a[0], a[1], a[2], a[3]);
}
template <>
__device__ __forceinline__ void dft<5>(double2 (&a)[5]) {
  constexpr double C1 = 0.30901699437494742410, C2 = -0.80901699437494742410;  // cos(2 pi m / 5)
  constexpr double S1 = 0.95105651629515357212, S2 = 0.58778525229247312917;   // sin(2 pi m / 5)
  const double2 p1 = a[1] + a[4], p2 = a[2] + a[3], d1 = mul_mi(a[1] - a[4]), d2 = mul_mi(a[2] - a[3]);
  const double2 m1 = make_double2(a[0].x + C1 * p1.x + C2 * p2.x, a[0].y + C1 * p1.y + C2 * p2.y);
  const double2 m2 = make_double2(a[0].x + C2 * p1.x + C1 * p2.x, a[0].y + C2 * p1.y + C1 * p2.y);
  const double2 s1 = make_double2(S1 * d1.x + S2 * d2.x, S1 * d1.y + S2 * d2.y);
  const double2 s2 = make_double2(S2 * d1.x - S1 * d2.x, S2 * d1.y - S1 * d2.y);
  a[0] = a[0] + p1 + p2;
  a[1] = m1 + s1;
  a[4] = m1 - s1;
  a[2] = m2 + s2;
  a[3] = m2 - s2;
}
template <>
__device__ __forceinline__ void dft<8>(double2 (&a)[8]) {
  constexpr double H = 0.70710678118654752440;  // sqrt(1/2)
  dft4(a[0], a[2], a[4], a[6]);
  dft4(a[1], a[3], a[5], a[7]);
  const double2 o0 = a[1], o1 = make_double2(H * (a[3].x + a[3].y), H * (a[3].y - a[3].x)), o2 = mul_mi(a[5]),
                o3 = make_double2(H * (a[7].y - a[7].x), -H * (a[7].x + a[7].y));
  const double2 e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6];
  a[0] = e0 + o0;
  a[4] = e0 - o0;
  a[1] = e1 + o1;
  a[5] = e1 - o1;
  a[2] = e2 + o2;
  a[6] = e2 - o2;
  a[3] = e3 + o3;
  a[7] = e3 - o3;
}

// One stage of nb transforms.  Work item (transform b, butterfly u) reads
// points u + m*(n/R), writes q + R*(u - q) + s*t with q = u mod s; its
// twiddles are w^((u - q) t), absent in the last stage.  W > 0: the
// transforms are the W columns of a tile (item = W u + b); W = 0: rows
// (item = (n/R) b + u).  ld(b, i) and st(b, i, v) are the point accessors.
template <int R, int W, class LD, class ST>
__device__ __forceinline__ void spec_stage(const SpecPlan& P, int t, int nb, const LD& ld, const ST& st) {
  const int nr = P.n / R, s = P.str[t];
  const bool last = t == P.nst - 1;
  const int items = W ? W * nr : nb * nr;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    int b, u;
    if constexpr (W > 0) {
      b = it % W;
      u = it / W;
      if (b >= nb) continue;
    } else {
      b = spec_div(it, P.dn[t]);
      u = it - b * nr;
    }
    double2 a[R];
#pragma unroll
    for (int m = 0; m < R; ++m) a[m] = ld(b, u + m * nr);
    dft<R>(a);
    const int q = u - spec_div(u, P.ds[t]) * s, sp = u - q;
    if (!last) {
#pragma unroll
      for (int m = 1; m < R; ++m) a[m] = cmul(a[m], __ldg(P.tw + sp * m));
    }
#pragma unroll
    for (int m = 0; m < R; ++m) st(b, q + sp * R + s * m, a[m]);
  }
}

// the same for a prime radix without a butterfly of its own: every output
// is a sum over the R points (read again for each of them)
template <int W, class LD, class ST>
__device__ __forceinline__ void spec_stage_any(const SpecPlan& P, int t, int nb, const LD& ld, const ST& st) {
  const int R = P.rad[t], nr = P.n / R, s = P.str[t];
  const int items = W ? W * nr : nb * nr;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    int b, u;
    if constexpr (W > 0) {
      b = it % W;
      u = it / W;
      if (b >= nb) continue;
    } else {
      b = spec_div(it, P.dn[t]);
      u = it - b * nr;
    }
    const int q = u - spec_div(u, P.ds[t]) * s, sp = u - q;
    for (int m = 0; m < R; ++m) {
      double2 v = ld(b, u);
      int w = 0;  // (r m mod R): the twiddle of point r
      for (int r = 1; r < R; ++r) {
        w += m;
        if (w >= R) w -= R;
        v = v + cmul(ld(b, u + r * nr), __ldg(P.tw + w * nr));
      }
      st(b, q + sp * R + s * m, cmul(v, __ldg(P.tw + sp * m)));
    }
  }
}

template <int W, class LD, class ST>
__device__ __forceinline__ void spec_stage_sw(const SpecPlan& P, int t, int nb, const LD& ld, const ST& st) {
  switch (P.rad[t]) {
    case 8: spec_stage<8, W>(P, t, nb, ld, st); break;
    case 4: spec_stage<4, W>(P, t, nb, ld, st); break;
    case 2: spec_stage<2, W>(P, t, nb, ld, st); break;
    case 3: spec_stage<3, W>(P, t, nb, ld, st); break;
    case 5: spec_stage<5, W>(P, t, nb, ld, st); break;
    default: spec_stage_any<W>(P, t, nb, ld, st); break;
  }
}

// A row in shared memory: one padding element after every eight, so that
// the first stage's stores (radix 8, stride 8 between lanes) hit distinct
// banks.
__host__ __device__ __forceinline__ int spec_pad(int i) { return i + (i >> 3); }
__host__ __device__ __forceinline__ int spec_row(int n) { return spec_pad(n - 1) + 1; }

// The transforms between an input accessor and either shared memory
// (kToSmem; returns the buffer that holds the result) or an output
// accessor.  buf0, buf1: nb rows (at(b, i) = offset of point i).
template <int W, bool kToSmem, class IN, class OUT, class AT>
__device__ __forceinline__ double2* spec_fft(const SpecPlan& P, int nb, double2* buf0, double2* buf1, const IN& in,
                                             const OUT& out, const AT& at) {
  double2 *src = buf1, *dst = buf0;
  for (int t = 0; t < P.nst; ++t) {
    auto from = [&](int b, int i) { return src[at(b, i)]; };
    auto to = [&](int b, int i, double2 v) { dst[at(b, i)] = v; };
    const bool first = t == 0, direct = !kToSmem && t == P.nst - 1;
    if (first && direct) spec_stage_sw<W>(P, t, nb, in, out);
    else if (first) spec_stage_sw<W>(P, t, nb, in, to);
    else if (direct) spec_stage_sw<W>(P, t, nb, from, out);
    else spec_stage_sw<W>(P, t, nb, from, to);
    __syncthreads();
    double2* x = src;
    src = dst;
    dst = x;
  }
  return src;
}

}  // namespace anel
