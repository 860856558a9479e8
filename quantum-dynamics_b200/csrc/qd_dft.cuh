// qd_dft.cuh -- FP64 DFTs of up to 20 points in registers, natural order in and
// out.  SGN = -1: exp(-2 pi i n m / N), +1: exp(+...).
//
// Composite sizes are P x Q: n = p + P q, Q-point DFTs over q, twiddles
// W_N^{p c}, P-point DFTs over p, X[c + Q d].  Constants come from
// cos_turn() at compile time.
#pragma once
#include "qd_device.cuh"

// cos(2 pi n / d) by its Taylor series after reduction to the first octant
__host__ __device__ constexpr double cos_turn(long n, long d)
{
  n = 8 * (((n % d) + d) % d);
  d = 8 * d;
  if (2 * n > d) n = d - n;                      // cos is even and 1-periodic in turns
  double sign = 1.0;
  if (4 * n > d) {                               // cos(pi - x) = -cos(x)
    n = d / 2 - n;
    sign = -1.0;
  }
  const bool use_sin = 8 * n > d;                // cos(x) = sin(pi/2 - x)
  const double x = 6.283185307179586476925286766559 * (double)(use_sin ? d / 4 - n : n) / (double)d;
  const double x2 = x * x;
  double s = 0.0;
  for (int k = 11; k >= 1; k--)                  // Horner: 1 - x2/(1 2)(1 - x2/(3 4)(...)) or its sine form
    s = x2 / (use_sin ? (double)(2 * k) * (2 * k + 1) : (double)(2 * k - 1) * (2 * k)) * (1.0 - s);
  return sign * (use_sin ? x * (1.0 - s) : 1.0 - s);
}

// z * cos(2 pi n / d)
template <long N, long D> __device__ __forceinline__ double2 kscale(double2 z)
{
  constexpr double c = cos_turn(N, D);
  return make_double2(c * z.x, c * z.y);
}
// z * exp(SGN 2 pi i E / N)
template <int N, int E, int SGN, typename C> __device__ __forceinline__ C twk(C z)
{
  constexpr int e = E % N;
  if constexpr (e == 0) return z;
  else if constexpr (4 * e == N) return cmul_i(z, SGN);
  else if constexpr (2 * e == N) return mk(-z.x, -z.y);
  else if constexpr (4 * e == 3 * N) return cmul_i(z, -SGN);
  else {
    const C c = kscale<e, N>(z), s = kscale<4 * e - N, 4 * N>(z);    // sin x = cos(x - pi/2)
    return SGN > 0 ? mk(c.x - s.y, c.y + s.x) : mk(c.x + s.y, c.y - s.x);
  }
}

template <int N, int SGN, typename C> struct Dft;
#define QD_DFT_BASE(N)                                                                         \
  template <int SGN, typename C> struct Dft<N, SGN, C> {                                       \
    static __device__ __forceinline__ void run(C *v) { SmallDFT<N, C>::run(v, SGN, nullptr, 0); } \
  };
QD_DFT_BASE(2)
QD_DFT_BASE(3)
QD_DFT_BASE(4)
QD_DFT_BASE(8)
#undef QD_DFT_BASE

template <int SGN, typename C> struct Dft<5, SGN, C> {
  static __device__ __forceinline__ void run(C *v)
  {
    const C t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
    const C d1 = csub(v[1], v[4]), d2 = csub(v[2], v[3]);
    const C a1 = cadd(v[0], cadd(kscale<1, 5>(t1), kscale<2, 5>(t2)));
    const C a2 = cadd(v[0], cadd(kscale<2, 5>(t1), kscale<1, 5>(t2)));
    // sin(2 pi / 5) = cos(-2 pi / 20), sin(4 pi / 5) = cos(2 pi 3 / 20)
    const C b1 = cmul_i(cadd(kscale<1, 20>(d1), kscale<3, 20>(d2)), SGN);
    const C b2 = cmul_i(csub(kscale<3, 20>(d1), kscale<1, 20>(d2)), SGN);
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(a1, b1);
    v[4] = csub(a1, b1);
    v[2] = cadd(a2, b2);
    v[3] = csub(a2, b2);
  }
};

template <int P, int Q, int SGN, typename C> struct DftPxQ {
  template <int PP, int CC> static __device__ __forceinline__ void tw(C (&u)[P][Q])
  {
    if constexpr (CC < Q) {
      u[PP][CC] = twk<P * Q, PP * CC, SGN>(u[PP][CC]);
      tw<PP, CC + 1>(u);
    } else if constexpr (PP + 1 < P) {
      tw<PP + 1, 1>(u);
    }
  }
  static __device__ __forceinline__ void run(C *v)
  {
    C u[P][Q];
#pragma unroll
    for (int p = 0; p < P; p++) {
#pragma unroll
      for (int q = 0; q < Q; q++) u[p][q] = v[p + P * q];
      Dft<Q, SGN, C>::run(u[p]);
    }
    tw<1, 1>(u);
#pragma unroll
    for (int c = 0; c < Q; c++) {
      C s[P];
#pragma unroll
      for (int p = 0; p < P; p++) s[p] = u[p][c];
      Dft<P, SGN, C>::run(s);
#pragma unroll
      for (int d = 0; d < P; d++) v[c + Q * d] = s[d];
    }
  }
};
#define QD_DFT_PQ(N, P, Q)                                                                    \
  template <int SGN, typename C> struct Dft<N, SGN, C> {                                      \
    static __device__ __forceinline__ void run(C *v) { DftPxQ<P, Q, SGN, C>::run(v); }        \
  };
QD_DFT_PQ(6, 2, 3)
QD_DFT_PQ(9, 3, 3)
QD_DFT_PQ(10, 2, 5)
QD_DFT_PQ(12, 4, 3)
QD_DFT_PQ(15, 3, 5)
QD_DFT_PQ(16, 4, 4)
QD_DFT_PQ(18, 3, 6)
QD_DFT_PQ(20, 4, 5)
#undef QD_DFT_PQ
