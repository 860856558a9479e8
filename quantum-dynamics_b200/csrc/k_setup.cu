// k_setup.cu -- one-off tables of a propagation, built on the GPU in FP64.
//
//   FP64 form (the reference's tables, same arithmetic):
//     expV[k][j][i] = exp(-i V dt)                       setup_exp_ipot_dt    timeEvol.C:438-463
//     rot[l][j][i]  = exp(-i l(l+1)(I1_i + I2_j) dt/2)   setup_exp_irot_dt_2  timeEvol.C:465-491
//     kin[j][i]     = exp(-i(T1_i + T2_j) dt) / n1 / n2  setup_exp_ikin_dt    timeEvol.C:493-517
//   or, for the kernels of k_axis_f64.cu, the factors of rot and kin in R and in r
//   FP32 form: exp(-i V dt) and the separable factors of the rotational and
//   kinetic phases (exp(-i l(l+1) I1 dt/2), exp(-i l(l+1) I2 dt/2),
//   exp(-i T1 dt), exp(-i T2 dt)), each evaluated in FP64 with the phase
//   reduced to a fraction of a turn and rounded once to complex64, so the
//   complex64 propagation multiplies by unbiased unit-modulus factors.
//   Legendre matrices: P[k][l] = P_l(x_k) (LegendreP2.m:9-21 recurrence) and
//   WP[k][l] = (l+1/2) w_k P_l(x_k) (setup_weight_legendre, timeEvol.C:737-760).
#include "qd_kernels.h"

namespace {

__device__ __forceinline__ double turns(double phase_rad)
{
  const double t = phase_rad * 0.15915494309189533576888376337251;  // 1/(2 pi)
  return t - rint(t);
}

__global__ void k_tables_fp64(int n1, int n2, int nth, int nl, double dt, const double *pot,
                              const double *I1, const double *I2, const double *T1,
                              const double *T2, double2 *expV, double2 *rot, double2 *kin)
{
  const long n12 = (long)n1 * n2;
  const long nv = n12 * nth, nr = rot ? n12 * nl : 0, nk = rot ? n12 : 0;
  const double mdt = -dt, mdt2 = -dt / 2;
  for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < nv + nr + nk;
       g += (long)gridDim.x * blockDim.x) {
    double s, c;
    if (g < nv) {
      sincos(mdt * pot[g], &s, &c);
      expV[g] = make_double2(c, s);
    } else if (g < nv + nr) {
      const long q = g - nv;
      const int l = (int)(q / n12);
      const long ij = q % n12;
      const int j = (int)(ij / n1), i = (int)(ij % n1);
      const double x = (double)(l * (l + 1)) * (I1[i] + I2[j]);
      sincos(x * mdt2, &s, &c);
      rot[q] = make_double2(c, s);
    } else {
      const long ij = g - nv - nr;
      const int j = (int)(ij / n1), i = (int)(ij % n1);
      sincos((T1[i] + T2[j]) * mdt, &s, &c);
      kin[ij] = make_double2(c / n1 / n2, s / n1 / n2);
    }
  }
}

// the separable factors of rot and kin (without the 1/(n1 n2))
__global__ void k_factors_fp64(int n1, int n2, int nl, double dt, const double *I1,
                               const double *I2, const double *T1, const double *T2, double2 *zr1,
                               double2 *zr2, double2 *zk1, double2 *zk2)
{
  const int a1 = nl * n1, a2 = nl * n2;
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < a1 + a2 + n1 + n2;
       g += gridDim.x * blockDim.x) {
    double ph;
    double2 *dst;
    if (g < a1) {
      const int l = g / n1;
      ph = (double)(l * (l + 1)) * I1[g - l * n1] * (-dt / 2);
      dst = zr1 + g;
    } else if (g < a1 + a2) {
      const int q = g - a1, l = q / n2;
      ph = (double)(l * (l + 1)) * I2[q - l * n2] * (-dt / 2);
      dst = zr2 + q;
    } else if (g < a1 + a2 + n1) {
      const int i = g - a1 - a2;
      ph = T1[i] * -dt;
      dst = zk1 + i;
    } else {
      const int j = g - a1 - a2 - n1;
      ph = T2[j] * -dt;
      dst = zk2 + j;
    }
    double s, c;
    sincos(ph, &s, &c);
    *dst = make_double2(c, s);
  }
}

__global__ void k_tables_fp32(int n1, int n2, int nth, int nl, double dt, const double *pot,
                              const double *I1, const double *I2, const double *T1,
                              const double *T2, float2 *expV32, float2 *rc1, float2 *rc2,
                              float2 *kc1, float2 *kc2)
{
  const long nv = (long)n1 * n2 * nth;
  const long a1 = (long)nl * n1, a2 = (long)nl * n2;
  const long total = nv + a1 + a2 + n1 + n2;
  for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < total;
       g += (long)gridDim.x * blockDim.x) {
    // every phase in FP64 (exact turn reduction), rounded once to complex64
    double ph;
    float2 *dst;
    if (g < nv) {
      ph = -dt * pot[g];
      dst = expV32 + g;
    } else if (g < nv + a1) {
      const long q = g - nv;
      const int l = (int)(q / n1), i = (int)(q % n1);
      ph = -(double)(l * (l + 1)) * I1[i] * dt / 2;
      dst = rc1 + q;
    } else if (g < nv + a1 + a2) {
      const long q = g - nv - a1;
      const int l = (int)(q / n2), j = (int)(q % n2);
      ph = -(double)(l * (l + 1)) * I2[j] * dt / 2;
      dst = rc2 + q;
    } else if (g < nv + a1 + a2 + n1) {
      const int i = (int)(g - nv - a1 - a2);
      ph = -T1[i] * dt;
      dst = kc1 + i;
    } else {
      const int j = (int)(g - nv - a1 - a2 - n1);
      ph = -T2[j] * dt;
      dst = kc2 + j;
    }
    double s, c;
    sincospi(2.0 * turns(ph), &s, &c);
    *dst = make_float2((float)c, (float)s);
  }
}

__global__ void k_legendre_matrices(int nth, int nl, const double *w, const double *legendre,
                                    double *P, double *WP, float *P32, float *WP32,
                                    float *P32lo, float *WP32lo)
{
  const int total = nth * nl;
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
    const int k = g / nl, l = g % nl;
    const double p = legendre[l + (long)k * nl];
    const double f = l + 0.5;
    const double wp = f * w[k] * p;
    P[g] = p;
    WP[g] = wp;
    // float + float residual: the fixed rounding of a float-only matrix would
    // make F*B = I + O(1e-7) and drift the norm systematically step by step
    P32[g] = (float)p;
    WP32[g] = (float)wp;
    P32lo[g] = (float)(p - (double)(float)p);
    WP32lo[g] = (float)(wp - (double)(float)wp);
  }
}

// Angular basis at each node, one thread per node, output (m+1) x n
// column-major (leg[l + k*(m+1)]).  K = 0: P_0..P_m by the three-term
// recurrence of LegendreP2.m:9-21, unnormalised as theta.legendre is there.
// K > 0 (a centrifugal-sudden block, H3/main.m:98-101): the associated
// functions Pbar_{K+l}^K normalised to one on [-1, 1], started from
// Pbar_K^K = sqrt(1/2) prod_{j<=K} sqrt((2j+1)/(2j)) (1-x^2)^{1/2} and raised
// in degree by the standard normalised recurrence, then divided by
// sqrt(l + 1/2) to the reference's scaling.
__global__ void k_legendre_basis(int n, int K, int m, const double *x, double *out)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double xk = x[k];
  double *v = out + (long)k * (m + 1);
  if (K == 0) {
    double p0 = 1.0, p1 = xk;
    v[0] = 1.0;
    if (m >= 1) v[1] = xk;
    for (int i = 2; i <= m; i++) {
      const double p2 = (2.0 - 1.0 / i) * xk * p1 - (1.0 - 1.0 / i) * p0;
      v[i] = p2;
      p0 = p1;
      p1 = p2;
    }
    return;
  }
  const double s = sqrt(1.0 - xk * xk);
  double p0 = sqrt(0.5);
  for (int j = 1; j <= K; j++) p0 *= sqrt((2.0 * j + 1.0) / (2.0 * j)) * s;
  v[0] = p0 / sqrt(0.5);
  double p1 = 0.0;
  if (m >= 1) {
    p1 = sqrt(2.0 * K + 3.0) * xk * p0;
    v[1] = p1 / sqrt(1.5);
  }
  for (int l = 2; l <= m; l++) {
    const double j = K + l;
    const double a = sqrt((4.0 * j * j - 1.0) / (j * j - (double)K * K));
    const double b = sqrt(((j - 1) * (j - 1) - (double)K * K) / (4.0 * (j - 1) * (j - 1) - 1.0));
    const double p2 = a * (xk * p1 - b * p0);
    v[l] = p2 / sqrt(l + 0.5);
    p0 = p1;
    p1 = p2;
  }
}

}  // namespace

cudaError_t launch_setup_tables_fp64(int n1, int n2, int nth, int nl, double dt,
                                     const double *pot, const double *I1, const double *I2,
                                     const double *T1, const double *T2, double2 *expV,
                                     double2 *rot, double2 *kin, cudaStream_t s)
{
  k_tables_fp64<<<148 * 8, 256, 0, s>>>(n1, n2, nth, nl, dt, pot, I1, I2, T1, T2, expV, rot, kin);
  return cudaGetLastError();
}

cudaError_t launch_setup_factors_fp64(int n1, int n2, int nl, double dt, const double *I1,
                                      const double *I2, const double *T1, const double *T2,
                                      double2 *zr1, double2 *zr2, double2 *zk1, double2 *zk2,
                                      cudaStream_t s)
{
  const int n = nl * (n1 + n2) + n1 + n2;
  k_factors_fp64<<<(n + 255) / 256, 256, 0, s>>>(n1, n2, nl, dt, I1, I2, T1, T2, zr1, zr2, zk1, zk2);
  return cudaGetLastError();
}

cudaError_t launch_setup_tables_fp32(int n1, int n2, int nth, int nl, double dt,
                                     const double *pot, const double *I1, const double *I2,
                                     const double *T1, const double *T2, float2 *expV32,
                                     float2 *rc1, float2 *rc2, float2 *kc1, float2 *kc2,
                                     cudaStream_t s)
{
  k_tables_fp32<<<148 * 8, 256, 0, s>>>(n1, n2, nth, nl, dt, pot, I1, I2, T1, T2, expV32, rc1,
                                        rc2, kc1, kc2);
  return cudaGetLastError();
}

cudaError_t launch_legendre_matrices(int nth, int nl, const double *, const double *w,
                                     const double *legendre, double *P, double *WP,
                                     float *P32, float *WP32, float *P32lo, float *WP32lo,
                                     cudaStream_t s)
{
  k_legendre_matrices<<<(nth * nl + 255) / 256, 256, 0, s>>>(nth, nl, w, legendre, P, WP, P32,
                                                             WP32, P32lo, WP32lo);
  return cudaGetLastError();
}

namespace {
__global__ void k_widen_c(const float2 *src, double2 *dst, size_t n)
{
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    dst[i] = make_double2(src[i].x, src[i].y);
}
__global__ void k_narrow_c(const double2 *src, float2 *dst, size_t n)
{
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    dst[i] = make_float2((float)src[i].x, (float)src[i].y);
}
}  // namespace

cudaError_t launch_widen_c(const float2 *src, double2 *dst, size_t n, cudaStream_t s)
{
  k_widen_c<<<148 * 8, 256, 0, s>>>(src, dst, n);
  return cudaGetLastError();
}

cudaError_t launch_narrow_c(const double2 *src, float2 *dst, size_t n, cudaStream_t s)
{
  k_narrow_c<<<148 * 8, 256, 0, s>>>(src, dst, n);
  return cudaGetLastError();
}

cudaError_t launch_legendre_basis(int n, int K, int m, const double *x, double *legendre,
                                  cudaStream_t s)
{
  k_legendre_basis<<<(n + 127) / 128, 128, 0, s>>>(n, K, m, x, legendre);
  return cudaGetLastError();
}

// L2 flush of the timed propagation, second half: after the buffer has been
// written (cudaMemsetAsync), read it back, so that the L2 ends up holding
// clean lines of the buffer instead of dirty ones whose write-back would
// otherwise run during the next timed step.
__global__ void __launch_bounds__(512) k_l2_read(const uint4 *buf, size_t n, unsigned *sink)
{
  unsigned acc = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint4 v = buf[i];
    acc ^= v.x ^ v.y ^ v.z ^ v.w;
  }
  if (acc == 0x9e3779b9u) sink[0] = acc;     // keeps the loads; practically never taken
}

cudaError_t launch_l2_read(const void *buf, size_t bytes, cudaStream_t s)
{
  k_l2_read<<<148 * 4, 512, 0, s>>>(static_cast<const uint4 *>(buf), bytes / sizeof(uint4),
                                    reinterpret_cast<unsigned *>(const_cast<void *>(buf)));
  return cudaGetLastError();
}
