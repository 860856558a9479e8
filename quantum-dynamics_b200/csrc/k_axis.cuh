// k_axis.cuh -- the l-space part of one split-operator step for any grid whose
// sizes factor into two register transforms, in float and in double:
//     psi_l <- Rot(dt/2) IFFT2 [exp(-i(T1+T2)dt)/(n1 n2)] FFT2 Rot(dt/2) psi_l
// (evolution_dt, timeEvol.C:625-635; tables timeEvol.C:465-517).
//
// As in k_slice_rf.cu, whose sizes are compiled in, the separable phases make
// the slice operator a row operator then a column operator,
//     [D1 IFFT_R K1 FFT_R D1] (each row)  x  [D2 IFFT_r K2 FFT_r D2] (each column),
// and a length N = A B transform is a B-point and an A-point DFT in registers.
// Here A and B are run-time values, each pass a switch over the radices built
// (4 to 16, and 18 and 20 in a second kernel with more registers), so one
// kernel takes every grid of the form; what the shared-memory Stockham kernels
// (k_slice.cu, k_lines.cu) spend on radix loops, runtime divisions and a
// shared-memory round trip per radix is gone.  Three forms:
//   fused   one CTA per slice, the whole slice in shared memory: one read and
//           one write of psi_l a step;
//   rows, columns   two launches, a CTA per block of rows and per block of
//           columns: slices that do not fit, and more CTAs than slices.
// The row array keeps element i = a + A b of row j at j RS + a + bs b, with bs
// and RS found on the host by counting the bank conflicts of the three passes.
//
// Bound: HBM or L2 for the split forms (256 x 192 x 128 in double: 403 MB in
// 122 us, half the measured copy rate), the chain of passes on one CTA for
// grids of a few hundred slices.  Per step, Stockham kernels -> these (events
// around the launches): 256 x 192 x 128 double 471 -> 122 us, 128 x 128 x 64
// double 98 -> 28 us, 100 x 54 x 29 double 50 -> 18 us, 3 runs of 108 x 90 x 50
// float 99 -> 28 us, 8 of 96 x 96 x 48 float 105 -> 42 us.
#pragma once
#include "qd_dft.cuh"
#include "qd_kernels.h"

namespace axis {

template <typename R> struct Num;
template <> struct Num<float> {
  typedef float2 C;
  static __device__ __forceinline__ const float2 *r1(const LineParams &p) { return p.rc1; }
  static __device__ __forceinline__ const float2 *r2(const LineParams &p) { return p.rc2; }
  static __device__ __forceinline__ const float2 *k1(const LineParams &p) { return p.kc1; }
  // K2 / (n1 n2), the scale as value + residual
  static __device__ __forceinline__ float2 k2(const LineParams &p, int j)
  { return cscale2(__ldg(p.kc2 + j), p.kscale, p.kscale_lo); }
};
template <> struct Num<double> {
  typedef double2 C;
  static __device__ __forceinline__ const double2 *r1(const LineParams &p) { return p.zr1; }
  static __device__ __forceinline__ const double2 *r2(const LineParams &p) { return p.zr2; }
  static __device__ __forceinline__ const double2 *k1(const LineParams &p) { return p.zk1; }
  static __device__ __forceinline__ double2 k2(const LineParams &p, int j)
  { return cscale(__ldg(p.zk2 + j), 1.0 / ((double)p.n1 * p.n2)); }
};

enum Kind { FUSED = 0, ROWS = 1, COLS = 2 };
// threads: a fused slice keeps its CTA's warps on one SM; the split forms take
// smaller CTAs of about 2048 elements, several to an SM
template <int KIND> constexpr int threads() { return KIND == FUSED ? 256 : 128; }

template <int N> struct Radix { static constexpr int value = N; };
template <int MAXR, typename F> __device__ __forceinline__ void with_radix(int r, F f)
{
  switch (r) {
    case 4: f(Radix<4>()); break;
    case 5: f(Radix<5>()); break;
    case 6: f(Radix<6>()); break;
    case 8: f(Radix<8>()); break;
    case 9: f(Radix<9>()); break;
    case 10: f(Radix<10>()); break;
    case 12: f(Radix<12>()); break;
    case 15: f(Radix<15>()); break;
    case 16: f(Radix<16>()); break;
    default:
      if constexpr (MAXR > 16) {
        if (r == 18) f(Radix<18>());
        else if (r == 20) f(Radix<20>());
      }
  }
}

template <typename R, int KIND, int MAXR>
__global__ void __launch_bounds__(threads<KIND>(), (MAXR > 16 || KIND == FUSED ? 2 : 4))
    k_axis(LineParams p, AxisPlan ax)
{
  typedef typename Num<R>::C C;
  constexpr int NT = threads<KIND>();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[32];
  const int tid = threadIdx.x;
  const int n1 = p.n1, n2 = p.n2, A1 = ax.A1, B1 = ax.B1, A2 = ax.A2, B2 = ax.B2;
  const int bs = ax.bs, RS = ax.RS;
  const int per_slice = KIND == FUSED ? 1 : KIND == ROWS ? ax.nrb : ax.ncb;
  pdl_trigger();
  if (KIND != COLS && (int)blockIdx.x >= p.nruns * p.nl * per_slice) {   // flux preparation
    pdl_wait();
    const int q = ((int)blockIdx.x - p.nruns * p.nl * per_slice) * NT + tid;
    if (q < p.flux.nruns * p.flux.nth * p.flux.n1) flux_point<C>(p.flux, q);
    return;
  }
  const int sl = blockIdx.x / per_slice, blk = blockIdx.x - sl * per_slice;
  const int l = rot_row(p, sl);                       // slice = run * nl + l; l = table row
  const int j0 = KIND == ROWS ? blk * ax.hr : 0, q0 = KIND == COLS ? blk * ax.tc : 0;
  const int nr = KIND == ROWS ? min(ax.hr, n2 - j0) : n2;
  const int nq = KIND == COLS ? ax.tc : n1;           // columns of the tile (COLS: some past n1)
  C *X = reinterpret_cast<C *>(smem);
  C *tab = X + (KIND == COLS ? n2 * ax.tc : nr * RS);
  C *r1 = tab, *k1 = r1 + (KIND == COLS ? 0 : n1), *T1 = k1 + (KIND == COLS ? 0 : n1);
  C *r2 = T1 + (KIND == COLS ? 0 : n1), *k2 = r2 + n2, *t2 = k2 + n2;
  C *g = reinterpret_cast<C *>(p.lpsi) + (long)sl * p.n12;
  if (KIND != COLS) {
    const C *tw = reinterpret_cast<const C *>(p.tw1);
    for (int e = tid; e < n1; e += NT) {
      r1[e] = __ldg(Num<R>::r1(p) + l * n1 + e);
      k1[e] = __ldg(Num<R>::k1(p) + e);
      const int c = __umulhi((unsigned)e, ax.mA1), a = e - c * A1;
      T1[e] = __ldg(tw + a * c);                      // W_n1^(a c) at c A1 + a
    }
  }
  if (KIND != ROWS) {
    const C *tw = reinterpret_cast<const C *>(p.tw2);
    for (int e = tid; e < n2; e += NT) {
      r2[e] = __ldg(Num<R>::r2(p) + l * n2 + e);
      k2[e] = Num<R>::k2(p, e);
      t2[e] = __ldg(tw + e);
    }
  }
  pdl_wait();                                         // psi_l: the previous launch's output
  __syncthreads();
  // energy step: this thread's shares of sum T1 |row FFT|^2, sum T2 |column FFT|^2
  // and sum (I1 + I2) |psi_l|^2 (as in k_slice_rf.cu)
  const bool en = p.esum != nullptr;
  double e_k1 = 0.0, e_k2 = 0.0, e_r = 0.0;

  if (KIND != COLS) {
    // items (j, a): elements a + A1 b, D1, B1-point DFT over b, W^(a c) -> slot a of block c
    with_radix<MAXR>(B1, [&](auto rad) {
      constexpr int B = decltype(rad)::value;
      for (int e = tid; e < nr * A1; e += NT) {
        const int j = __umulhi((unsigned)e, ax.mA1), a = e - j * A1;
        const C *src = g + (long)(j0 + j) * n1 + a;
        C v[B];
#pragma unroll
        for (int b = 0; b < B; b++) v[b] = src[A1 * b];
#pragma unroll
        for (int b = 0; b < B; b++) v[b] = cmul(v[b], r1[a + A1 * b]);
        Dft<B, -1, C>::run(v);
        C *d = X + j * RS + a;
#pragma unroll
        for (int c = 0; c < B; c++) d[bs * c] = c ? cmul(v[c], T1[c * A1 + a]) : v[c];
      }
    });
    __syncthreads();
    // items (j, c): A1-point DFT over the slots of block c -> frequency c + B1 d; K1; inverse
    with_radix<MAXR>(A1, [&](auto rad) {
      constexpr int A = decltype(rad)::value;
      for (int e = tid; e < nr * B1; e += NT) {
        const int j = __umulhi((unsigned)e, ax.mB1), c = e - j * B1;
        C *d = X + j * RS + bs * c;
        C v[A];
#pragma unroll
        for (int a = 0; a < A; a++) v[a] = d[a];
        Dft<A, -1, C>::run(v);
        if (en) {
#pragma unroll
          for (int k = 0; k < A; k++) {
            const double2 z = to_z(v[k]);
            e_k1 += (z.x * z.x + z.y * z.y) * __ldg(p.T1 + c + B1 * k);
          }
        }
#pragma unroll
        for (int k = 0; k < A; k++) v[k] = cmul(v[k], k1[c + B1 * k]);
        Dft<A, +1, C>::run(v);
#pragma unroll
        for (int a = 0; a < A; a++) d[a] = v[a];
      }
    });
    __syncthreads();
    // items (j, a): W^(-a c), B1-point inverse DFT over c -> element a + A1 b, D1
    with_radix<MAXR>(B1, [&](auto rad) {
      constexpr int B = decltype(rad)::value;
      for (int e = tid; e < nr * A1; e += NT) {
        const int j = __umulhi((unsigned)e, ax.mA1), a = e - j * A1;
        C *d = X + j * RS + a;
        C v[B];
#pragma unroll
        for (int c = 0; c < B; c++) v[c] = c ? cmul(d[bs * c], cconj(T1[c * A1 + a])) : d[0];
        Dft<B, +1, C>::run(v);
        if (KIND == ROWS) {
          C *dst = g + (long)(j0 + j) * n1 + a;
#pragma unroll
          for (int b = 0; b < B; b++) dst[A1 * b] = cmul(v[b], r1[a + A1 * b]);
        } else {
#pragma unroll
          for (int b = 0; b < B; b++) d[bs * b] = cmul(v[b], r1[a + A1 * b]);
        }
      }
    });
    if (KIND == FUSED) __syncthreads();
  }

  if (KIND != ROWS) {
    // column qq of the tile: offset qq + (bs - A1) (qq / A1) in a row of the row array, or
    // qq in a row of the column tile; rows a' + A2 b
    const int rs = KIND == FUSED ? RS : ax.tc;
    auto pcol = [&](int qq) {
      return KIND == FUSED ? qq + (bs - A1) * (int)__umulhi((unsigned)qq, ax.mA1) : qq;
    };
    // items (qq, a'): D2, B2-point DFT over b, W^(a' c) -> rows a' + A2 c
    with_radix<MAXR>(B2, [&](auto rad) {
      constexpr int B = decltype(rad)::value;
      for (int e = tid; e < nq * A2; e += NT) {
        const int a = __umulhi((unsigned)e, ax.mQ), qq = e - a * nq;
        if (KIND == COLS && q0 + qq >= n1) continue;
        C *d = X + a * rs + pcol(qq);
        C v[B];
        if (KIND == COLS) {
          const C *src = g + (long)a * n1 + q0 + qq;
#pragma unroll
          for (int b = 0; b < B; b++) v[b] = src[(long)(A2 * b) * n1];
        } else {
#pragma unroll
          for (int b = 0; b < B; b++) v[b] = d[A2 * b * rs];
        }
#pragma unroll
        for (int b = 0; b < B; b++) v[b] = cmul(v[b], r2[a + A2 * b]);
        Dft<B, -1, C>::run(v);
#pragma unroll
        for (int c = 0; c < B; c++) d[A2 * c * rs] = c ? cmul(v[c], t2[a * c]) : v[c];
      }
    });
    __syncthreads();
    // items (qq, c): A2-point DFT over rows a' + A2 c, K2 / (n1 n2), inverse, W^(-a' c)
    with_radix<MAXR>(A2, [&](auto rad) {
      constexpr int A = decltype(rad)::value;
      for (int e = tid; e < nq * B2; e += NT) {
        const int c = __umulhi((unsigned)e, ax.mQ), qq = e - c * nq;
        if (KIND == COLS && q0 + qq >= n1) continue;
        C *d = X + A2 * c * rs + pcol(qq);
        C v[A];
#pragma unroll
        for (int a = 0; a < A; a++) v[a] = d[a * rs];
        Dft<A, -1, C>::run(v);
        if (en) {
#pragma unroll
          for (int k = 0; k < A; k++) {
            const double2 z = to_z(v[k]);
            e_k2 += (z.x * z.x + z.y * z.y) * __ldg(p.T2 + c + B2 * k);
          }
        }
#pragma unroll
        for (int k = 0; k < A; k++) v[k] = cmul(v[k], k2[c + B2 * k]);
        Dft<A, +1, C>::run(v);
#pragma unroll
        for (int a = 0; a < A; a++) d[a * rs] = a ? cmul(v[a], cconj(t2[c * a])) : v[a];
      }
    });
    __syncthreads();
    // items (qq, a'): B2-point inverse DFT over c -> rows a' + A2 b, D2 -> global
    with_radix<MAXR>(B2, [&](auto rad) {
      constexpr int B = decltype(rad)::value;
      for (int e = tid; e < nq * A2; e += NT) {
        const int a = __umulhi((unsigned)e, ax.mQ), qq = e - a * nq;
        if (KIND == COLS && q0 + qq >= n1) continue;
        const C *d = X + a * rs + pcol(qq);
        C v[B];
#pragma unroll
        for (int c = 0; c < B; c++) v[c] = d[A2 * c * rs];
        Dft<B, +1, C>::run(v);
        C *dst = g + (long)a * n1 + q0 + qq;
#pragma unroll
        for (int b = 0; b < B; b++) {
          v[b] = cmul(v[b], r2[a + A2 * b]);
          dst[(long)(A2 * b) * n1] = v[b];
        }
        if (en) {
          const double i1 = __ldg(p.I1 + q0 + qq);
#pragma unroll
          for (int b = 0; b < B; b++) {
            const double2 z = to_z(v[b]);
            e_r += (z.x * z.x + z.y * z.y) * (i1 + __ldg(p.I2 + a + A2 * b));
          }
        }
      }
    });
  }
  if (en) {
    // E_kin (dr1 dr2 applied on the host) = [n2 S1 + S2 / n1] / (n1 n2): S1 sums T1 over the
    // row transforms of D1 psi, S2 sums T2 over the column transforms of the row operator's
    // output, which carries the factor n1 of the unnormalised row transform pair
    const int run = sl / p.nl, ll = sl - run * p.nl;
    const double wl = p.orth ? 1.0 : 1.0 / (ll + 0.5);
    const double jj = (double)l;                       // rotational quantum number j = K + l
    const double ek = block_sum(e_k1 / n1 + e_k2 / ((double)n1 * n1 * n2), red);
    if (tid == 0) atomicAdd(p.esum + 3 * run, ek * wl);
    if (KIND != ROWS) {
      const double er = block_sum(e_r, red);
      if (tid == 0) atomicAdd(p.esum + 3 * run + 1, er * jj * (jj + 1.0) * wl);
    }
  }
}

template <typename R, int KIND> size_t smem_bytes(const AxisPlan &ax, int n1, int n2)
{
  const size_t tile = KIND == FUSED ? (size_t)n2 * ax.RS
                    : KIND == ROWS ? (size_t)ax.hr * ax.RS : (size_t)n2 * ax.tc;
  return 2 * sizeof(R) * (tile + (KIND != COLS ? 3 * n1 : 0) + (KIND != ROWS ? 3 * n2 : 0));
}

template <typename R, int KIND, int MAXR>
cudaError_t launch_one(const LineParams &p, const AxisPlan &ax, cudaStream_t s)
{
  const size_t sm = smem_bytes<R, KIND>(ax, p.n1, p.n2);
  cudaError_t e = cudaFuncSetAttribute(k_axis<R, KIND, MAXR>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  const int per = KIND == FUSED ? 1 : KIND == ROWS ? ax.nrb : ax.ncb;
  cfg.gridDim = dim3((unsigned)(p.nruns * p.nl * per + (KIND != COLS ? p.flux_ctas : 0)));
  cfg.blockDim = dim3(threads<KIND>());
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_axis<R, KIND, MAXR>, p, ax);
  return cudaGetLastError();
}

template <typename R, int MAXR>
cudaError_t launch_class(const LineParams &p, const AxisPlan &ax, cudaStream_t s)
{
  if (p.cluster == SLICE_AX) return launch_one<R, FUSED, MAXR>(p, ax, s);
  cudaError_t e = launch_one<R, ROWS, MAXR>(p, ax, s);
  return e != cudaSuccess ? e : launch_one<R, COLS, MAXR>(p, ax, s);
}

template <typename R> cudaError_t launch(const LineParams &p, cudaStream_t s)
{
  AxisPlan ax;
  if (!axis_plan(p.n1, p.n2, 2 * sizeof(R), p.cluster == SLICE_AX, ax)) return cudaErrorInvalidValue;
  return ax.max_radix > 16 ? launch_class<R, 20>(p, ax, s) : launch_class<R, 16>(p, ax, s);
}

}  // namespace axis
