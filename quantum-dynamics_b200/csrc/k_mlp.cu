// k_mlp.cu -- a small permutation-symmetric MLP surrogate of a triatomic
// potential energy surface, trained and evaluated by this library's own
// kernels.  No counterpart in the reference, which calls its PES routines
// (Fortran/MEX, e.g. FH2/HSW/HSWMex.C) at every grid point; the plain PES
// stays the judge of the surrogate (|dV| on the grid, |dP(E)|) and its
// fallback.
//
// Network: features of the internuclear distances (atom 1 + diatom 2 3),
//   p_ij = exp(-r_ij / 1.5 bohr),  f = (p23, p12 + p13, p12 p13),
// invariant under exchanging atoms 2 and 3, standardised; then four dense
// layers of width 64 with SiLU, and a linear scalar output (standardised V).
// Weights, products, accumulation and Adam are FP32.  (Products on BF16-rounded
// weights left 5.3 meV RMS on the C1 grid against 3.0 meV with FP32 weights,
// same training.)
//
// A training step is two launches.  k_mlp_step takes tiles of 32 samples
// through the whole network in shared memory, forward and backward, with all
// weights beside them; the weight gradients of a CTA's tiles are summed in that
// CTA's row of a partial array.
// k_mlp_adam sums the rows in order and updates the weights.  (One launch per
// layer and direction, activations in global memory and the weight gradients
// on 8 CTAs with atomics, took 342 us a step at 4096 samples; this form takes 20.)
// Inference: one fused kernel per tile of 64 to 512 points (features from the
// Jacobi geometry, all layers in shared memory).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include "qd_err.h"

namespace {

constexpr int W = 64;                   // hidden width
constexpr int NF = 3;                   // features
constexpr int NL = 4;                   // hidden layers
// parameter layout (floats): W1[64][3] b1[64] | W2[64][64] b2 | W3 | W4 | Wo[64] bo
constexpr int layer_off(int l) { return l == 0 ? 0 : W * NF + W + (l - 1) * (W * W + W); }
constexpr int OFF_WO = layer_off(NL), OFF_BO = OFF_WO + W;
constexpr int NPARAM = OFF_BO + 1;
constexpr float FEAT_SCALE = 1.5f;      // bohr

__device__ __forceinline__ float silu(float z) { return z / (1.f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z)
{
  const float s = 1.f / (1.f + __expf(-z));
  return s * (1.f + z * (1.f - s));
}

struct Norm {
  float fmean[NF], fstd[NF];            // feature standardisation
  float vmean, vstd;                    // target standardisation
};

__device__ __forceinline__ void features(float r12, float r23, float r13, const Norm &nm, float *f)
{
  const float p12 = __expf(-r12 / FEAT_SCALE), p23 = __expf(-r23 / FEAT_SCALE),
              p13 = __expf(-r13 / FEAT_SCALE);
  f[0] = (p23 - nm.fmean[0]) / nm.fstd[0];
  f[1] = (p12 + p13 - nm.fmean[1]) / nm.fstd[1];
  f[2] = (p12 * p13 - nm.fmean[2]) / nm.fstd[2];
}

__global__ void k_features(int n, const double *r12, const double *r23, const double *r13,
                           Norm nm, float *F)
{
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    float f[NF];
    features((float)r12[s], (float)r23[s], (float)r13[s], nm, f);
    for (int c = 0; c < NF; c++) F[(long)s * NF + c] = f[c];
  }
}

// Forward and backward over samples [0, n) in tiles of TS, one CTA to a tile at
// a time: part[blockIdx][0..NPARAM) = this CTA's share of d(mean squared
// error)/d(parameters) (GRADS), part[blockIdx][NPARAM] its sum of squared errors.
// 256 threads; a layer's 32 x 64 outputs are 4 samples x 4 outputs a thread over
// one half of the contraction, read four at a time (4 16-byte loads per 32 FMAs;
// 2 x 4 outputs over all of it, 6 loads, took 22.0 us a step at 4096 samples,
// halves 20.6), its weight gradient 4 x 4 entries a thread over the 32 samples
// (2 per 16), straight to the partial row, so that the backward layers are one loop
// (unrolled, with 48 sums in registers, the step waited for instructions: 19.8).
// Bound: the return path of the shared-memory loads (19 000 cycles of one tile's
// 16-byte loads at four cycles each, 10 us; the FMAs take 4 us); smaller tiles
// would not fill more SMs by much and double the weight traffic per sample.
constexpr int TS = 32;                    // samples of a tile
constexpr int LDA = W + 4;                // row stride: 16-byte rows, conflict-free quarter-warps
constexpr int PSTRIDE = (NPARAM + 1 + 3) / 4 * 4;
struct StepSmem {
  float w[NL - 1][W][LDA];                // layers 2..4
  float a[NL][TS][LDA], s[NL][TS][LDA];   // activations, SiLU'(z)
  float d[2][TS][LDA];                    // backward signal, ping-pong
  float x[8][256];                        // halves of a contraction, exchanged
  float f[TS][4];                         // features, and 1 for the bias
  float e[TS];                            // 2 (y - t) / n_total
  float w1[W][NF], b[NL][W], wo[W];
};

// Adds the two halves of a contraction: thread tid holds 4 x 4 partial sums, and of
// their total rows 2 kh, 2 kh + 1 go to z (the other two rows to thread tid ^ 128).
// Between two calls stands the block barrier at the end of a layer.
__device__ __forceinline__ void exchange(StepSmem &m, int kh, int tid, const float (&acc)[4][4],
                                         float (&z)[2][4])
{
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) m.x[4 * i + j][tid ^ 128] = kh ? acc[i][j] : acc[2 + i][j];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) z[i][j] = (kh ? acc[2 + i][j] : acc[i][j]) + m.x[4 * i + j][tid];
}

template <bool GRADS>
__global__ void __launch_bounds__(256, 1) k_mlp_step(int n, float inv_total, const float *F,
                                                     const float *target, const float *w,
                                                     float *part)
{
  extern __shared__ float4 step_sm4[];
  StepSmem &m = *reinterpret_cast<StepSmem *>(step_sm4);
  __shared__ float red[8];
  const int tid = threadIdx.x, tr = tid >> 4, tc = tid & 15;
  const int kh = tid >> 7, tq = tr & 7;   // half of a contraction, its first sample
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");     // the weights: the last step's update
  float fr[NF];                           // features of a tile's sample tid, read ahead
#define QD_FEATURES(s0)                                                    \
  _Pragma("unroll") for (int c = 0; c < NF; c++)                           \
    fr[c] = tid < TS && (s0) + tid < n ? F[(long)((s0) + tid) * NF + c] : 0.f
  {                                       // 16-byte weight rows, all loads in flight together
    static_assert(NL * W == 256 && W * NF <= 256, "one bias and one first weight a thread");
    constexpr int PT = W * W / 4 / 256;
    float4 v[NL - 1][PT];
#pragma unroll
    for (int l = 1; l < NL; l++)
#pragma unroll
      for (int q = 0; q < PT; q++)
        v[l - 1][q] = reinterpret_cast<const float4 *>(w + layer_off(l))[tid + 256 * q];
    const float v1 = tid < W * NF ? w[tid] : 0.f, vo = tid < W ? w[OFF_WO + tid] : 0.f;
    const float vb = w[layer_off(tid / W) + W * (tid / W ? W : NF) + tid % W];
    QD_FEATURES((int)blockIdx.x * TS);
#pragma unroll
    for (int l = 1; l < NL; l++)
#pragma unroll
      for (int q = 0; q < PT; q++) {
        const int x = tid + 256 * q;
        *reinterpret_cast<float4 *>(&m.w[l - 1][x / (W / 4)][4 * (x % (W / 4))]) = v[l - 1][q];
      }
    if (tid < W * NF) m.w1[tid / NF][tid % NF] = v1;
    m.b[tid / W][tid % W] = vb;
    if (tid < W) m.wo[tid] = vo;
  }
  const float bo = w[OFF_BO];
  static_assert(layer_off(1) % 4 == 0 && (W * W + W) % 4 == 0, "16-byte weight rows");

  float *out = part + (size_t)blockIdx.x * PSTRIDE;
  float g1 = 0.f;                         // layer 1: dW[tid / 4][tid % 4], the bias at 3
  float go = 0.f, gbo = 0.f;              // output weight tid - 64 and its bias
  float l2 = 0.f;
  for (int s0 = blockIdx.x * TS; s0 < n; s0 += gridDim.x * TS) {
    if (tid < TS) *reinterpret_cast<float4 *>(m.f[tid]) = make_float4(fr[0], fr[1], fr[2], 1.f);
    const float tgt = s0 + (tid >> 3) < n ? target[s0 + (tid >> 3)] : 0.f;   // of the output stage
    QD_FEATURES(s0 + (int)gridDim.x * TS);
    __syncthreads();                      // features (and, first time, the weights) in place
    {                                     // layer 1: output o of samples s
      const int o = tid & (W - 1);
      const float w0 = m.w1[o][0], w1 = m.w1[o][1], w2 = m.w1[o][2], b = m.b[0][o];
#pragma unroll
      for (int s = tid / W; s < TS; s += 256 / W) {
        const float z = fmaf(m.f[s][2], w2, fmaf(m.f[s][1], w1, fmaf(m.f[s][0], w0, b)));
        m.a[0][s][o] = silu(z);
        if (GRADS) m.s[0][s][o] = dsilu(z);
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int l = 1; l < NL; l++) {
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = kh ? 0.f : m.b[l][tc + 16 * j];
#pragma unroll
      for (int k4 = 0; k4 < W / 2; k4 += 4) {
        const int k = kh * (W / 2) + k4;
        float4 a[4], v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = *reinterpret_cast<const float4 *>(&m.a[l - 1][tq + 8 * i][k]);
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = *reinterpret_cast<const float4 *>(&m.w[l - 1][tc + 16 * j][k]);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++)
            acc[i][j] = fmaf(a[i].w, v[j].w, fmaf(a[i].z, v[j].z,
                        fmaf(a[i].y, v[j].y, fmaf(a[i].x, v[j].x, acc[i][j]))));
      }
      float z[2][4];
      exchange(m, kh, tid, acc, z);
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int s = tq + 8 * (2 * kh + i);
          m.a[l][s][tc + 16 * j] = silu(z[i][j]);
          if (GRADS) m.s[l][s][tc + 16 * j] = dsilu(z[i][j]);
        }
      __syncthreads();
    }
    {                                     // output, loss and its gradient: 8 threads a sample
      const int s = tid >> 3, k0 = (tid & 7) * 4;
      float acc = 0.f;
#pragma unroll
      for (int k = k0; k < W; k += 32)
#pragma unroll
        for (int i = 0; i < 4; i++) acc = fmaf(m.a[NL - 1][s][k + i], m.wo[k + i], acc);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      const float d = s0 + s < n ? acc + bo - tgt : 0.f;
      const float e = 2.f * d * inv_total;
      if ((tid & 7) == 0) {
        l2 = fmaf(d, d, l2);
        m.e[s] = e;
      }
      if (GRADS)
#pragma unroll
        for (int k = k0; k < W; k += 32)
#pragma unroll
          for (int i = 0; i < 4; i++) m.d[0][s][k + i] = e * m.wo[k + i] * m.s[NL - 1][s][k + i];
    }
    __syncthreads();
    if (!GRADS) continue;
    if (tid >= W && tid < 2 * W)          // output weights
#pragma unroll 8
      for (int s = 0; s < TS; s++) {
        go = fmaf(m.e[s], m.a[NL - 1][s][tid - W], go);
        gbo += m.e[s];
      }
    const bool more = s0 != (int)blockIdx.x * TS;     // a tile after the CTA's first
#pragma unroll 1
    for (int l = NL - 1; l >= 1; l--) {
      float (*D)[LDA] = m.d[(NL - 1 - l) & 1], (*Dp)[LDA] = m.d[(NL - l) & 1];
      // dW[o][k] += sum_s D[s][o] A[s][k], entries [4 tr + i][4 tc + j]; the bias: tid < 64
      float *gw = out + layer_off(l) + 4 * tr * W + 4 * tc, *gbp = out + layer_off(l) + W * W + tid;
      float g[4][4] = {}, gb = 0.f;
      if (more) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float4 t = *reinterpret_cast<const float4 *>(gw + i * W);
          g[i][0] = t.x; g[i][1] = t.y; g[i][2] = t.z; g[i][3] = t.w;
        }
        if (tid < W) gb = *gbp;
      }
#pragma unroll 16
      for (int s = 0; s < TS; s++) {
        const float4 x = *reinterpret_cast<const float4 *>(&D[s][4 * tr]);
        const float4 y = *reinterpret_cast<const float4 *>(&m.a[l - 1][s][4 * tc]);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) g[i][j] = fmaf(xs[i], ys[j], g[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
        *reinterpret_cast<float4 *>(gw + i * W) = make_float4(g[i][0], g[i][1], g[i][2], g[i][3]);
      if (tid < W) {
#pragma unroll 8
        for (int s = 0; s < TS; s++) gb += D[s][tid];
        *gbp = gb;
      }
      // D below: (sum_o D[s][o] W[o][k]) SiLU'(z[s][k]), k = 4 tc + j
      float acc[4][4] = {}, y[2][4];
#pragma unroll
      for (int o4 = 0; o4 < W / 2; o4 += 4) {
        const int o = kh * (W / 2) + o4;
        float4 x[4], v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) x[i] = *reinterpret_cast<const float4 *>(&D[tq + 8 * i][o]);
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = *reinterpret_cast<const float4 *>(&m.w[l - 1][o + q][4 * tc]);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
          for (int q = 0; q < 4; q++) {
            acc[i][0] = fmaf(xs[q], v[q].x, acc[i][0]);
            acc[i][1] = fmaf(xs[q], v[q].y, acc[i][1]);
            acc[i][2] = fmaf(xs[q], v[q].z, acc[i][2]);
            acc[i][3] = fmaf(xs[q], v[q].w, acc[i][3]);
          }
        }
      }
      exchange(m, kh, tid, acc, y);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int s = tq + 8 * (2 * kh + i);
        const float4 z = *reinterpret_cast<const float4 *>(&m.s[l - 1][s][4 * tc]);
        *reinterpret_cast<float4 *>(&Dp[s][4 * tc]) =
            make_float4(y[i][0] * z.x, y[i][1] * z.y, y[i][2] * z.z, y[i][3] * z.w);
      }
      __syncthreads();
    }
#pragma unroll 8
    for (int s = 0; s < TS; s++) g1 = fmaf(m.d[(NL - 1) & 1][s][tid >> 2], m.f[s][tid & 3], g1);
    __syncthreads();                      // before the next tile's features
  }

#undef QD_FEATURES

#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l2 += __shfl_xor_sync(0xffffffffu, l2, o);
  if ((tid & 31) == 0) red[tid >> 5] = l2;
  __syncthreads();
  if (tid == 0) {
    float t = 0.f;
    for (int x = 0; x < 8; x++) t += red[x];
    out[NPARAM] = t;
  }
  if (!GRADS) return;
  if ((tid & 3) < NF) out[(tid >> 2) * NF + (tid & 3)] = g1;
  else out[W * NF + (tid >> 2)] = g1;
  if (tid >= W && tid < 2 * W) out[OFF_WO + tid - W] = go;
  if (tid == W) out[OFF_BO] = gbo;
}

// Sums the partial rows of a step: the gradient of parameter p into grad (if
// given, no update), else Adam; the squared errors are added to *loss (set if
// `first`).  32 parameters a CTA, eight threads each over the rows in turn.
struct AdamArgs { float lr, b1, b2, eps, c1, c2; };
__global__ void __launch_bounds__(256) k_mlp_adam(int rows, const float *part, float *w, float *m,
                                                  float *v, AdamArgs a, int first, float *loss,
                                                  float *grad)
{
  __shared__ float red[8][33];
  const int q = threadIdx.x & 31, r0 = threadIdx.x >> 5, p = blockIdx.x * 32 + q;
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");     // the step's partial rows
  float t = 0.f;
  if (p <= NPARAM)
#pragma unroll 16
    for (int r = r0; r < rows; r += 8) t += part[(size_t)r * PSTRIDE + p];
  red[r0][q] = t;
  __syncthreads();
  if (r0 != 0 || p > NPARAM) return;
  float g = 0.f;
#pragma unroll
  for (int x = 0; x < 8; x++) g += red[x][q];
  if (p == NPARAM) {
    *loss = first ? g : *loss + g;
  } else if (grad) {
    grad[p] = g;
  } else {
    const float mi = a.b1 * m[p] + (1.f - a.b1) * g, vi = a.b2 * v[p] + (1.f - a.b2) * g * g;
    m[p] = mi;
    v[p] = vi;
    w[p] -= a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
  }
}

// sums of the unstandardised features and V and of their squares, eight per CTA
__global__ void __launch_bounds__(256) k_mlp_moments(long n, const double *r12, const double *r23,
                                                     const double *r13, const double *V, double *out)
{
  __shared__ double red[8][8];
  double s[8] = {};
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double p12 = exp(-r12[i] / FEAT_SCALE), p23 = exp(-r23[i] / FEAT_SCALE),
                 p13 = exp(-r13[i] / FEAT_SCALE);
    const double f[4] = {p23, p12 + p13, p12 * p13, V[i]};
#pragma unroll
    for (int c = 0; c < 4; c++) {
      s[c] += f[c];
      s[4 + c] += f[c] * f[c];
    }
  }
#pragma unroll
  for (int c = 0; c < 8; c++) {
    for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][c] = s[c];
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    double t = 0.0;
    for (int x = 0; x < 8; x++) t += red[x][threadIdx.x];
    out[blockIdx.x * 8 + threadIdx.x] = t;
  }
}

// standardised targets
__global__ void k_targets(long n, const double *V, Norm nm, float *T)
{
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    T[i] = (float)((V[i] - nm.vmean) / nm.vstd);
}

// a launch that lets the next kernel's prologue overlap it (both kernels of a
// step wait for the one before at entry)
template <typename... P, typename... A>
cudaError_t launch_chained(void (*k)(P...), unsigned grid, size_t smem, A... args)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  qd_count_launches(1);
  return cudaLaunchKernelEx(&cfg, k, args...);
}

template <bool GRADS>
cudaError_t launch_step(int rows, int n, float inv_total, const float *F, const float *T,
                        const float *w, float *part)
{
  const cudaError_t e = cudaFuncSetAttribute(
      k_mlp_step<GRADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StepSmem));
  if (e != cudaSuccess) return e;
  return launch_chained(k_mlp_step<GRADS>, (unsigned)rows, sizeof(StepSmem), n, inv_total, F, T, w, part);
}

cudaError_t launch_adam(int rows, const float *part, float *w, float *m, float *v, const AdamArgs &a,
                        int first, float *loss, float *grad)
{
  return launch_chained(k_mlp_adam, (NPARAM + 32) / 32, 0, rows, part, w, m, v, a, first, loss, grad);
}

// Fused inference on the Jacobi grid (H3/H3PESJacobi.m:5-27 geometry): per
// tile of points, features, four SiLU layers and the output in shared memory;
// V = vmax where a distance <= rmin, else min(V_mlp, vmax) if cap.
struct GridArgs {
  int n1, n2, nth;
  const double *R, *r, *x;
  double f2, f3, vmax, rmin;
  int cap;
};
// Every layer's weights stay in shared memory for the whole launch (loaded once
// per CTA), activations of GP points at a time in place, transposed ([k][point]).
// A thread forms 8 points (4 in tiles below 256) x 2, 4 or 8 outputs as paired FP32 FMAs (fma.rn.f32x2, two
// points a register pair): at 512 points, per k, 2 16-byte loads of activations
// and 2 of weights for 32 paired FMAs.  A 16-byte shared load costs four cycles of
// the return path even when its lanes read one address, so loads per FMA are what
// a tile is chosen by.  Bound: the products (12.4 kFMA per point, 0.36 ms at the FP32 rate on
// 128 x 128 x 64) and the SiLUs (256 exponentials and divisions a point) together.
// There: scalar FMAs, 4 x 4 outputs a thread with scalar loads 1.18 ms; 8 x 4 with
// 16-byte loads 0.96; 8 x 4 paired, weights stored twice (a pair (w, w) one load)
// 0.91, stored once 0.83; 8 x 8 0.77.
constexpr int GT = 512;
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b)
{
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v)
{
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
template <int GP>
struct GridSmem {
  float w[NL - 1][W][W];                  // layers 2..4: [k][o]
  float h[W][GP];                         // activations
  float w1[W][NF], b[NL][W], wo[W];
  float f[GP][NF];
  unsigned char mask[GP];
};
template <int GP>
__global__ void __launch_bounds__(GT, 1) k_mlp_grid(GridArgs g, Norm nm, const float *wq,
                                                    double *pot, long npts, const double *r12p,
                                                    const double *r23p, const double *r13p)
{
  extern __shared__ float4 grid_sm4[];
  GridSmem<GP> &m = *reinterpret_cast<GridSmem<GP> *>(grid_sm4);
  constexpr int PP = GP < 256 ? 4 : 8, PO = GP * W / (GT * PP);   // points and outputs a thread
  constexpr int WV = PO < 4 ? PO : 4;     // weights of a load
  // points 4 tp.. (and GP/2 + 4 tp..), outputs PO to..
  const int tid = threadIdx.x, tp = tid % (GP / PP), to = tid / (GP / PP);
  for (int x = tid; x < (NL - 1) * W * W; x += GT) {
    const int l = x / (W * W), k = x / W % W, o = x % W;
    m.w[l][k][o] = wq[layer_off(l + 1) + o * W + k];
  }
  for (int x = tid; x < W * NF; x += GT) m.w1[x / NF][x % NF] = wq[x];
  for (int x = tid; x < NL * W; x += GT)
    m.b[x / W][x % W] = wq[layer_off(x / W) + W * (x / W ? W : NF) + x % W];
  if (tid < W) m.wo[tid] = wq[OFF_WO + tid];
  const float bo = wq[OFF_BO];
  for (long base = (long)blockIdx.x * GP; base < npts; base += (long)gridDim.x * GP) {
    if (tid < GP) {
      const long q = base + tid;
      float f[NF] = {0.f, 0.f, 0.f};
      unsigned char ok = 0;
      if (q < npts) {
        double r12, r23, r13;
        if (r12p) {
          r12 = r12p[q]; r23 = r23p[q]; r13 = r13p[q];
          ok = 1;
        } else {
          const int i = (int)(q % g.n1), j = (int)((q / g.n1) % g.n2), k = (int)(q / ((long)g.n1 * g.n2));
          const double Rv = g.R[i], rv = g.r[j], c = g.x[k];
          const double a = g.f2 * rv, b = g.f3 * rv;
          r23 = rv;
          r12 = sqrt(a * a + Rv * Rv - 2.0 * g.f2 * rv * Rv * c);
          r13 = sqrt(b * b + Rv * Rv + 2.0 * g.f3 * rv * Rv * c);
          ok = (r12 > g.rmin && r13 > g.rmin && r23 > g.rmin) ? 1 : 0;
        }
        features((float)r12, (float)r23, (float)r13, nm, f);
      }
      for (int c = 0; c < NF; c++) m.f[tid][c] = f[c];
      m.mask[tid] = ok;
    }
    __syncthreads();                      // features (and, first time, the weights) in place
    {
      const int s = tid % GP;
      const float f0 = m.f[s][0], f1 = m.f[s][1], f2 = m.f[s][2];
#pragma unroll 4
      for (int o = tid / GP; o < W; o += GT / GP)
        m.h[o][s] = silu(fmaf(f2, m.w1[o][2], fmaf(f1, m.w1[o][1], fmaf(f0, m.w1[o][0], m.b[0][o]))));
    }
    __syncthreads();
#pragma unroll 1
    for (int l = 1; l < NL; l++) {
      f32x2 acc[PP / 2][PO];               // point pairs x outputs
#pragma unroll
      for (int j = 0; j < PO; j++) {
        const float bj = m.b[l][PO * to + j];
#pragma unroll
        for (int i = 0; i < PP / 2; i++) acc[i][j] = pack2(bj, bj);
      }
#pragma unroll 2
      for (int k = 0; k < W; k++) {
        f32x2 a[PP / 2];
#pragma unroll
        for (int i = 0; i < PP / 2; i += 2) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(&m.h[k][(i ? GP / 2 : 0) + 4 * tp]);
          a[i] = v.x;
          a[i + 1] = v.y;
        }
#pragma unroll
        for (int j = 0; j < PO; j += WV) {
          float w[WV];
          if constexpr (WV == 4) {
            const float4 v = *reinterpret_cast<const float4 *>(&m.w[l - 1][k][PO * to + j]);
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
          } else {
            const float2 v = *reinterpret_cast<const float2 *>(&m.w[l - 1][k][PO * to + j]);
            w[0] = v.x; w[1] = v.y;
          }
#pragma unroll
          for (int c = 0; c < WV; c++) {
            const f32x2 ww = pack2(w[c], w[c]);
#pragma unroll
            for (int i = 0; i < PP / 2; i++) acc[i][j + c] = fma2(a[i], ww, acc[i][j + c]);
          }
        }
      }
      __syncthreads();                    // every read of the activations is done
#pragma unroll
      for (int j = 0; j < PO; j++)
#pragma unroll
        for (int i = 0; i < PP / 2; i += 2) {
          const float2 u = unpack2(acc[i][j]), v = unpack2(acc[i + 1][j]);
          *reinterpret_cast<float4 *>(&m.h[PO * to + j][(i ? GP / 2 : 0) + 4 * tp]) =
              make_float4(silu(u.x), silu(u.y), silu(v.x), silu(v.y));
        }
      __syncthreads();
    }
    if (tid < GP) {                       // output: one thread a point, halves folded pairwise
      float p[W / 2];
#pragma unroll
      for (int k = 0; k < W / 2; k++)
        p[k] = m.h[k][tid] * m.wo[k] + m.h[k + W / 2][tid] * m.wo[k + W / 2];
#pragma unroll
      for (int o = W / 4; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; k++) p[k] += p[k + o];
      const long q = base + tid;
      if (q < npts) {
        double v = (double)(p[0] + bo) * nm.vstd + nm.vmean;
        if (!r12p) {
          if (!m.mask[tid]) v = g.vmax;
          else if (g.cap) v = fmin(v, g.vmax);
        }
        pot[q] = v;
      }
    }
    __syncthreads();
  }
}

template <int GP>
cudaError_t run_mlp_grid(const GridArgs &g, const Norm &nm, const float *wq, double *pot, long npts,
                         const double *r12p, const double *r23p, const double *r13p)
{
  const cudaError_t e = cudaFuncSetAttribute(
      k_mlp_grid<GP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GridSmem<GP>));
  if (e != cudaSuccess) return e;
  const long blocks = (npts + GP - 1) / GP;
  k_mlp_grid<GP><<<(unsigned)(blocks < 148 ? blocks : 148), GT, sizeof(GridSmem<GP>)>>>(
      g, nm, wq, pot, npts, r12p, r23p, r13p);
  return cudaSuccess;
}
cudaError_t launch_mlp_grid(const GridArgs &g, const Norm &nm, const float *wq, double *pot,
                            long npts, const double *r12p, const double *r23p, const double *r13p)
{
  // The tile whose rounds over the 148 SMs take least: a launch takes 10 us and 12,
  // 16.5, 28 or 52 us a round of 64, 128, 256 or 512 points an SM (512 points 22, 26, 38
  // and 62 us, 303 104 386, 268, 235 and 219).  Costs in half microseconds.
  auto cost = [&](long points, long half_us) { return (npts + 148 * points - 1) / (148 * points) * half_us; };
  const long t64 = cost(64, 24), t128 = cost(128, 33), t256 = cost(256, 56), t512 = cost(512, 104);
  const long least = std::min(std::min(t64, t128), std::min(t256, t512));
  const auto run = least == t512 ? run_mlp_grid<512> : least == t256 ? run_mlp_grid<256>
                 : least == t128 ? run_mlp_grid<128> : run_mlp_grid<64>;
  const cudaError_t e = run(g, nm, wq, pot, npts, r12p, r23p, r13p);
  if (e != cudaSuccess) return e;
  qd_count_launches(1);
  return cudaGetLastError();
}

}  // namespace

// ---- host side -----------------------------------------------------------

struct qd_mlp {
  Norm norm{};
  std::vector<float> w;                 // FP32 masters (host copy)
  float *d_w = nullptr, *d_m = nullptr, *d_v = nullptr;
  long step = 0;
  ~qd_mlp()
  {
    for (float *p : {d_w, d_m, d_v}) cudaFree(p);
  }
};

namespace {

// splitmix64 + Box-Muller free uniform init (He-uniform per layer), seeded
uint64_t mix(uint64_t &s)
{
  uint64_t z = (s += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

int upload_params(qd_mlp *m)
{
  QD_CU(cudaMemcpy(m->d_w, m->w.data(), sizeof(float) * NPARAM, cudaMemcpyHostToDevice));
  return QD_OK;
}

}  // namespace

extern "C" {

int qd_mlp_create(qd_mlp **out, uint64_t seed)
{
  if (!out) return qd_errf(QD_ERR_INVALID, "NULL argument");
  qd_mlp *m = new qd_mlp();
  m->w.assign(NPARAM, 0.f);
  uint64_t s = seed;
  for (int l = 0; l <= NL; l++) {
    const int K = l == 0 ? NF : W, nout = l == NL ? 1 : W;
    const int off = l == NL ? OFF_WO : layer_off(l);
    const double a = std::sqrt(6.0 / K);
    for (int x = 0; x < nout * K; x++)
      m->w[off + x] = (float)(a * (2.0 * (double)(mix(s) >> 11) / 9007199254740992.0 - 1.0));
  }
  for (int c = 0; c < NF; c++) { m->norm.fmean[c] = 0.f; m->norm.fstd[c] = 1.f; }
  m->norm.vmean = 0.f;
  m->norm.vstd = 1.f;
  for (float **p : {&m->d_w, &m->d_m, &m->d_v})
    if (cudaMalloc(p, sizeof(float) * NPARAM) != cudaSuccess) {
      cudaGetLastError();
      delete m;
      return qd_errf(QD_ERR_NOMEM, "qd_mlp_create: cudaMalloc failed");
    }
  cudaMemset(m->d_m, 0, sizeof(float) * NPARAM);
  cudaMemset(m->d_v, 0, sizeof(float) * NPARAM);
  int rc = upload_params(m);
  if (rc != QD_OK) { delete m; return rc; }
  *out = m;
  return QD_OK;
}

int qd_mlp_destroy(qd_mlp *m)
{
  delete m;
  return QD_OK;
}

int32_t qd_mlp_n_params(void) { return NPARAM; }

int qd_mlp_get_params(qd_mlp *m, float *w_out, float norm_out[8])
{
  if (!m || !w_out) return qd_errf(QD_ERR_INVALID, "NULL argument");
  QD_CU(cudaMemcpy(w_out, m->d_w, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
  if (norm_out) {
    for (int c = 0; c < NF; c++) { norm_out[c] = m->norm.fmean[c]; norm_out[NF + c] = m->norm.fstd[c]; }
    norm_out[6] = m->norm.vmean;
    norm_out[7] = m->norm.vstd;
  }
  return QD_OK;
}

int qd_mlp_set_params(qd_mlp *m, const float *w, const float norm[8])
{
  if (!m || !w) return qd_errf(QD_ERR_INVALID, "NULL argument");
  m->w.assign(w, w + NPARAM);
  if (norm) {
    for (int c = 0; c < NF; c++) { m->norm.fmean[c] = norm[c]; m->norm.fstd[c] = norm[NF + c]; }
    m->norm.vmean = norm[6];
    m->norm.vstd = norm[7];
  }
  return upload_params(m);
}

// standardisation of features and targets from a training set: FP64 sums on the
// device, one row per CTA, added up here in order
int qd_mlp_fit_normalisation(qd_mlp *m, int64_t n, const double *r12, const double *r23,
                             const double *r13, const double *V)
{
  if (!m || n < 2 || !r12 || !r23 || !r13 || !V) return qd_errf(QD_ERR_INVALID, "bad argument");
  const int blocks = (int)((n + 255) / 256 < 148 * 4 ? (n + 255) / 256 : 148 * 4);
  qd_scratch buf(sizeof(double) * (4 * (size_t)n + 8 * blocks));
  double *d = buf.at<double>();
  if (!d) return qd_errf(QD_ERR_NOMEM, "qd_mlp_fit_normalisation: %zu bytes", buf.bytes);
  const double *src[4] = {r12, r23, r13, V};
  for (int q = 0; q < 4; q++)
    QD_CU(cudaMemcpy(d + q * n, src[q], sizeof(double) * n, cudaMemcpyHostToDevice));
  k_mlp_moments<<<blocks, 256>>>(n, d, d + n, d + 2 * n, d + 3 * n, d + 4 * n);
  qd_count_launches(1);
  QD_CU(cudaGetLastError());
  std::vector<double> rows(8 * (size_t)blocks);
  QD_CU(cudaMemcpy(rows.data(), d + 4 * n, sizeof(double) * rows.size(), cudaMemcpyDeviceToHost));
  double s[8] = {};
  for (int b = 0; b < blocks; b++)
    for (int c = 0; c < 8; c++) s[c] += rows[8 * b + c];
  float *mean[4] = {&m->norm.fmean[0], &m->norm.fmean[1], &m->norm.fmean[2], &m->norm.vmean};
  float *std[4] = {&m->norm.fstd[0], &m->norm.fstd[1], &m->norm.fstd[2], &m->norm.vstd};
  for (int c = 0; c < 4; c++) {
    const double mu = s[c] / n, var = s[4 + c] / n - mu * mu;
    *mean[c] = (float)mu;
    *std[c] = (float)std::sqrt(var > 1e-30 ? var : 1e-30);
  }
  return QD_OK;
}

// Loss (mean squared error of the standardised V) and, if grad_out, its
// gradient with respect to the FP32 parameters, for n samples in one batch.
// With train_steps > 0 instead: that many Adam steps over the data in
// minibatches of `batch` samples (in order, wrapping), learning rate lr
// decaying geometrically to lr_end; loss_out gets the last epoch's mean loss.
int qd_mlp_train(qd_mlp *m, int64_t n, const double *r12, const double *r23, const double *r13,
                 const double *V, int32_t train_steps, int32_t batch, double lr, double lr_end,
                 float *grad_out, double *loss_out)
{
  if (!m || n < 1 || !r12 || !r23 || !r13 || !V || batch < 1)
    return qd_errf(QD_ERR_INVALID, "qd_mlp_train: bad argument");
  const int B = (int)(train_steps > 0 ? (batch < n ? batch : n) : n);
  // one CTA per tile of the batch, 148 at most (one per SM: 140 KB of shared memory)
  const int maxrows = (B + TS - 1) / TS < 148 ? (B + TS - 1) / TS : 148;
  const size_t nd = 4 * (size_t)n;
  const size_t nf = (size_t)n * NF + n + (size_t)maxrows * PSTRIDE + PSTRIDE + 4;
  qd_scratch buf(sizeof(double) * nd + sizeof(float) * nf);
  double *dr = buf.at<double>();
  if (!dr) return qd_errf(QD_ERR_NOMEM, "qd_mlp_train: %zu bytes", buf.bytes);
  float *part = reinterpret_cast<float *>(dr + nd);           // 16-byte rows: first after the doubles
  float *grad = part + (size_t)maxrows * PSTRIDE, *loss = grad + PSTRIDE;
  float *F = loss + 4, *T = F + (size_t)n * NF;
  const double *src[4] = {r12, r23, r13, V};
  for (int q = 0; q < 4; q++)
    QD_CU(cudaMemcpy(dr + q * n, src[q], sizeof(double) * n, cudaMemcpyHostToDevice));
  const int gb = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  k_features<<<gb, 256>>>((int)n, dr, dr + n, dr + 2 * n, m->norm, F);
  k_targets<<<gb, 256>>>(n, dr + 3 * n, m->norm, T);
  qd_count_launches(2);
  QD_CU(cudaGetLastError());
  int64_t counted = n;                                        // samples in *loss
  if (train_steps <= 0) {                                     // gradient / loss only
    const float inv = 1.f / (float)n;
    QD_CU(grad_out ? launch_step<true>(maxrows, (int)n, inv, F, T, m->d_w, part)
                   : launch_step<false>(maxrows, (int)n, inv, F, T, m->d_w, part));
    QD_CU(launch_adam(maxrows, part, nullptr, nullptr, nullptr, AdamArgs{}, 1, loss, grad));
    if (grad_out)
      QD_CU(cudaMemcpy(grad_out, grad, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
  } else {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const double decay = train_steps > 1 ? std::pow(lr_end / lr, 1.0 / (train_steps - 1)) : 1.0;
    double lr_t = lr;
    int64_t s0 = 0;
    for (int st = 0; st < train_steps; st++) {
      const int b = (int)(s0 + B <= n ? B : n - s0);
      const int rows = (b + TS - 1) / TS < maxrows ? (b + TS - 1) / TS : maxrows;
      QD_CU(launch_step<true>(rows, b, 1.f / (float)b, F + s0 * NF, T + s0, m->d_w, part));
      m->step++;
      const AdamArgs a{(float)lr_t, b1, b2, eps, 1.f - std::pow(b1, (float)m->step),
                       1.f - std::pow(b2, (float)m->step)};
      // the first step of an epoch starts its loss
      QD_CU(launch_adam(rows, part, m->d_w, m->d_m, m->d_v, a, s0 == 0, loss, nullptr));
      lr_t *= decay;
      s0 += b;
      counted = s0;
      if (s0 >= n) s0 = 0;
    }
    m->w.resize(NPARAM);
    QD_CU(cudaMemcpy(m->w.data(), m->d_w, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
  }
  float l = 0.f;
  QD_CU(cudaMemcpy(&l, loss, sizeof(float), cudaMemcpyDeviceToHost));
  if (loss_out) *loss_out = l / (double)counted;
  return QD_OK;
}

// V (hartree) at n geometries (r12, r23, r13 in bohr)
int qd_mlp_eval(qd_mlp *m, int64_t n, const double *r12, const double *r23, const double *r13,
                double *V_out)
{
  if (!m || n < 1 || !r12 || !r23 || !r13 || !V_out) return qd_errf(QD_ERR_INVALID, "bad argument");
  qd_scratch buf(sizeof(double) * 4 * (size_t)n);
  double *d = buf.at<double>();
  if (!d) return qd_errf(QD_ERR_NOMEM, "qd_mlp_eval: %zu bytes of device memory", buf.bytes);
  cudaError_t e = cudaMemcpy(d, r12, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, r23, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + 2 * n, r13, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    GridArgs g{};
    e = launch_mlp_grid(g, m->norm, m->d_w, d + 3 * n, n, d, d + n, d + 2 * n);
  }
  if (e == cudaSuccess) e = qd_fetch(V_out, d + 3 * n, sizeof(double) * n);
  if (e != cudaSuccess) return qd_errf(QD_ERR_CUDA, "qd_mlp_eval: %s", cudaGetErrorString(e));
  return QD_OK;
}

// the surrogate on the Jacobi grid, the layout and masking of qd_potential_jacobi
int qd_mlp_potential(qd_mlp *m, const qd_radial *R, const qd_radial *r, const qd_angle *theta,
                     const double masses[3], double vmax, double rmin, int32_t cap, double *pot_out)
{
  if (!m || !R || !r || !theta || !masses || !pot_out || !R->r || !r->r || !theta->x)
    return qd_errf(QD_ERR_INVALID, "NULL argument");
  if (R->n < 1 || r->n < 1 || theta->n < 1 || !(masses[1] + masses[2] > 0))
    return qd_errf(QD_ERR_INVALID, "bad grid or masses");
  GridArgs g{};
  g.n1 = R->n; g.n2 = r->n; g.nth = theta->n;
  g.f2 = masses[2] / (masses[1] + masses[2]);
  g.f3 = 1.0 - g.f2;
  g.vmax = vmax; g.rmin = rmin; g.cap = cap ? 1 : 0;
  const long n = (long)g.n1 * g.n2 * g.nth;
  qd_scratch buf(sizeof(double) * ((size_t)n + g.n1 + g.n2 + g.nth));
  double *d = buf.at<double>();
  if (!d) return qd_errf(QD_ERR_NOMEM, "qd_mlp_potential: %zu bytes of device memory", buf.bytes);
  double *dR = d + n, *dr = dR + g.n1, *dx = dr + g.n2;
  cudaError_t e = cudaMemcpy(dR, R->r, sizeof(double) * g.n1, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dr, r->r, sizeof(double) * g.n2, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dx, theta->x, sizeof(double) * g.nth, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    g.R = dR; g.r = dr; g.x = dx;
    e = launch_mlp_grid(g, m->norm, m->d_w, d, n, nullptr, nullptr, nullptr);
  }
  if (e == cudaSuccess) e = qd_fetch(pot_out, d, sizeof(double) * n);
  if (e != cudaSuccess) return qd_errf(QD_ERR_CUDA, "qd_mlp_potential: %s", cudaGetErrorString(e));
  return QD_OK;
}

}  // extern "C"
