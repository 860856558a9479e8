// k_axis_f32.cu -- the l-space part of one complex64 split-operator step for any
// grid whose sizes are two groups of one or two radices (every even product of
// 2, 3 and 5 from 6 to 256 but 8 and 162, and some larger ones up to 800):
//     psi_l <- Rot(dt/2) IFFT2 [exp(-i(T1+T2)dt)/(n1 n2)] FFT2 Rot(dt/2) psi_l
// (evolution_dt, timeEvol.C:625-635; tables timeEvol.C:465-517).
//
// The separable kinetic phase K1 K2 makes the transform part a row operator then
// a column operator (k_slice_rf.cu, whose sizes are compiled in),
//     Rot x [IFFT_r K2 FFT_r] (each column) x [IFFT_R K1 FFT_R] (each row) x Rot,
// one launch each, a CTA per block of rows and per block of 16 columns; Rot(dt/2)
// is applied as the row launch loads and as the column launch stores.
//
// The transforms are the Stockham transforms of k_slice.cu and k_lines.cu --
// the same radices in the same order with the same complex64 twiddles -- with
// the stages taken in two groups, each in registers.  A grid's rounding of its
// twiddles shifts the wavepacket's norm by up to 1e-7 a step, either way and
// different for each factorisation; keeping theirs (and Rot as the one rounded
// product of its factors) keeps the results to the random part of the rounding.
// With n = A B, B the product of the first group:
//   pass 1, item a < A:  elements a + A b, the first group's B-point DFT -> slot a of block c
//   pass 2, item c < B:  slots a of block c, the second group's A-point DFT with its
//                        twiddles -> element c + B d
// and the inverse is the same two passes with conjugate twiddles, so each
// operator is four passes over two buffers (X in blocks, Y in natural order).
// A Stockham stage per radix through shared memory, with a runtime division per
// element, was what the other kernels spent their time on.
//
// Bound: the latency of four dependent passes per CTA and two launches for grids
// of a few hundred slices, then L2 (8 runs of 96 x 96 x 48: 113 MB in 45 us).
// Per step, best Stockham form -> this: 3 runs of 108 x 90 x 50 99 -> 26 us,
// 144 x 120 x 64 52 -> 24 us, 200 x 180 x 40 93 -> 30 us.
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>
#include "qd_dft.cuh"
#include "qd_kernels.h"

namespace {

enum Kind { ROWS = 0, COLS = 1 };
constexpr int NT = 128;               // threads per CTA
constexpr int STATIC_SMEM = 32 * sizeof(double);   // of the energy sums
constexpr int TCOLS = 16;             // columns of a tile: whole 128-byte segments

// one dimension: stages (r1, r2) then (r3, r4); r2 = r4 = 1 for single-stage groups
struct Axis {
  int n, A, B;
  int first, second;                  // codes of the two groups: 16 r + r'
  unsigned mA, mB;                    // e / A, e / B = umulhi(e, m)
};
struct Plan {
  Axis x1, x2;
  int bs, RS, RY;                     // row buffers: X block and row stride, Y row stride
  int hr, nrb, ncb;                   // rows per CTA, row blocks, column blocks
};

// z times the complex64 twiddle exp(SGN 2 pi i E / N)
template <int N, int E, int SGN> __device__ __forceinline__ float2 twc(float2 z)
{
  if constexpr (E % N == 0) return z;
  else if constexpr (4 * (E % N) == N) return cmul_i(z, SGN);
  else if constexpr (2 * (E % N) == N) return make_float2(-z.x, -z.y);
  else if constexpr (4 * (E % N) == 3 * N) return cmul_i(z, -SGN);
  else {
    constexpr float c = (float)cos_turn(E, N), s = (float)cos_turn(4 * E - N, 4 * N);
    return cmul(z, make_float2(c, SGN > 0 ? s : -s));
  }
}

// one radix; 5 with the complex64 roots of the table form
template <int R, int SGN> __device__ __forceinline__ void radix(float2 *v)
{
  if constexpr (R == 5) {
    constexpr float c1 = (float)cos_turn(1, 5), c2 = (float)cos_turn(2, 5);
    constexpr float s1 = (float)cos_turn(1, 20), s2 = (float)cos_turn(3, 20);
    const float2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
    const float2 d1 = csub(v[1], v[4]), d2 = csub(v[2], v[3]);
    const float2 a1 = cadd(v[0], make_float2(fmaf(c2, t2.x, c1 * t1.x), fmaf(c2, t2.y, c1 * t1.y)));
    const float2 a2 = cadd(v[0], make_float2(fmaf(c1, t2.x, c2 * t1.x), fmaf(c1, t2.y, c2 * t1.y)));
    const float2 b1 = cmul_i(make_float2(fmaf(s2, d2.x, s1 * d1.x), fmaf(s2, d2.y, s1 * d1.y)), SGN);
    const float2 b2 = cmul_i(make_float2(fmaf(-s1, d2.x, s2 * d1.x), fmaf(-s1, d2.y, s2 * d1.y)), SGN);
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(a1, b1);
    v[4] = csub(a1, b1);
    v[2] = cadd(a2, b2);
    v[3] = csub(a2, b2);
  } else if constexpr (R > 1) {
    SmallDFT<R, float2>::run(v, SGN, nullptr, 0);
  }
}

// the first group on v[b], b < R1 R2 (natural order in and out)
template <int R1, int R2, int SGN> struct First {
  template <int PP, int CC> static __device__ __forceinline__ void tw(float2 (&u)[R2][R1])
  {
    if constexpr (CC < R1) {
      u[PP][CC] = twc<R1 * R2, PP * CC, SGN>(u[PP][CC]);
      tw<PP, CC + 1>(u);
    } else if constexpr (PP + 1 < R2) {
      tw<PP + 1, 1>(u);
    }
  }
  static __device__ __forceinline__ void run(float2 *v)
  {
    if constexpr (R2 == 1) {
      radix<R1, SGN>(v);
    } else {
      float2 u[R2][R1];
#pragma unroll
      for (int p = 0; p < R2; p++) {
#pragma unroll
        for (int q = 0; q < R1; q++) u[p][q] = v[p + R2 * q];
        radix<R1, SGN>(u[p]);
      }
      tw<1, 1>(u);
#pragma unroll
      for (int c = 0; c < R1; c++) {
        float2 s[R2];
#pragma unroll
        for (int p = 0; p < R2; p++) s[p] = u[p][c];
        radix<R2, SGN>(s);
#pragma unroll
        for (int d = 0; d < R2; d++) v[c + R1 * d] = s[d];
      }
    }
  }
};

// the second group on v[a], a < R3 R4, of block c: t points at the block's
// twiddles, entries B apart (axis_f32_twiddles)
template <int R3, int R4, int SGN> __device__ __forceinline__ void second(float2 *v, const float2 *t, int B)
{
  auto by = [&](float2 z, int e) {
    float2 w = t[e * B];
    if (SGN > 0) w.y = -w.y;
    return cmul(z, w);
  };
  float2 u[R4][R3];
#pragma unroll
  for (int p = 0; p < R4; p++) {
#pragma unroll
    for (int q = 0; q < R3; q++) u[p][q] = q ? by(v[p + R4 * q], q - 1) : v[p];
    radix<R3, SGN>(u[p]);
  }
  if constexpr (R4 == 1) {
#pragma unroll
    for (int q = 0; q < R3; q++) v[q] = u[0][q];
  } else {
#pragma unroll
    for (int m = 0; m < R3; m++) {
      float2 s[R4];
#pragma unroll
      for (int p = 0; p < R4; p++) s[p] = p ? by(u[p][m], R3 - 1 + (p - 1) * R3 + m) : u[0][m];
      radix<R4, SGN>(s);
#pragma unroll
      for (int d = 0; d < R4; d++) v[m + R3 * d] = s[d];
    }
  }
}

template <int R, int RR> struct Group { static constexpr int r = R, rr = RR; };
template <bool BIG, typename F> __device__ __forceinline__ void with_group(int code, F f)
{
#define QD_GROUP(R, RR) case 16 * R + RR: f(Group<R, RR>()); return;
  switch (code) {
    QD_GROUP(2, 1) QD_GROUP(3, 1) QD_GROUP(4, 1) QD_GROUP(5, 1) QD_GROUP(8, 1)
    QD_GROUP(2, 3) QD_GROUP(2, 5) QD_GROUP(3, 3) QD_GROUP(3, 5) QD_GROUP(4, 3) QD_GROUP(8, 2)
  }
  if constexpr (BIG) switch (code) {
    QD_GROUP(4, 5) QD_GROUP(5, 5) QD_GROUP(8, 3) QD_GROUP(8, 4)
  }
#undef QD_GROUP
}

// BIG: a group of more than 16 points, whose values take more registers; the
// others run at 64 registers, up to eight CTAs per SM (step of 3 runs of 108 x 90 x 50:
// 48.4 us at 128 registers for all, 40.4 so; 200 x 180 x 40 46.5 and 39.7)
template <int KIND, bool BIG>
__global__ void __launch_bounds__(NT, BIG ? 5 : 8) k_axis_f32(LineParams p, Plan ax)
{
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[STATIC_SMEM / sizeof(double)];
  const int tid = threadIdx.x;
  const int n1 = p.n1, n2 = p.n2;
  const int per_slice = KIND == ROWS ? ax.nrb : ax.ncb;
  pdl_trigger();
  if (KIND == ROWS && (int)blockIdx.x >= p.nruns * p.nl * per_slice) {   // flux preparation
    pdl_wait();
    const int q = ((int)blockIdx.x - p.nruns * p.nl * per_slice) * NT + tid;
    if (q < p.flux.nruns * p.flux.nth * p.flux.n1) flux_point<float2>(p.flux, q);
    return;
  }
  const int sl = blockIdx.x / per_slice, blk = blockIdx.x - sl * per_slice;
  const int l = rot_row(p, sl);                       // slice = run * nl + l; l = table row
  const Axis &x = KIND == ROWS ? ax.x1 : ax.x2;
  const int n = x.n, A = x.A, B = x.B;
  // ROWS: rows j0 .. j0 + nr - 1; COLS: columns q0 .. q0 + nr - 1 (lines of the transform)
  const int j0 = blk * ax.hr, q0 = blk * TCOLS;
  const int nr = KIND == ROWS ? min(ax.hr, n2 - j0) : min(TCOLS, n1 - q0);
  float2 *X = reinterpret_cast<float2 *>(smem);
  float2 *Y = X + (KIND == ROWS ? ax.hr * ax.RS : n2 * TCOLS);
  float2 *d = Y + (KIND == ROWS ? ax.hr * ax.RY : n2 * TCOLS), *k = d + n, *t = k + n;
  float2 *g = reinterpret_cast<float2 *>(p.lpsi) + (long)sl * p.n12;
  {
    const float2 *rc = KIND == ROWS ? p.rc1 + l * n1 : p.rc2 + l * n2;
    const float2 *kc = KIND == ROWS ? p.kc1 : p.kc2, *ts = KIND == ROWS ? p.ts1 : p.ts2;
    for (int e = tid; e < n; e += NT) {
      d[e] = __ldg(rc + e);
      k[e] = __ldg(kc + e);
      t[e] = __ldg(ts + e);
    }
  }
  pdl_wait();                                         // psi_l: the previous launch's output
  __syncthreads();
  // element strides: in X (block, slot, line), in Y (element, line), in global memory
  const int xb = KIND == ROWS ? ax.bs : A * TCOLS, xs = KIND == ROWS ? 1 : TCOLS;
  const int xl = KIND == ROWS ? ax.RS : 1, ys = KIND == ROWS ? 1 : TCOLS;
  const int yl = KIND == ROWS ? ax.RY : 1, gs = KIND == ROWS ? 1 : n1, gl = KIND == ROWS ? n1 : 1;
  float2 *gb = g + (KIND == ROWS ? (long)j0 * n1 : (long)q0);
  // item e of m slots (m = A or B): its line and slot; rows: slots fastest, columns: lines
  auto item = [&](int e, unsigned magic, int m, int &line, int &slot) {
    if (KIND == ROWS) {
      line = __umulhi((unsigned)e, magic);
      slot = e - line * m;
      return line < nr;
    }
    line = e % TCOLS;
    slot = e / TCOLS;
    return line < nr;
  };
  const int lines = KIND == ROWS ? nr : TCOLS;
  // energy step: this thread's shares of sum T |FFT|^2 and (COLS) of sum (I1 + I2) |psi_l|^2,
  // squared in FP64 like the split kernels' (k_lines.cu)
  const bool en = p.esum != nullptr;
  double e_k = 0.0, e_r = 0.0;

  with_group<BIG>(x.first, [&](auto gr) {             // global (ROWS: Rot) -> X
    typedef decltype(gr) G;
    constexpr int NB = G::r * G::rr;
    for (int e = tid; e < lines * A; e += NT) {
      int line, a;
      if (!item(e, x.mA, A, line, a)) continue;
      const float2 *s = gb + (long)line * gl + (long)a * gs;
      float2 v[NB];
#pragma unroll
      for (int b = 0; b < NB; b++) v[b] = s[(long)(A * b) * gs];
      if (KIND == ROWS) {
        const float2 r2 = __ldg(p.rc2 + l * n2 + j0 + line);
#pragma unroll
        for (int b = 0; b < NB; b++) v[b] = cmul(v[b], cmul(d[a + A * b], r2));
      }
      First<G::r, G::rr, -1>::run(v);
#pragma unroll
      for (int c = 0; c < NB; c++) X[line * xl + c * xb + a * xs] = v[c];
    }
  });
  __syncthreads();
  with_group<BIG>(x.second, [&](auto gr) {            // X -> K -> Y
    typedef decltype(gr) G;
    constexpr int NA = G::r * G::rr;
    for (int e = tid; e < lines * B; e += NT) {
      int line, c;
      if (!item(e, x.mB, B, line, c)) continue;
      const float2 *s = X + line * xl + c * xb;
      float2 v[NA];
#pragma unroll
      for (int a = 0; a < NA; a++) v[a] = s[a * xs];
      second<G::r, G::rr, -1>(v, t + c, B);
      if (en) {
        const double *T = KIND == ROWS ? p.T1 : p.T2;
#pragma unroll
        for (int f = 0; f < NA; f++) {
          const double2 z = to_z(v[f]);
          e_k += (z.x * z.x + z.y * z.y) * __ldg(T + c + B * f);
        }
      }
      // (the scale 1 / (n1 n2) on the values, not in the table: a rounded table entry
      // would scale its frequency alike on every step)
#pragma unroll
      for (int f = 0; f < NA; f++) {
        v[f] = cmul(v[f], k[c + B * f]);
        Y[line * yl + (c + B * f) * ys] = KIND == ROWS ? v[f] : cscale2(v[f], p.kscale, p.kscale_lo);
      }
    }
  });
  __syncthreads();
  with_group<BIG>(x.first, [&](auto gr) {             // Y -> X, inverse
    typedef decltype(gr) G;
    constexpr int NB = G::r * G::rr;
    for (int e = tid; e < lines * A; e += NT) {
      int line, a;
      if (!item(e, x.mA, A, line, a)) continue;
      const float2 *s = Y + line * yl + a * ys;
      float2 v[NB];
#pragma unroll
      for (int b = 0; b < NB; b++) v[b] = s[A * b * ys];
      First<G::r, G::rr, +1>::run(v);
#pragma unroll
      for (int c = 0; c < NB; c++) X[line * xl + c * xb + a * xs] = v[c];
    }
  });
  __syncthreads();
  with_group<BIG>(x.second, [&](auto gr) {            // X (COLS: Rot) -> global
    typedef decltype(gr) G;
    constexpr int NA = G::r * G::rr;
    for (int e = tid; e < lines * B; e += NT) {
      int line, c;
      if (!item(e, x.mB, B, line, c)) continue;
      const float2 *s = X + line * xl + c * xb;
      float2 v[NA];
#pragma unroll
      for (int a = 0; a < NA; a++) v[a] = s[a * xs];
      second<G::r, G::rr, +1>(v, t + c, B);
      float2 *o = gb + (long)line * gl + (long)c * gs;
      const float2 r1 = KIND == COLS ? __ldg(p.rc1 + l * n1 + q0 + line) : make_float2(1.f, 0.f);
#pragma unroll
      for (int f = 0; f < NA; f++) {
        if (KIND == COLS) v[f] = cmul(v[f], cmul(r1, d[c + B * f]));
        o[(long)(B * f) * gs] = v[f];
      }
      if (KIND == COLS && en) {
        const double i1 = __ldg(p.I1 + q0 + line);
#pragma unroll
        for (int f = 0; f < NA; f++) {
          const double2 z = to_z(v[f]);
          e_r += (z.x * z.x + z.y * z.y) * (i1 + __ldg(p.I2 + c + B * f));
        }
      }
    }
  });
  if (en) {
    // E_kin (dr1 dr2 applied on the host) = [n2 S1 + S2 / n1] / (n1 n2): S1 sums T1 over the
    // row transforms of D1 psi, S2 sums T2 over the column transforms of the row operator's
    // output, which carries the factor n1 of the unnormalised row transform pair
    const int run = sl / p.nl, ll = sl - run * p.nl;
    const double wl = p.orth ? 1.0 : 1.0 / (ll + 0.5);
    const double jj = (double)l;                       // rotational quantum number j = K + l
    const double ek = block_sum(KIND == ROWS ? e_k / n1 : e_k / ((double)n1 * n1 * n2), red);
    if (tid == 0) atomicAdd(p.esum + 3 * run, ek * wl);
    if (KIND == COLS) {
      const double er = block_sum(e_r, red);
      if (tid == 0) atomicAdd(p.esum + 3 * run + 1, er * jj * (jj + 1.0) * wl);
    }
  }
}

template <int KIND, bool BIG> cudaError_t launch_one(const LineParams &p, const Plan &ax, cudaStream_t s)
{
  const size_t sm = sizeof(float2) * (KIND == ROWS ? (size_t)ax.hr * (ax.RS + ax.RY) + 3 * p.n1
                                                   : 2 * (size_t)p.n2 * TCOLS + 3 * p.n2);
  const cudaError_t e = allow_smem(k_axis_f32<KIND, BIG>, STATIC_SMEM);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  const int per = KIND == ROWS ? ax.nrb : ax.ncb;
  cfg.gridDim = dim3((unsigned)(p.nruns * p.nl * per + (KIND == ROWS ? p.flux_ctas : 0)));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_axis_f32<KIND, BIG>, p, ax);
  return cudaGetLastError();
}

// the two groups of n's Stockham stages (greedy 8, 4, 2, 3, 5, as the FftPlan of
// the same size): a cut with at most two stages a side and the smaller larger product
bool stages(int n, std::vector<int> &first, std::vector<int> &second)
{
  std::vector<int> r;
  for (int m = n; m > 1;) {
    int f = 0;
    for (int c : {8, 4, 2, 3, 5})
      if (m % c == 0) { f = c; break; }
    if (!f) return false;
    r.push_back(f);
    m /= f;
  }
  int best = 33;
  for (size_t cut = 1; cut < r.size(); cut++) {
    if (cut > 2 || r.size() - cut > 2) continue;
    int a = 1, b = 1;
    for (size_t x = 0; x < r.size(); x++) (x < cut ? b : a) *= r[x];
    if (std::max(a, b) < best) {
      best = std::max(a, b);
      first.assign(r.begin(), r.begin() + cut);
      second.assign(r.begin() + cut, r.end());
    }
  }
  return best < 33;
}

unsigned magic(int d) { return (unsigned)(((1ull << 32) + d - 1) / d); }   // e / d = umulhi(e, magic), e < 2^16

bool axis(int n, Axis &x)
{
  std::vector<int> f, s;
  if (!stages(n, f, s)) return false;
  x.n = n;
  x.B = f[0] * (f.size() > 1 ? f[1] : 1);
  x.A = s[0] * (s.size() > 1 ? s[1] : 1);
  x.first = 16 * f[0] + (f.size() > 1 ? f[1] : 1);
  x.second = 16 * s[0] + (s.size() > 1 ? s[1] : 1);
  x.mA = magic(x.A);
  x.mB = magic(x.B);
  return true;
}

// shared-memory wavefronts of one access by 32 threads to elements x(thread): half-warps
// of 8-byte accesses over 16 bank pairs
template <typename F> int wavefronts(F x)
{
  int total = 0;
  for (int t0 = 0; t0 < 32; t0 += 16) {
    int hits[16] = {}, worst = 0;
    for (int t = t0; t < t0 + 16; t++) worst = std::max(worst, ++hits[x(t) & 15]);
    total += worst;
  }
  return total;
}

// strides of the row buffers with the fewest wavefronts over the passes (a CTA's first
// warp stands for all): X by blocks c bs + a, Y in natural order
void row_layout(const Axis &x, int &bs, int &RS, int &RY)
{
  int best = 1 << 30;
  for (int b = x.A; b <= x.A + 2; b++)
    for (int pad = 0; pad < 16; pad++) {
      const int rs = b * x.B + pad;
      int w = 0;
      for (int c = 0; c < x.B; c++)
        w += wavefronts([&](int t) { return t / x.A * rs + t % x.A + b * c; });
      for (int a = 0; a < x.A; a++)
        w += wavefronts([&](int t) { return t / x.B * rs + b * (t % x.B) + a; });
      if (w * 1024 + rs < best) {
        best = w * 1024 + rs;
        bs = b;
        RS = rs;
      }
    }
  best = 1 << 30;
  for (int pad = 0; pad < 16; pad++) {
    const int ry = x.n + pad;
    const int w = x.A * wavefronts([&](int t) { return t / x.B * ry + t % x.B; }) +
                  x.B * wavefronts([&](int t) { return t / x.A * ry + t % x.A; });
    if (w * 1024 + ry < best) {
      best = w * 1024 + ry;
      RY = ry;
    }
  }
}

// The plan of an n1 x n2 grid: false if a size is not two built groups.
bool plan(int n1, int n2, Plan &out)
{
  static std::mutex mu;
  static std::map<std::pair<int, int>, Plan> plans;
  std::lock_guard<std::mutex> lock(mu);
  const auto it = plans.find({n1, n2});
  if (it != plans.end()) {
    out = it->second;
    return true;
  }
  Plan p{};
  if (!axis(n1, p.x1) || !axis(n2, p.x2)) return false;
  row_layout(p.x1, p.bs, p.RS, p.RY);
  p.ncb = (n1 + TCOLS - 1) / TCOLS;
  plans[{n1, n2}] = p;
  out = p;
  return true;
}

}  // namespace

bool axis_f32_ok(int n1, int n2)
{
  Plan ax;
  return plan(n1, n2, ax);
}

int axis_threads() { return NT; }

// Rows per CTA of the row launches (both precisions): about 2048 elements, and
// fewer where that leaves less than two CTAs per SM (FP64 step: 64 x 64 x 39
// 26 -> 22 us, 100 x 54 x 29 26 -> 21 us; four per SM cost as much as they gain)
int axis_rows(int n1, int n2, int slices)
{
  const long fill = (long)n2 * slices / 296;
  const int most = std::max(1, std::min(n2, 2048 / n1));
  const int hr = (int)std::max(1L, std::min((long)most, fill));
  const int blocks = (n2 + hr - 1) / hr;
  return (n2 + blocks - 1) / blocks;
}

// second-group twiddles of a size from its n complex64 roots, laid out [entry][c]
// (consecutive items read consecutive values): entries q - 1 (0 < q < r3) are
// W^(q c r4), entries r3 - 1 + (p - 1) r3 + m (0 < p < r4, m < r3) are W^(p (c + B m))
std::vector<float2> axis_f32_twiddles(int n, const std::vector<float2> &roots)
{
  std::vector<float2> t(n, make_float2(0.f, 0.f));
  Axis x;
  if (!axis(n, x)) return t;
  const int r3 = x.second / 16, r4 = x.second % 16;
  for (int c = 0; c < x.B; c++) {
    for (int q = 1; q < r3; q++) t[(q - 1) * x.B + c] = roots[q * c * r4];
    for (int p = 1; p < r4; p++)
      for (int m = 0; m < r3; m++) t[(r3 - 1 + (p - 1) * r3 + m) * x.B + c] = roots[p * (c + x.B * m)];
  }
  return t;
}

cudaError_t launch_axis_f32(const LineParams &p, cudaStream_t s)
{
  Plan ax;
  if (!plan(p.n1, p.n2, ax)) return cudaErrorInvalidValue;
  ax.hr = axis_rows(p.n1, p.n2, p.nruns * p.nl);
  ax.nrb = (p.n2 + ax.hr - 1) / ax.hr;
  const bool big1 = std::max(ax.x1.A, ax.x1.B) > 16, big2 = std::max(ax.x2.A, ax.x2.B) > 16;
  const cudaError_t e = big1 ? launch_one<ROWS, true>(p, ax, s) : launch_one<ROWS, false>(p, ax, s);
  if (e != cudaSuccess) return e;
  return big2 ? launch_one<COLS, true>(p, ax, s) : launch_one<COLS, false>(p, ax, s);
}
