// k_axis_f64.cu -- the l-space part of one FP64 split-operator step for any grid
// whose sizes factor into two register transforms:
//     psi_l <- Rot(dt/2) IFFT2 [exp(-i(T1+T2)dt)/(n1 n2)] FFT2 Rot(dt/2) psi_l
// (evolution_dt, timeEvol.C:625-635; tables timeEvol.C:465-517).
//
// As in k_slice_rf.cu, whose sizes are compiled in, the separable phases make
// the slice operator a row operator then a column operator,
//     [D1 IFFT_R K1 FFT_R D1] (each row)  x  [D2 IFFT_r K2 FFT_r D2] (each column),
// and a length N = A B transform is a B-point and an A-point DFT in registers.
// Here A and B are run-time values, each pass a switch over the radices built
// (4 to 10, to 16 and to 20 in kernels of their own, with the registers that
// takes), so every grid of the form is taken.  Two launches a step, a CTA per block of
// rows and per block of columns (about 2048 elements, several CTAs to an SM):
// a slice in complex128 rarely fits one SM's shared memory, and where it does a
// CTA per slice was slower (64 x 64 x 39: 18.3 us against 15.0, 96 x 96 x 48: 29
// against 19).  The shared-memory Stockham kernels (k_lines.cu) take three
// launches, a shared-memory round trip per radix and runtime divisions, and
// read a rotational table as large as the wavepacket twice.
// The row array keeps element i = a + A b of row j at j RS + a + bs b, with bs
// and RS found on the host by counting the bank conflicts of the three passes.
//
// Bound: HBM, or L2 for states that stay there (256 x 192 x 128: 403 MB in 122 us,
// half the measured copy rate).  Per step, Stockham kernels -> these (events
// around the launches): 256 x 192 x 128 471 -> 122 us, 128 x 128 x 64 98 -> 25 us,
// 64 x 64 x 39 38 -> 15 us, 100 x 54 x 29 50 -> 15 us.
#include <algorithm>
#include <map>
#include <mutex>
#include "qd_dft.cuh"
#include "qd_kernels.h"

namespace {

enum Kind { ROWS = 0, COLS = 1 };
constexpr int NT = 128;                               // threads per CTA
constexpr int STATIC_SMEM = 32 * sizeof(double);      // of the energy sums

// factors of a grid, row layout and block sizes
struct Plan {
  int A1, B1, A2, B2;      // n1 = A1 B1, n2 = A2 B2
  int bs, RS;              // row array: block and row stride
  int hr, nrb, tc, ncb;    // rows per CTA and blocks, columns per CTA and blocks
  unsigned mA1, mB1, mQ;   // e / A1, e / B1, e / tc = umulhi(e, m)
};

template <int N> struct Radix { static constexpr int value = N; };
template <int MAXR, typename F> __device__ __forceinline__ void with_radix(int r, F f)
{
#define QD_RADIX(N) case N: f(Radix<N>()); return;
  switch (r) {
    QD_RADIX(4) QD_RADIX(5) QD_RADIX(6) QD_RADIX(8) QD_RADIX(9) QD_RADIX(10)
  }
  if constexpr (MAXR > 10) switch (r) {
    QD_RADIX(12) QD_RADIX(15) QD_RADIX(16)
  }
  if constexpr (MAXR > 16) switch (r) {
    QD_RADIX(18) QD_RADIX(20)
  }
#undef QD_RADIX
}

// kernels by the larger radix of their dimension, as its values take the
// registers (step of 200 x 180 x 40 82 -> 76 us, of 3 runs of 108 x 90 x 50 79 -> 76,
// against one kernel for both dimensions and all radices up to 16)
// 11 to 16: four CTAs, 128 registers (256 x 192 x 128 123 us; five at 102 registers 124,
// three at 168 137; 128 x 128 x 64 25, 28 and 32)
template <int KIND, int MAXR>
__global__ void __launch_bounds__(NT, MAXR > 16 ? 2 : MAXR > 10 ? 4 : 5) k_axis_f64(LineParams p, Plan ax)
{
  typedef double2 C;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[STATIC_SMEM / sizeof(double)];
  const int tid = threadIdx.x;
  const int n1 = p.n1, n2 = p.n2, A1 = ax.A1, B1 = ax.B1, A2 = ax.A2, B2 = ax.B2;
  const int bs = ax.bs, RS = ax.RS;
  const int per_slice = KIND == ROWS ? ax.nrb : ax.ncb;
  pdl_trigger();
  if (KIND == ROWS && (int)blockIdx.x >= p.nruns * p.nl * per_slice) {   // flux preparation
    pdl_wait();
    const int q = ((int)blockIdx.x - p.nruns * p.nl * per_slice) * NT + tid;
    if (q < p.flux.nruns * p.flux.nth * p.flux.n1) flux_point<C>(p.flux, q);
    return;
  }
  const int sl = blockIdx.x / per_slice, blk = blockIdx.x - sl * per_slice;
  const int l = rot_row(p, sl);                       // slice = run * nl + l; l = table row
  const int j0 = KIND == ROWS ? blk * ax.hr : 0, q0 = KIND == COLS ? blk * ax.tc : 0;
  const int nr = min(ax.hr, n2 - j0), nq = ax.tc;     // rows; columns of a tile (some past n1)
  C *X = reinterpret_cast<C *>(smem);
  C *tab = X + (KIND == COLS ? n2 * ax.tc : nr * RS);
  C *r1 = tab, *k1 = r1 + n1, *T1 = k1 + n1;          // ROWS
  C *r2 = tab, *k2 = r2 + n2, *t2 = k2 + n2;          // COLS
  C *g = reinterpret_cast<C *>(p.lpsi) + (long)sl * p.n12;
  if (KIND == ROWS) {
    const C *tw = reinterpret_cast<const C *>(p.tw1);
    for (int e = tid; e < n1; e += NT) {
      r1[e] = __ldg(p.zr1 + l * n1 + e);
      k1[e] = __ldg(p.zk1 + e);
      const int c = __umulhi((unsigned)e, ax.mA1), a = e - c * A1;
      T1[e] = __ldg(tw + a * c);                      // W_n1^(a c) at c A1 + a
    }
  }
  if (KIND == COLS) {
    const double ks = 1.0 / ((double)n1 * n2);
    const C *tw = reinterpret_cast<const C *>(p.tw2);
    for (int e = tid; e < n2; e += NT) {
      r2[e] = __ldg(p.zr2 + l * n2 + e);
      k2[e] = cscale(__ldg(p.zk2 + e), ks);
      t2[e] = __ldg(tw + e);
    }
  }
  pdl_wait();                                         // psi_l: the previous launch's output
  __syncthreads();
  // energy step: this thread's shares of sum T1 |row FFT|^2, sum T2 |column FFT|^2
  // and sum (I1 + I2) |psi_l|^2 (as in k_slice_rf.cu)
  const bool en = p.esum != nullptr;
  double e_k1 = 0.0, e_k2 = 0.0, e_r = 0.0;

  if (KIND == ROWS) {
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
            const double2 z = v[k];
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
        const C *d = X + j * RS + a;
        C v[B];
#pragma unroll
        for (int c = 0; c < B; c++) v[c] = c ? cmul(d[bs * c], cconj(T1[c * A1 + a])) : d[0];
        Dft<B, +1, C>::run(v);
        C *dst = g + (long)(j0 + j) * n1 + a;
#pragma unroll
        for (int b = 0; b < B; b++) dst[A1 * b] = cmul(v[b], r1[a + A1 * b]);
      }
    });
  }

  if (KIND == COLS) {
    // column qq of the tile at qq in its row; rows a' + A2 b
    const int rs = ax.tc;
    // items (qq, a'): D2, B2-point DFT over b, W^(a' c) -> rows a' + A2 c
    with_radix<MAXR>(B2, [&](auto rad) {
      constexpr int B = decltype(rad)::value;
      for (int e = tid; e < nq * A2; e += NT) {
        const int a = __umulhi((unsigned)e, ax.mQ), qq = e - a * nq;
        if (q0 + qq >= n1) continue;
        C *d = X + a * rs + qq;
        C v[B];
        const C *src = g + (long)a * n1 + q0 + qq;
#pragma unroll
        for (int b = 0; b < B; b++) v[b] = src[(long)(A2 * b) * n1];
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
        if (q0 + qq >= n1) continue;
        C *d = X + A2 * c * rs + qq;
        C v[A];
#pragma unroll
        for (int a = 0; a < A; a++) v[a] = d[a * rs];
        Dft<A, -1, C>::run(v);
        if (en) {
#pragma unroll
          for (int k = 0; k < A; k++) {
            const double2 z = v[k];
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
        if (q0 + qq >= n1) continue;
        const C *d = X + a * rs + qq;
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
            const double2 z = v[b];
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
    if (KIND == COLS) {
      const double er = block_sum(e_r, red);
      if (tid == 0) atomicAdd(p.esum + 3 * run + 1, er * jj * (jj + 1.0) * wl);
    }
  }
}

template <int KIND> size_t smem_bytes(const Plan &ax, int n1, int n2)
{
  return sizeof(double2) * (KIND == ROWS ? (size_t)ax.hr * ax.RS + 3 * n1 : (size_t)n2 * ax.tc + 3 * n2);
}

template <int KIND, int MAXR>
cudaError_t launch_one(const LineParams &p, const Plan &ax, cudaStream_t s)
{
  const size_t sm = smem_bytes<KIND>(ax, p.n1, p.n2);
  const cudaError_t e = allow_smem(k_axis_f64<KIND, MAXR>, STATIC_SMEM);
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
  cudaLaunchKernelEx(&cfg, k_axis_f64<KIND, MAXR>, p, ax);
  return cudaGetLastError();
}

template <int KIND> cudaError_t launch_kind(const LineParams &p, const Plan &ax, cudaStream_t s)
{
  const int r = KIND == ROWS ? ax.A1 : ax.A2;            // the larger radix
  return r > 16 ? launch_one<KIND, 20>(p, ax, s) : r > 10 ? launch_one<KIND, 16>(p, ax, s)
                                                          : launch_one<KIND, 10>(p, ax, s);
}

// n = A B with both radices built, the larger as small as it goes, A >= B (the
// row pass reads runs of A elements)
bool factor(int n, int &A, int &B)
{
  static const int built[] = {4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20};
  A = 0;
  for (int a : built)
    for (int b : built)
      if (a * b == n && a >= b && (A == 0 || a < A)) {
        A = a;
        B = b;
      }
  return A != 0;
}

// shared-memory wavefronts of one access by 32 threads to elements x(thread):
// accesses go by groups of 128 bytes' worth of threads
template <typename F> int wavefronts(int elem, F x)
{
  const int group = 128 / elem;
  int total = 0;
  for (int t0 = 0; t0 < 32; t0 += group) {
    int hits[16] = {}, worst = 0;
    for (int t = t0; t < t0 + group; t++) worst = std::max(worst, ++hits[x(t) % group]);
    total += worst;
  }
  return total;
}

// bs >= A and RS >= bs B with the fewest wavefronts over the row passes (a CTA's first
// warp stands for all), the smallest such array
void row_layout(int A, int B, int elem, int &bs, int &RS)
{
  int best = 1 << 30;
  for (int b = A; b <= A + 2; b++)
    for (int pad = 0; pad < 128 / elem; pad++) {
      const int rs = b * B + pad;
      int w = 0;
      for (int c = 0; c < B; c++)
        w += 2 * wavefronts(elem, [&](int t) { return t / A * rs + t % A + b * c; });
      for (int a = 0; a < A; a++)
        w += 2 * wavefronts(elem, [&](int t) { return t / B * rs + b * (t % B) + a; });
      w = w * 1024 + rs;
      if (w < best) {
        best = w;
        bs = b;
        RS = rs;
      }
    }
}

unsigned magic(int d) { return (unsigned)(((1ull << 32) + d - 1) / d); }   // e / d = umulhi(e, magic), e < 2^16

// The plan of an n1 x n2 grid: false if a size has no two built factors.
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
  Plan x{};
  if (!factor(n1, x.A1, x.B1) || !factor(n2, x.A2, x.B2)) return false;
  row_layout(x.A1, x.B1, sizeof(double2), x.bs, x.RS);
  x.mA1 = magic(x.A1);
  x.mB1 = magic(x.B1);
  plans[{n1, n2}] = x;
  out = x;
  return true;
}

}  // namespace

bool axis_f64_ok(int n1, int n2)
{
  Plan ax;
  return plan(n1, n2, ax);
}

cudaError_t launch_axis_f64(const LineParams &p, cudaStream_t s)
{
  Plan ax;
  if (!plan(p.n1, p.n2, ax)) return cudaErrorInvalidValue;
  ax.hr = axis_rows(p.n1, p.n2, p.nruns * p.nl);
  ax.nrb = (p.n2 + ax.hr - 1) / ax.hr;
  // columns of a tile: 16 where four CTAs' tiles still fit an SM and there are two CTAs
  // per SM of them (step of 128 x 128 x 64 53.3 -> 51.3 us, of 4 runs of 144 x 120 x 64
  // 196 -> 189), else 8, one 128-byte segment (72 x 192: 119 us, 123 with 16)
  ax.tc = p.n2 <= 160 && (long)p.nruns * p.nl * ((p.n1 + 15) / 16) >= 296 ? 16 : 8;
  ax.ncb = (p.n1 + ax.tc - 1) / ax.tc;
  ax.mQ = magic(ax.tc);
  const cudaError_t e = launch_kind<ROWS>(p, ax, s);
  return e != cudaSuccess ? e : launch_kind<COLS>(p, ax, s);
}
