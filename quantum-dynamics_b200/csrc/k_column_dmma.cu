// k_column_dmma.cu -- the FP64 column pass on the FP64 tensor cores.
//
// Per tile of 8 grid columns, the work of k_column.cu (B, absorber, surface
// rows, norm, exp(-iVdt), F) as two GEMMs of mma.sync m16n8k8 .f64.  One
// 16-row operand holds eight grid columns: rows 0-7 their real parts, rows
// 8-15 their imaginary parts, so the thread that gets an accumulator's real
// value also gets its imaginary one and the theta-space work needs no exchange.
//   GEMM1  psi_theta[col][k] = sum_l psi_l[col][l] P[k][l]
//   GEMM2  psi_l[col][l] = (l + 1/2) sum_k (w_k psi_theta[col][k]) P[k][l]
// Both read ONE copy of P (n_theta x n_l, 128 KB at 128 x 128), which stays in
// shared memory while the CTA walks its tiles: w_k is applied to the
// theta-space values and l + 1/2 to the results (two copies, P and (l+1/2) w P,
// would not fit).  The contraction index of an mma may be permuted freely: slot
// (t, i) takes index 2t + i, so GEMM1's operand of P is one 16-byte load.
//
// Bound: FP64 tensor throughput (measured 37.0 TFLOP/s for back-to-back
// m16n8k8, one warp per scheduler or more; plain DFMA chains 34).  FP64
// operands need 8 x 8 values in registers per thread to keep plain FMAs fed
// from shared memory; with mma the warps of an SM read about 64 B a clock.
// Four groups of four warps an SM with a tile of 8 columns each, so that every
// scheduler has a warp of each and one group's loads, phases and stores run under
// the others' products; two groups of eight warps with 16 columns left the tensor
// pipe idle longer (256 x 192 x 128: 235 us against 228, step of 128 x 128 x 64 51.1
// against 48.1).  Per launch, against the SIMT kernel: 256 x 192 x 128 (6.4 GFLOP)
// 835 -> 228 us, 128 x 128 x 64 87 -> 33 us, 64 x 64 x 40 30 -> 14 us (each with 5 us
// of event and launch time).
//
// Shared layouts: a tile is [row][9] complex (9: every 16-byte access of a
// warp touches the eight bank groups evenly); P is [k][nlp], nlp a multiple of
// 16, with the 16-byte units of row k permuted by XOR (swz) so that both the
// pair loads along l (GEMM1) and the loads down k (GEMM2) are free of conflicts.
#include "qd_kernels.h"

namespace {

constexpr int TC = 8;           // grid columns of a tile
constexpr int LD = TC + 1;      // tile row stride (complex)
constexpr int WN = 4;           // warps of a group: its tile's outputs are theirs in turn
constexpr int GT = 32 * WN;     // threads of a group
constexpr int MAXGRP = 16;      // groups of eight angles or orders

__device__ __forceinline__ void dmma(double (&c)[4], const double2 a0, const double2 a1,
                                     double b0, double b1)
{
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0.x), "d"(a0.y), "d"(a1.x), "d"(a1.y), "d"(b0), "d"(b1));
}

// permutation of the 16-byte units of row k of P, within groups of eight
__device__ __forceinline__ int swz(int k) { return ((k & 1) << 2) ^ (((k >> 1) & 3) << 1); }

__device__ __forceinline__ void cp16(void *dst, const void *src, bool valid)
{
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = valid ? 16 : 0;                 // 0: fill the 16 bytes with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d), "l"(src), "r"(n)
               : "memory");
}

__host__ __device__ inline int pad8(int n) { return (n + 7) & ~7; }
__host__ __device__ inline int pad16(int n) { return (n + 15) & ~15; }
inline size_t dmma_smem(int nth, int nl, int tiles)
{
  const size_t rows = pad8(nth) > pad8(nl) ? pad8(nth) : pad8(nl);
  return sizeof(double) * (size_t)pad8(nth) * pad16(nl) + tiles * sizeof(double2) * rows * LD +
         sizeof(double) * pad8(nth);
}

// acc[n] = tile (column g) x P over kb blocks of 8 contraction
// indices; the warp's n-th output group: rows 8 (wn + WN n) + ... of the result.
// The XOR of P's units changes with a block's parity only (GEMM1) or not at
// all (GEMM2), so a lane's addresses advance by constants.
template <int NI, bool FWD>
__device__ __forceinline__ void gemm(double (&acc)[NI][4], const double2 *tile, const double *P,
                                     int nlp, int kb, int ngrp, int wn, int g, int t)
{
#pragma unroll
  for (int n = 0; n < NI; n++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[n][i] = 0.0;
  const double2 *row = tile + 2 * t * LD + g;
  const double *pk[NI];                 // FWD: P[2t][8 grp + g]; else P[8 grp + g][..]
  int o0[NI], o1[NI];                   // FWD: rows 2t, 2t + 1; else even, odd block
#pragma unroll
  for (int n = 0; n < NI; n++) {
    const int grp = wn + WN * n, k = FWD ? 2 * t : 8 * grp + g;
    if (FWD) {
      const int u = 4 * grp + (g >> 1);
      pk[n] = P + (g & 1);
      o0[n] = k * nlp + 2 * (u ^ swz(k));
      o1[n] = (k + 1) * nlp + 2 * (u ^ swz(k + 1));
    } else {
      pk[n] = P + k * nlp;
      o0[n] = 2 * (t ^ swz(k));
      o1[n] = 2 * ((4 + t) ^ swz(k));
    }
  }
  auto block = [&](int b) {
    const double2 a0 = row[0], a1 = row[LD];
    row += 8 * LD;
#pragma unroll
    for (int n = 0; n < NI; n++) {
      if (wn + WN * n >= ngrp) break;             // the same for the whole warp
      double b0, b1;
      if (FWD) {                                  // P[8 b + 2t, + 1][8 grp + g]
        b0 = pk[n][o0[n]];
        b1 = pk[n][o1[n]];
        pk[n] += 8 * nlp;
      } else {                                    // P[8 grp + g][8 b + 2t, + 1]
        const double2 v = *reinterpret_cast<const double2 *>(pk[n] + ((b & 1) ? o1[n] : o0[n]));
        b0 = v.x;
        b1 = v.y;
        if (b & 1) pk[n] += 16;
      }
      dmma(acc[n], a0, a1, b0, b1);
    }
  };
  int b = 0;
  for (; b + 4 <= kb; b += 4) {
    block(0);
    block(1);
    block(2);
    block(3);
  }
  for (; b < kb; b++) block(b);
}

// NG groups of four warps, each with its own tiles and its own barrier: one
// group's loads, theta-space work and stores overlap the others' products.  In
// a group warp wn takes every fourth group of eight outputs, NI of them.
template <int NG, int NI, int MODE>
__global__ void __launch_bounds__(NG * GT, 4 / NG) k_column_dmma(ColumnParams p)
{
  constexpr int NT = NG * GT;
  extern __shared__ __align__(16) unsigned char smem[];
  const int nthp = pad8(p.nth), nlp = pad16(p.nl), nl8 = pad8(p.nl);
  const int rows = nthp > nl8 ? nthp : nl8;
  const int tid = threadIdx.x, grp = tid / GT, gtid = tid % GT;
  const int lane = tid & 31, g = lane >> 2, t = lane & 3;
  double2 *cur = reinterpret_cast<double2 *>(smem) + grp * rows * LD;   // the group's tile [rows][LD]
  double *P = reinterpret_cast<double *>(reinterpret_cast<double2 *>(smem) + NG * rows * LD);
  double *w = P + nthp * nlp;
  const int wn = gtid >> 5;
  const int n12 = (int)p.n12;
  const int tpr = (n12 + TC - 1) / TC;                // tiles per run
  const int ntiles = tpr * p.nruns;
  const int kgrp = nthp >> 3, lgrp = nl8 >> 3;
  pdl_trigger();

  auto group_sync = [&] {
    asm volatile("bar.sync %0, %1;" :: "r"(1 + grp), "r"(GT) : "memory");
  };
  auto run_at = [&](int at) { return p.run_order ? p.run_order[at] : at; };
  auto load_P = [&](int set) {                        // by the whole CTA
    const double *src = p.P + set * p.set_stride;
    const int half = nlp >> 1;
    for (int x = tid; x < nthp * half; x += NT) {
      const int k = x / half, u = x - k * half, l = 2 * u;
      const double *s = src + k * p.nl + l;
      const bool in = k < p.nth;
      reinterpret_cast<double2 *>(P)[k * half + (u ^ swz(k))] =
          make_double2(in && l < p.nl ? __ldg(s) : 0.0, in && l + 1 < p.nl ? __ldg(s + 1) : 0.0);
    }
  };
  // the l-space tile (MID, TAIL) into the group's buffer, rows past n_l and columns past the grid zero
  auto fetch = [&](int tile) {
    if (MODE != COL_HEAD && tile < ntiles) {
      const int at = tile / tpr, c = gtid % TC, q = (tile - at * tpr) * TC + c;
      const double2 *src = reinterpret_cast<const double2 *>(p.lpsi) + (long)run_at(at) * p.nl * p.n12;
      const double2 *s = src + (long)(gtid / TC) * n12 + q;
      double2 *d = cur + (gtid / TC) * LD + c;
      for (int l = gtid / TC; l < nl8; l += GT / TC, s += (long)(GT / TC) * n12, d += GT / TC * LD) {
        const bool ok = l < p.nl && q < n12;
        cp16(d, ok ? s : src, ok);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  for (int k = tid; k < nthp; k += NT) w[k] = k < p.nth ? p.w[k] : 0.0;
  // the CTA's tiles blockIdx.x + i gridDim.x, group i % NG; `at` is their position in the runs' order
  int at = (int)blockIdx.x / tpr, run = run_at(at), set = p.run_set ? p.run_set[run] : 0;
  load_P(set);
  pdl_wait();                                         // psi_l: the l-space pass's output
  int mine = blockIdx.x + grp * gridDim.x;            // this group's next tile
  fetch(mine);
  __syncthreads();                                    // P and w in place
  const int k0 = 8 * wn + 2 * t;                      // this thread's first angle and first order
  // all groups walk the runs of the CTA's tiles in step, as they share P
  for (int tile0 = blockIdx.x; tile0 < ntiles;) {
    at = tile0 / tpr;
    run = run_at(at);
    const int end = (at + 1) * tpr;                   // first tile of the next run
    const int s = p.run_set ? p.run_set[run] : 0;
    if (s != set) {                                   // the same for the whole CTA
      __syncthreads();                                // every read of the old P is done
      set = s;
      load_P(set);
      __syncthreads();
    }
    const long zoff = (long)run * p.nth * p.n12, voff = (long)run * p.vrun;
    double nsum = 0.0, esum = 0.0;
    for (; mine < end; ) {
      const int p0 = (mine - at * tpr) * TC;
      mine += NG * gridDim.x;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      group_sync();                                   // the tile in place

      double acc[NI][4];
      if (MODE != COL_HEAD) {
        // exp(-iVdt) of this thread's values, in flight during GEMM1
        const int q = p0 + g;
        const bool in = q < n12;
        double2 ph[NI][2];
        if (MODE == COL_MID) {
          const double2 *v = p.expV + voff + (long)k0 * n12 + q;
#pragma unroll
          for (int n = 0; n < NI; n++)
#pragma unroll
            for (int i = 0; i < 2; i++)
              if (k0 + 8 * WN * n + i < p.nth && in) ph[n][i] = __ldg(v + (long)(8 * WN * n + i) * n12);
        }
        gemm<NI, false>(acc, cur, P, nlp, lgrp, kgrp, wn, g, t);
        group_sync();                                 // every read of the l-space tile is done
        if (MODE == COL_TAIL) fetch(mine);
        const int j = in ? q / p.n1 : 0, i1 = in ? q - j * p.n1 : 0;
        const double d = in && p.d1 ? p.d1[i1] * p.d2[j] : 1.0;
        const bool fl = in && p.do_flux && j >= p.surf_j0 && j < p.surf_j0 + p.surf_nrows;
        double2 *surf = reinterpret_cast<double2 *>(p.surf) +
                        ((long)run * p.surf_nrows + (fl ? j - p.surf_j0 : 0)) * p.nth * p.n1 + i1;
#pragma unroll
        for (int n = 0; n < NI; n++) {
          if (wn + WN * n >= kgrp) break;
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const int k = k0 + 8 * WN * n + i;
            double2 v = make_double2(acc[n][i], acc[n][2 + i]);
            if (k < p.nth && in) {
              const double wk = w[k];
              if (p.esum)
                esum += wk * (v.x * v.x + v.y * v.y) * p.pot[voff + (long)k * n12 + q];
              v = cscale(v, d);
              if (fl) surf[k * p.n1] = v;
              nsum += wk * (v.x * v.x + v.y * v.y);
              if (MODE == COL_TAIL && p.out_z) p.psi_z[zoff + (long)k * n12 + q] = v;
              if (MODE == COL_MID) v = cscale(cmul(v, ph[n][i]), wk);
            } else {
              v = make_double2(0.0, 0.0);
            }
            if (MODE == COL_MID) cur[k * LD + g] = v;
          }
        }
        if (MODE == COL_TAIL) continue;
      } else {
        for (int x = gtid; x < nthp * TC; x += GT) {
          const int k = x / TC, c = x % TC, q = p0 + c;
          const long o = (long)k * n12 + q;
          double2 z = make_double2(0.0, 0.0);
          if (k < p.nth && q < n12) {
            z = p.psi_z[zoff + o];
            double s, co;
            sincos(p.dt * p.pot[voff + o], &s, &co);  // exp(-i V dt) = (co, -s)
            double2 f = make_double2(co, -s);
            if (p.prestep) {
              // psi / sqrt(v) * v = psi * sqrt(v), principal branch
              // (pre_evolution_with_potential_dt_2, timeEvol.C:519-538)
              double sh, ch;
              sincos(0.5 * atan2(-s, co), &sh, &ch);
              f = make_double2(ch, sh);
            }
            z = cscale(cmul(z, f), w[k]);
          }
          cur[k * LD + c] = z;
        }
      }
      group_sync();                                   // the theta-space tile in place
      gemm<NI, true>(acc, cur, P, nlp, kgrp, lgrp, wn, g, t);
      group_sync();                                   // every read of it is done
      fetch(mine);
      const int q = p0 + g;
      if (q < n12) {
        double2 *dst = reinterpret_cast<double2 *>(p.lpsi) + ((long)run * p.nl + k0) * p.n12 + q;
#pragma unroll
        for (int n = 0; n < NI; n++)
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const int l = k0 + 8 * WN * n + i;
            if (l < p.nl)
              dst[(long)(8 * WN * n + i) * n12] =
                  make_double2((l + 0.5) * acc[n][i], (l + 0.5) * acc[n][2 + i]);
          }
      }
    }
    if (MODE != COL_HEAD) {                           // this thread's sums over the run's tiles
      for (int o = 16; o > 0; o >>= 1) {
        nsum += __shfl_xor_sync(0xffffffffu, nsum, o);
        esum += __shfl_xor_sync(0xffffffffu, esum, o);
      }
      if (lane == 0 && p.norm_out) atomicAdd(p.norm_out + run, nsum);
      if (lane == 0 && p.esum) atomicAdd(p.esum + 3 * run + 2, esum);
    }
    tile0 += (end - tile0 + gridDim.x - 1) / gridDim.x * gridDim.x;   // the CTA's first tile past this run
  }
}

template <int NG, int NI, int MODE>
cudaError_t launch(const ColumnParams &p, cudaStream_t s)
{
  const size_t sm = dmma_smem(p.nth, p.nl, NG);
  const cudaError_t e = allow_smem(k_column_dmma<NG, NI, MODE>);
  if (e != cudaSuccess) return e;
  const long ctas = ((p.n12 + TC - 1) / TC * p.nruns + NG - 1) / NG;  // a tile for every group
  const long slots = 148 * (4 / NG);                  // CTAs resident at once
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ctas < slots ? ctas : slots));
  cfg.blockDim = dim3(NG * GT);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_column_dmma<NG, NI, MODE>, p);
  return cudaGetLastError();
}

template <int NG, int NI> cudaError_t launch_mode(const ColumnParams &p, int mode, cudaStream_t s)
{
  switch (mode) {
    case COL_HEAD: return launch<NG, NI, COL_HEAD>(p, s);
    case COL_MID: return launch<NG, NI, COL_MID>(p, s);
    default: return launch<NG, NI, COL_TAIL>(p, s);
  }
}

}  // namespace

// P and four tiles in shared memory, and no more than MAXGRP groups on either side
bool column_dmma_ok(int nth, int nl)
{
  return pad8(nth) <= 8 * MAXGRP && pad8(nl) <= 8 * MAXGRP && dmma_smem(nth, nl, 4) <= 227 * 1024;
}

cudaError_t launch_column_dmma(const ColumnParams &p, int mode, cudaStream_t s)
{
  // 64 angles and orders or fewer: P and two tiles take 51 KB at most, and two CTAs
  // of two groups share an SM (step of 128 x 128 x 64 48.1 us; one CTA of four groups
  // 49.6, four of one group 57.7, as four copies of P are loaded); more: one CTA
  return pad8(p.nth) <= 64 && pad8(p.nl) <= 64 ? launch_mode<2, 2>(p, mode, s)
                                               : launch_mode<4, 4>(p, mode, s);
}
