// k_axis_f32.cu -- the float form of the kernels of k_axis.cuh, and the host
// side of both: factors, row layout and block sizes of a grid.
#include <map>
#include <mutex>
#include <tuple>
#include "k_axis.cuh"

cudaError_t launch_axis_f32(const LineParams &p, cudaStream_t s) { return axis::launch<float>(p, s); }

namespace {

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

}  // namespace

// The forms of k_axis.cuh for an n1 x n2 grid of elem-byte values: false if a
// size has no two built factors or (fused) the slice does not fit.
bool axis_plan(int n1, int n2, int elem, bool fused, AxisPlan &out)
{
  static std::mutex mu;
  static std::map<std::tuple<int, int, int, bool>, AxisPlan> plans;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(n1, n2, elem, fused);
  const auto it = plans.find(key);
  if (it != plans.end()) {
    out = it->second;
    return true;
  }
  AxisPlan x{};
  if (!factor(n1, x.A1, x.B1) || !factor(n2, x.A2, x.B2)) return false;
  x.max_radix = std::max(x.A1, x.A2);
  row_layout(x.A1, x.B1, elem, x.bs, x.RS);
  // blocks of the split forms: about 2048 elements of 16 bytes or 4096 of 8
  const int target = 32768 / elem;
  x.hr = std::max(1, std::min(n2, target / n1));
  x.nrb = (n2 + x.hr - 1) / x.hr;
  x.hr = (n2 + x.nrb - 1) / x.nrb;
  x.tc = 128 / elem;                         // whole 128-byte segments
  x.ncb = (n1 + x.tc - 1) / x.tc;
  x.mA1 = magic(x.A1);
  x.mB1 = magic(x.B1);
  x.mQ = magic(fused ? n1 : x.tc);
  if (fused && (elem == 8 ? axis::smem_bytes<float, axis::FUSED>(x, n1, n2)
                          : axis::smem_bytes<double, axis::FUSED>(x, n1, n2)) > 227 * 1024)
    return false;
  plans[key] = x;
  out = x;
  return true;
}

int axis_threads(int cluster)
{
  return cluster == SLICE_AX ? axis::threads<axis::FUSED>() : axis::threads<axis::ROWS>();
}
