// Spatial order of external points: by Morton code in the points' own box, 21 bits an axis,
// equal codes in the caller's order, so that consecutive points make a compact group.
//
// The order is that of a stable sort of (code, index).  Runs of 512 are sorted by counting (a
// thread per point compares its code with the run's others, in shared memory); each further
// pass merges eight runs into one: a point's place is its place in its own run plus, for the
// other seven, the number of codes below its own (or equal, in the runs before), found by seven
// binary searches that go in step.  No pass waits for anything but the one before, and 512 x
// 8^k points take 1 + k launches.
//
// Bound by latency: 30k points 73 us for all eight launches (box 7, runs 20, two merges 33, gathers
// 10) against 2.1 ms for finding the box, coding, sorting and gathering on the host; 1M 0.94 ms
// (runs 0.23, four merges 0.65) against 110 ms.
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace bit {

namespace {

constexpr int kRun = 512;   // points sorted by one CTA
constexpr int kWays = 8;    // runs merged in a pass
constexpr int BT = 256;

__device__ __forceinline__ unsigned long long to_key(double v) {  // increasing
  const long long b = __double_as_longlong(v);
  return (unsigned long long)(b ^ ((b >> 63) | (long long)0x8000000000000000ull));
}
__host__ __device__ inline double from_key(unsigned long long k) {
  const unsigned long long b = k >> 63 ? k ^ 0x8000000000000000ull : ~k;
  double v;
  memcpy(&v, &b, sizeof v);
  return v;
}

// box: ~key of the lower bounds, key of the upper ones, then whether some coordinate is NaN
// (all maxima, so zeroed beforehand).
__global__ void __launch_bounds__(BT) k_points_box(int m, const double* x, const double* y, const double* z,
                                                   unsigned long long* box) {
  unsigned long long b[7] = {0, 0, 0, 0, 0, 0, 0};
  for (long long i = blockIdx.x * (long long)BT + threadIdx.x; i < m; i += (long long)gridDim.x * BT) {
    const double v[3] = {x[i], y[i], z[i]};
    for (int q = 0; q < 3; q++) {
      const unsigned long long k = to_key(v[q]);
      b[q] = max(b[q], ~k);
      b[3 + q] = max(b[3 + q], k);
      if (isnan(v[q])) b[6] = 1;
    }
  }
  for (int q = 0; q < 7; q++) {
    for (int o = 16; o; o >>= 1) b[q] = max(b[q], __shfl_xor_sync(0xffffffffu, b[q], o));
    if ((threadIdx.x & 31) == 0 && b[q]) atomicMax(&box[q], b[q]);
  }
}

__device__ __forceinline__ unsigned long long spread3(unsigned long long v) {
  v &= 0x1fffff;
  v = (v | v << 32) & 0x1f00000000ffffULL;
  v = (v | v << 16) & 0x1f0000ff0000ffULL;
  v = (v | v << 8) & 0x100f00f00f00f00fULL;
  v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
  v = (v | v << 2) & 0x1249249249249249ULL;
  return v;
}

__global__ void __launch_bounds__(kRun) k_points_runs(int m, const double* x, const double* y, const double* z,
                                                      const unsigned long long* box, unsigned long long* code,
                                                      int* ord) {
  __shared__ ulonglong2 s_code[kRun / 2];
  unsigned long long* c1 = reinterpret_cast<unsigned long long*>(s_code);
  const int t = threadIdx.x;
  const long long i = (long long)blockIdx.x * kRun + t;
  unsigned long long mine = ~0ull;  // past the end: after every code
  if (i < m) {
    const double v[3] = {x[i], y[i], z[i]};
    mine = 0;
    for (int a = 0; a < 3; a++) {
      const double lo = from_key(~box[a]), hi = from_key(box[3 + a]);
      const double s = hi > lo ? (v[a] - lo) / (hi - lo) : 0.0;
      const double f = s * 2097151.0;
      mine |= spread3((unsigned long long)(f > 0.0 ? fmin(f, 2097151.0) : 0.0)) << a;
    }
  }
  c1[t] = mine;
  __syncthreads();
  int rank = 0;
  for (int k = 0; k < kRun / 2; k++) {
    const ulonglong2 o = s_code[k];
    rank += (o.x < mine || (o.x == mine && 2 * k < t)) + (o.y < mine || (o.y == mine && 2 * k + 1 < t));
  }
  if (i < m) {
    code[i - t + rank] = mine;
    ord[i - t + rank] = (int)i;
  }
}

// Runs of `run` (a power of two; the last may be shorter), eight to one.
__global__ void __launch_bounds__(BT) k_points_merge(int m, long long run, const unsigned long long* code,
                                                     const int* ord, unsigned long long* code2, int* ord2) {
  const long long i = blockIdx.x * (long long)BT + threadIdx.x;
  if (i >= m) return;
  const unsigned long long mine = code[i];
  const long long own = i / run, first = own / kWays * kWays, base = first * run;
  // at[s]: the codes of run s found to come before; the target is the first that does not
  long long at[kWays], len[kWays];
#pragma unroll
  for (int s = 0; s < kWays; s++) {
    const long long b = base + s * run;
    len[s] = first + s == own || b >= m ? 0 : min(run, (long long)m - b);
    at[s] = 0;
  }
  for (long long step = run; step; step >>= 1) {
#pragma unroll
    for (int s = 0; s < kWays; s++) {
      if (at[s] + step > len[s]) continue;
      const unsigned long long o = code[base + s * run + at[s] + step - 1];
      if (o < mine || (o == mine && first + s < own)) at[s] += step;
    }
  }
  long long to = base + (i - own * run);
#pragma unroll
  for (int s = 0; s < kWays; s++) to += at[s];
  code2[to] = mine;
  ord2[to] = ord[i];
}

__global__ void k_points_gather(int m, const int* ord, const double* a, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) out[i] = a[ord[i]];
}

}  // namespace

// Copies the points over and puts them in order: sorted position i holds point ord[i].  lo, hi:
// their box.  Fails on a NaN.
void order_points(Ctx* c, int m, const double* const host[3], DBuf<double> sorted[3], DBuf<int>& ord, double lo[3],
                  double hi[3]) {
  cudaStream_t s = c->stream;
  DBuf<double> raw[3];
  DBuf<unsigned long long> box, code, code2;
  DBuf<int> ord2;
  box.ensure(c, 7);
  for (int a = 0; a < 3; a++) {
    raw[a].ensure(c, m);
    copy_h2d(c, raw[a].p, host[a], m * sizeof(double));
  }
  BIT_CUDA(cudaMemsetAsync(box.p, 0, 7 * sizeof(unsigned long long), s));
  const unsigned nb = std::min<unsigned>(grid_for(m, BT), 2 * c->num_sms);
  count_launch(), k_points_box<<<nb, BT, 0, s>>>(m, raw[0].p, raw[1].p, raw[2].p, box.p);
  BIT_CHECK_LAUNCH();
  code.ensure(c, m);
  ord.ensure(c, m);
  count_launch(), k_points_runs<<<grid_for(m, kRun), kRun, 0, s>>>(m, raw[0].p, raw[1].p, raw[2].p, box.p, code.p,
                                                                  ord.p);
  BIT_CHECK_LAUNCH();
  if (m > kRun) {
    code2.ensure(c, m);
    ord2.ensure(c, m);
  }
  for (long long run = kRun; run < m; run *= kWays) {
    count_launch(), k_points_merge<<<grid_for(m, BT), BT, 0, s>>>(m, run, code.p, ord.p, code2.p, ord2.p);
    BIT_CHECK_LAUNCH();
    std::swap(code.p, code2.p);
    std::swap(code.n, code2.n);
    std::swap(ord.p, ord2.p);
    std::swap(ord.n, ord2.n);
  }
  code.release();
  code2.release();
  ord2.release();
  for (int a = 0; a < 3; a++) {
    sorted[a].ensure(c, m);
    count_launch(), k_points_gather<<<grid_for(m, 256), 256, 0, s>>>(m, ord.p, raw[a].p, sorted[a].p);
    BIT_CHECK_LAUNCH();
    raw[a].release();
  }
  unsigned long long h[7];
  copy_d2h_batch(c, {{h, box.p, sizeof h}});
  if (h[6]) fail(BIT_ERR_INVALID_ARGUMENT, "point coordinates contain NaN");
  for (int a = 0; a < 3; a++) {
    lo[a] = from_key(~h[a]);
    hi[a] = from_key(h[3 + a]);
  }
}

}  // namespace bit
