// What the near-field kernels of the potentials (near.cu) and the fields (near_field.cu) share.
#pragma once

#include <limits.h>

#include "common.cuh"
#include "fp64math.cuh"

namespace bit {

// How the potentials' kernels take a list of cnt targets: blocks of 64, two a lane (the last
// one if 49 or more are left); a block of 32, one a lane, if more than 32 of at most 48 are
// left; the rest (at most 32) with a power of two of lanes to a target.
struct NearSteps {
  int full, one, tail;  // blocks of 64, of 32, targets left
};
__host__ __device__ __forceinline__ NearSteps near_steps(int cnt) {
  NearSteps s;
  s.full = cnt >> 6;
  int r = cnt & 63;
  if (r > 48) { s.full++; r = 0; }
  s.one = r > 32;
  s.tail = s.one ? r - 32 : r;
  return s;
}
// log2 of the lanes that share one of r (1..32) targets
__host__ __device__ __forceinline__ int near_tail_shift(int r) {
  int k = 0;
  while (k < 5 && (r << (k + 1)) <= 32) k++;
  return k;
}
// The time one source takes against cnt targets, in 1/32 of a step of one target a lane.
__host__ __device__ __forceinline__ int near_weight(int cnt) {
  const NearSteps s = near_steps(cnt);
  return 64 * s.full + 32 * s.one + (s.tail ? 32 >> near_tail_shift(s.tail) : 0);
}

struct NearArgs {
  const int *g_tstart, *g_tcount;
  const double *tx, *ty, *tz;
  const long long *off, *moff;
  const int* cnt;
  const int* node;
  const unsigned* mask;
  const int *start, *nummemb;
  const double4* nodec;
  const void* src;  // double4 in tree order; mixed: records of two sources
  const double4* src64;
  const float4* nodeh;  // per node: half extents of the box, rounded up
  const double* sw;
  const SysEval* sys;  // per system: near_del, kappa, intg, near_sign, self_term, particles
  const int* g_sys;    // per group: system
  double *out, *out_y, *out_z;  // potential, or the three field components
  int* err;
  // mixed potentials: close pairs left out of the FP32 sums, per target (k_close)
  int* ccnt;    // tiles recorded for the target
  int2* crec;   // up to kCloseRec (near entry, first source of the tile) per target
  int2* clist;  // (target, group) of every target with a record
  int* cn;      // entries of clist
  int cap;               // mixed potentials: records of a tile at most (k_close)
  const int* pstart;     // first record of each leaf's FP32 sources
  const unsigned short* tgt;  // targets of each near entry
  const long long* pre;  // of every 32nd: work (near_weight x sources) of its group's before it
  const long long* tot;  // per group: work of all its entries
  const int* leaf_of;  // leaf of each sorted position
  const int2* items;   // (group, part | parts << 16)
  double* part;        // scratch of the groups in several parts, from part_off[g]
  const long long* part_off;
  int* part_done;      // parts of the group that are done
};

constexpr int kCloseRec = 2;  // record slots per target; beyond them k_close scans them all

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Knuth two-sum: s + e accumulates b with the rounding error of each step kept in e.
__device__ __forceinline__ void two_sum(float& s, float& e, float b) {
  float t = s + b;
  float bp = t - s;
  e += (s - (t - bp)) + (b - bp);
  s = t;
}

// Close pairs in the mixed path.  FP32 leaf-centred coordinates carry an absolute error of
// about 6e-8 of their magnitude, so a pair much closer than the leaf's size loses relative
// accuracy in its FP32 difference (two particles 1e-4 apart in a leaf of size 0.1 give
// ~1e-5).  Pairs closer than r_t = 1/32 of the source leaf's radius (r^2 below thr) are
// left out of the FP32 sum and summed in FP64 from the FP64 sources instead, with the
// reference's rules (including its r^2 <= 1e-14 skip, which only such pairs can meet:
// thr >= 2e-14).  Every other pair keeps at most ~4e-6 relative error, far below 1e-6 of a
// target's total.  Close pairs can only occur where a target lies within r_t of the source
// leaf's box (its own leaf, or a neighbour's boundary), and only where the kernel's del is
// below thr (FP32 r^2 >= del).  Everywhere else a warp runs the plain loop, with no test at all;
// near the box the potentials' warps watch the least r^2 and take the tile again, testing every
// pair, where a close one was met (tile32), and the fields' test every pair at once.
constexpr float kCloseFrac = 1.0f / 1024.0f;  // (1/32)^2
constexpr float kThrMin = 2e-14f;             // above the 1e-14 skip of src/constants.h:35
// r_t^2 of a leaf of squared radius sqradius
__host__ __device__ __forceinline__ float near_close_thr(double sqradius) {
  return fmaxf((float)sqradius * kCloseFrac, kThrMin);
}

// Squared distance from a point (relative to a leaf's centre) to the leaf's box (half
// extents h, rounded up); 0 inside.
__device__ __forceinline__ float box_d2(float x, float y, float z, float4 h) {
  const float dx = fmaxf(fabsf(x) - h.x, 0.f), dy = fmaxf(fabsf(y) - h.y, 0.f),
              dz = fmaxf(fabsf(z) - h.z, 0.f);
  return dx * dx + dy * dy + dz * dz;
}

// FP32 r^2 of a pair (identical wherever it is formed, so the FP32 and FP64 sums split the
// pairs exactly).
__device__ __forceinline__ float r2_32(float xt, float yt, float zt, float4 s, float del) {
  const float dx = s.x - xt, dy = s.y - yt, dz = s.z - zt;
  return fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, del)));
}

// Target t left close pairs of near entry e, in the tile that begins at source toff, out of its
// FP32 sum.  Several warps may record for a target; k_close puts the records in order.
__device__ __forceinline__ void record_close(const NearArgs& a, int t, int g, long long e, int toff) {
  if (!a.ccnt) return;  // (null where no pair can be close)
  const int c = atomicAdd(&a.ccnt[t], 1);
  if (c < kCloseRec) a.crec[(long long)t * kCloseRec + c] = make_int2((int)e, toff);
  if (c == 0) a.clist[atomicAdd(a.cn, 1)] = make_int2(t, g);
}

constexpr int kRec = 32;               // bytes of a source record: one FP64 source, two FP32 ones
constexpr int kSmemMax = 227 * 1024;  // shared memory of a CTA

// Pack the set bits of a group mask (W words, lane l holds word l) into tl in ascending order.
__device__ __forceinline__ void pack_list(unsigned wd, int W, unsigned short* tl) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  int base = 0;
  for (int j = 0; j < W; j++) {
    const unsigned b = __shfl_sync(0xffffffffu, wd, j);
    if ((b >> lane) & 1u) tl[base + __popc(b & lt)] = (unsigned short)(32 * j + lane);
    base += __popc(b);
  }
  __syncwarp();
}

// -------------------------------------------------------------------------------- FP64 pair
// One pair's q / sqrt(r^2 + del) or q e^(-kappa R) / R (src/tree3d.cpp:4765-4769, 3609-3618)
// added to acc.  1/R: the hardware seed rsqrt.approx.ftz.f64 and one third-order Newton step,
// y (1 + e/2 + 3 e^2 / 8) with e = 1 - x y^2, which takes a seed error e0 to about (5/16) e0^3; the
// exponential: exp_scaled.  12 (Coulomb) / 25 (screened) FP64 operations.  EPS: a pair with
// r^2 <= 1e-14 adds nothing; SELF: nor does the target's own source (`own`); both are evaluated
// with charge 0 at R = 1.  UF: the exponential may underflow; without, kappa R of every pair and
// kappa itself are below kExpNoUnderflow (SysEval::underflow).
template <int KER, bool EPS, bool SELF, bool UF, int COPIES = kExpTabCopies>
__device__ __forceinline__ void pair64(double x, double y, double z, double4 s, double del,
                                       ExpScale k, const double2* tab, bool own, double& acc) {
  const double dx = x - s.x, dy = y - s.y, dz = z - s.z;
  double rr = fma(dx, dx, fma(dy, dy, fma(dz, dz, del)));
  double q = s.w;
  if (EPS || SELF) {
    const bool skip = (SELF && own) || (EPS && !(rr > kEpsNear));
    q = skip ? 0.0 : q;
    rr = skip ? 1.0 : rr;
  }
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(rr));
  const double t = rr * y0;
  const double e = fma(-t, y0, 1.0);
  const double f = fma(e, 0.375, 0.5);
  if (KER == BIT_KERNEL_COULOMB) {
    acc = fma(q * y0, fma(e, f, 1.0), acc);
  } else {
    const double ec = e * f;
    const double ri = fma(y0, ec, y0);
    acc = fma(q * exp_scaled<UF, COPIES>(fma(t, ec, t), k, tab), ri, acc);
  }
}

struct Range64 {
  const double4* src;  // the tile
  int n;               // its sources
  double del;
  ExpScale k;
  const double2* tab;
};

// Two targets against every source of the tile, two sources (four pairs) at a time; o0, o1:
// the targets' own tile index (SELF).  (Four sources: 3% faster at 2M, 20% slower on leaves
// of 55.)
template <int KER, bool EPS, bool SELF, bool UF>
__device__ __forceinline__ void two64(const Range64& r, double x0, double y0, double z0, double x1,
                                      double y1, double z1, int o0, int o1, double& p0, double& p1) {
  constexpr int UN = 2;
  double a0[UN], a1[UN];
#pragma unroll
  for (int u = 0; u < UN; u++) a0[u] = a1[u] = 0.0;
  auto add = [&](int j, int u) {
    const double4 s = r.src[j];
    pair64<KER, EPS, SELF, UF>(x0, y0, z0, s, r.del, r.k, r.tab, j == o0, a0[u]);
    pair64<KER, EPS, SELF, UF>(x1, y1, z1, s, r.del, r.k, r.tab, j == o1, a1[u]);
  };
  int j = 0;
#pragma unroll 1
  for (; j + UN - 1 < r.n; j += UN) {
#pragma unroll
    for (int u = 0; u < UN; u++) add(j + u, u);
  }
#pragma unroll 1
  for (; j < r.n; j++) add(j, 0);
  p0 = a0[0] + a0[1];
  p1 = a1[0] + a1[1];
}

// One target against sources j, j + step, ... of the tile.
template <int KER, bool EPS, bool SELF, bool UF>
__device__ __forceinline__ double one64(const Range64& r, double x, double y, double z, int o, int j,
                                        int step) {
  constexpr int UN = 4;
  double a[UN] = {0.0, 0.0, 0.0, 0.0};
  auto add = [&](int k, int u) {
    pair64<KER, EPS, SELF, UF>(x, y, z, r.src[k], r.del, r.k, r.tab, k == o, a[u]);
  };
#pragma unroll 1
  for (; j + (UN - 1) * step < r.n; j += UN * step) {
#pragma unroll
    for (int u = 0; u < UN; u++) add(j + u * step, u);
  }
#pragma unroll 1
  for (; j < r.n; j += step) add(j, 0);
  return (a[0] + a[2]) + (a[1] + a[3]);
}

// Two FP32 numbers in one 64-bit register (packed arithmetic: one issue slot for two).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 v;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}

// A value that all lanes of the warp hold, in a form whose uniformity the compiler sees: loops and
// addresses that follow from it stay in uniform registers (k_far<9, 1, float> at 100k, theta 0.15: 230
// us with its first entry from a plain load, 218 so).
__device__ __forceinline__ int warp_uniform(int v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ long long warp_uniform(long long v) {
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)v), hi = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32));
  return (long long)((unsigned long long)hi << 32 | lo);
}

// First source (a multiple of 8, or all ns) of an entry of weight wt that lies d or more into its
// work.
__device__ __forceinline__ int cut(long long d, int wt, int ns) {
  if (d <= 0) return 0;
  if (d >= (long long)wt * ns) return ns;
  const long long j = (d + 8LL * wt - 1) / (8LL * wt) * 8;
  return j < ns ? (int)j : ns;
}

// Where warp v of nv begins its run of a group's work.
__device__ __forceinline__ long long run_begin(long long tot, int nv, int v) {
  return tot / nv * v + tot % nv * v / nv;
}
// The entry of a group's [e0, e1) that work T lies in: the last that begins at T or before (e1 if
// there is no entry: a group may have none); P: where it begins.  pre: where the work of every
// 32nd entry of the list begins (kept for those alone, and counts in 16 bits: a list of small
// leaves at a small theta is most of a request's memory); work: an entry's.  By a whole warp.
template <class Work>
__device__ __forceinline__ long long run_entry(const long long* pre, long long e0, long long e1, long long T,
                                               Work work, long long& P) {
  const int lane = threadIdx.x & 31;
  P = 0;
  if (e0 >= e1) return e1;
  long long k = e0 >> 5, begin = 0;  // the block of 32 entries, and where it begins
  for (long long b = k + 1, last = (e1 - 1) >> 5; b <= last; b += 32) {
    const long long at = b + lane <= last ? pre[b + lane] : LLONG_MAX;
    const int c = __popc(__ballot_sync(0xffffffffu, at <= T));
    if (c) begin = __shfl_sync(0xffffffffu, at, c - 1);
    k += c;
    if (c < 32) break;
  }
  const long long s = max(e0, k << 5);
  const bool in = s + lane < min(e1, (k + 1) << 5);
  const long long v = in ? work(s + lane) : 0;
  long long inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const long long t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  const int n = __popc(__ballot_sync(0xffffffffu, in && begin + inc - v <= T));
  P = warp_uniform(begin + __shfl_sync(0xffffffffu, inc - v, n - 1));
  return s + n - 1;
}
// A group's near entry: its work.
__device__ __forceinline__ long long near_work(const NearArgs& a, long long e) {
  return (long long)near_weight(a.tgt[e]) * a.nummemb[a.node[e]];
}

// The parts' scratch of `count` sums, or whether the parts are taken in turn for want of room: it is
// asked for last, so that nothing an evaluation cannot do without is short of it.
bool parts_in_turn(Ctx* c, Lists* L, DBuf<double>& part, size_t count);
// The arguments common to every near-field launch of this plan (near_field.cu).
NearArgs near_args(Tree* t, Lists* L, const EvalPlan& P, const double* tx, const double* ty,
                   const double* tz);

}  // namespace bit
