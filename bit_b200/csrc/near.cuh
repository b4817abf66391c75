// What the near-field kernels of the potentials (near.cu) and the fields (near_field.cu) share.
#pragma once

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
  const int *order, *g_tstart, *g_tcount;
  const double *tx, *ty, *tz;
  const long long *off, *moff;
  const int* cnt;
  const int* node;
  const unsigned* mask;
  const int *start, *nummemb;
  const double4* nodec;
  const void* src;  // double4 in tree order; mixed: float4 (fields), records of two sources (potentials)
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
  int tile;     // sources per tile
  int split;    // fields: threads per target, 0 the rule, else at most this many
  // potentials
  const int* pstart;     // first record of each leaf's FP32 sources
  const int* tgt;        // targets of each near entry
  const long long* pre;  // work (near_weight x sources) of the group's entries before it
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
// below thr (FP32 r^2 >= del), so a warp runs the checked loop on those tiles and the plain
// loop, with no test at all, everywhere else.
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

// The arguments common to every near-field launch of this plan (near_field.cu).
NearArgs near_args(Tree* t, Lists* L, const EvalPlan& P, const double* tx, const double* ty,
                   const double* tz);

}  // namespace bit
