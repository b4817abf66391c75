// Far field: Taylor expansion about every accepted cluster (treetaylorpotential,
// shielded_treetaylorpot, treetaylorforce; src/tree3d.cpp:4468-4640, 3004-3227, 456-810),
// one CTA per target group.
//
// Potentials: the reference's Taylor polynomial regrouped in solid harmonics
// (gen_harmonics.py), the same value to rounding.  k_far_coefs turns every node's Cartesian
// moments into the coefficients of the evaluation's kernel and parameters.  The CTA's warps
// then take the group's far entries, each a contiguous run.  A warp packs the targets of its
// entry (the set bits of the entry's mask) into a dense list while a TMA bulk copy brings
// the cluster's coefficients (a padded block, no multicast) into the warp's shared-memory
// slot, and its lanes run the unrolled evaluation for one target each, against those
// coefficients (warp-uniform loads).  Each warp accumulates into its own shared-memory row;
// rows are summed in warp order at the end, so the result does not depend on timing.  The
// target-centre offset is formed in FP64; the mixed path rounds it once to FP32 and runs
// the evaluation in FP32, accumulating with two-sum.
//
// Fields: the gradients of the same polynomials (k_far_field); with a kernel order, the
// reference's recurrences (gen_farfield.py) on the moments themselves.
#include <algorithm>

#include "common.cuh"
#include "near.cuh"
#include "tma.cuh"

namespace bit {
// Precision-generic math used by the generated recurrences.
__device__ __forceinline__ double sqrt_t(double x) { return sqrt(x); }
__device__ __forceinline__ float sqrt_t(float x) { return sqrtf(x); }
__device__ __forceinline__ double rsqrt_t(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }
__device__ __forceinline__ double exp_t(double x) { return exp(x); }
__device__ __forceinline__ float exp_t(float x) { return expf(x); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double pow_t(double a, double b) { return pow(a, b); }
__device__ __forceinline__ float pow_t(float a, float b) { return powf(a, b); }
template <class T>
struct V4 {
  T x, y, z, w;
};
// Four consecutive moments; M is 16-byte aligned.
__device__ __forceinline__ V4<float> ld4(const float* M, int q) {
  const float4 v = reinterpret_cast<const float4*>(M)[q];
  return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ V4<double> ld4(const double* M, int q) {
  const double2 a = reinterpret_cast<const double2*>(M)[2 * q];
  const double2 b = reinterpret_cast<const double2*>(M)[2 * q + 1];
  return {a.x, a.y, b.x, b.y};
}
}  // namespace bit

#include "generated/farfield_gen.cuh"
#include "generated/harmonics_gen.cuh"

namespace bit {

namespace {

struct FarArgs {
  const int *order, *g_tstart, *g_tcount;
  const double *tx, *ty, *tz;
  const long long *off, *moff;
  const int* cnt;
  const int* node;
  const unsigned* mask;
  const double4* nodec;
  const double* mom;         // T(nterms of the node's system) moments per node
  const long long* mom_off;  // first moment of each node
  const void* coef;          // float or double: every node's coefficients (potential kernels)
  int stride;                // elements from one node's coefficients to the next's
  int chunk;                 // targets of a CTA, at most
  int rows;                  // those of the largest chunk, rounded up to 32
  int* err;                  // device error flags (a bounded wait that gave up: 8)
  const unsigned short* tgt;  // targets of each far entry
  const int* cut;            // per group: first entry of each warp's share (group_shares)
  const SysEval* sys;        // per system: far_add, kappa, far_sign
  const int* g_sys;          // per group: system
  double *out, *out_y, *out_z;
};

template <class T>
struct WarpAcc;  // per-warp accumulator rows in shared memory
template <>
struct WarpAcc<float> {
  static constexpr int words = 2;  // hi, lo
  __device__ static void add(float* row, int rows, int i, float v) {
    float& s = row[i];
    float& e = row[rows + i];
    float t = s + v, bp = t - s;
    e += (s - (t - bp)) + (v - bp);
    s = t;
  }
  __device__ static double get(const float* row, int rows, int i) {
    return (double)row[i] + (double)row[rows + i];
  }
};
template <>
struct WarpAcc<double> {
  static constexpr int words = 1;
  __device__ static void add(double* row, int, int i, double v) { row[i] += v; }
  __device__ static double get(const double* row, int, int i) { return row[i]; }
};

constexpr int NWF = 4;  // warps per CTA, force (three accumulators)
// Warps per CTA, potentials.  Resident CTAs per SM: two at 128 registers, where every order's
// evaluation fits without spills; three (80 registers) up to nterms 6, whose leaves and
// entries are small in use, so that more warps cover the per-entry work.  Device time in us,
// two / three / four CTAs: FP64 screened, 2M clustered, nterms 9: 4116 / 4471 / 4748; mixed:
// 2585 / 2587 / 2889; 300k in leaves of 100, nterms 5, FP64: 791 / 635 / 619, mixed 663 / 514
// / 449 (at four, nterms 6 starts to spill).  A second slot per warp (the next entry's
// coefficients in flight during this one's evaluation) and two targets per lane were both
// within 1% or slower.
constexpr int NWP = kFarWarps;
constexpr int far_blocks(int nt) { return nt <= 6 ? 3 : 2; }

constexpr size_t force_smem(size_t moment_bytes) {
  return 3 * kGroupMax * sizeof(double) + NWF * kGroupMax * sizeof(unsigned short) +
         NWF * kGroupMax * 3 * sizeof(double) + NWF * moment_bytes;
}

// ---- coefficients of the potential kernels ------------------------------------------------

// Kind of a system's far field: bit 0 screened, bit 1 regularised (delta > 0).
constexpr int FAR_SCREENED = 1, FAR_REG = 2;

__host__ __device__ constexpr int far_count(int nt, int kind) {
  return kind & FAR_REG ? harm_count_reg(nt) : harm_count(nt);
}
// A node's block: its coefficients, then the scaling length H, padded to 16-byte TMA copies.
__host__ __device__ constexpr int far_block(int nt, int kind) {
  return (far_count(nt, kind) + 1 + 3) / 4 * 4;
}

// Exponent of H = 2^e, the smallest power of two above the cluster's radius and (regularised)
// sqrt(|delta|; a field's may be negative): the scaled evaluation then works with ratios H /
// distance of at most about one, powers of delta / H^2 stay in range, and scaling by H is exact.
// A cluster of coincident particles has moments of degree 0 only, and takes the lowest exponent.
__device__ __forceinline__ int far_scale_exp(double sqradius, double delta) {
  const double s = fmax(sqradius, fabs(delta));
  if (!(s > 0.0)) return -100;
  if (!(s < 1e300)) return 100;
  const int e = ilogb(sqrt(s)) + 1;
  return e < -100 ? -100 : (e > 100 ? 100 : e);
}

// Canonical moment index t (i outer, j, k inner, i + j + k < nt) to shell order: by degree
// d, then i, then j descending.
__device__ int canon_shell_pos(int t, int nt, int& d) {
  int i = 0, j = 0;
  for (; t >= (nt - i) * (nt - i + 1) / 2; i++) t -= (nt - i) * (nt - i + 1) / 2;
  for (; t >= nt - i - j; j++) t -= nt - i - j;
  d = i + j + t;
  return d * (d + 1) * (d + 2) / 6 + (d - i) * (d - i + 1) / 2 + (d - i - j);
}

// One CTA per node: moments -> harmonic moments -> the coefficients of the node's system
// (gen_harmonics.py), all in FP64, stored once as T.  Every value is a short fixed sum, so
// the kernel is bound by latency; 2M clustered (4,319 nodes, nterms 9): 26 us a launch.
constexpr int kCoefThreads = 128;
template <class T>
__global__ void __launch_bounds__(kCoefThreads)
    k_far_coefs(const int* node_sys, const SysEval* sys, const double4* nodec, const double* mom,
                const long long* mom_off, T* coef, int stride) {
  constexpr int TMAX = num_terms(kNtermsMax);
  constexpr int KMAX = (kNtermsMax - 1) / 2 + 1;
  __shared__ double s_m[TMAX], s_a[TMAX];
  __shared__ double s_e[KMAX][2 * KMAX];  // lap^k f = sum_s s_e[k][s] E_s, scaled by H^2(k-s)
  const int node = blockIdx.x;
  const SysEval* se = sys + node_sys[node];
  const int nt = se->nterms, kind = se->far_kind;
  const int nm = num_terms(nt), cnt = far_count(nt, kind);
  // (an FP32 distance overflows past 3.4e38, where the potential is 0: keep H and the
  // coefficients finite)
  const double delta = kind & FAR_REG ? (sizeof(T) == 4 ? fmin(se->far_add, 3e38) : se->far_add) : 0.0;
  const int he = far_scale_exp(nodec[node].w, delta);
  const double* M = mom + mom_off[node];
  for (int t = threadIdx.x; t < nm; t += kCoefThreads) {
    int d;
    const int p = canon_shell_pos(t, nt, d);
    s_m[p] = ldexp(M[t], -he * d);
  }
  if (threadIdx.x == 0) {
    // (kappa H is held where its powers stay in range: past 2^13 every accepted pair's exponential
    // is 0 in FP32, past 2^100 in FP64, and a coefficient of infinity would make the 0 a NaN)
    const double cap = sizeof(T) == 4 ? 0x1p13 : 0x1p100;
    const double kh = kind & FAR_SCREENED ? fmin(fabs(ldexp(se->kappa, he)), cap) : 0.0;
    const double k2 = kh * kh, dd = ldexp(delta, -2 * he);
    for (int k = 0; k < KMAX; k++)
      for (int s = 0; s < 2 * KMAX; s++) s_e[k][s] = 0.0;
    s_e[0][0] = 1.0;
    for (int k = 0; k + 1 < KMAX; k++)
      for (int s = 0; s <= 2 * k; s++) {
        const double v = s_e[k][s];
        s_e[k + 1][s] += k2 * v;
        s_e[k + 1][s + 1] += 2 * s * v;
        s_e[k + 1][s + 2] -= dd * v;
      }
  }
  __syncthreads();
  for (int h = threadIdx.x; h < nm; h += kCoefThreads) {
    double a = 0.0;
    for (int e = kHarmBegin[h]; e < kHarmBegin[h + 1]; e++)
      a = fma(kHarmFactor[e], s_m[kHarmShell[e]], a);
    s_a[h] = a;
  }
  __syncthreads();
  const HarmCoef* hc = kHarmCoef + (kind & FAR_REG ? kHarmCoefBeginReg[nt] : kHarmCoefBegin[nt]);
  T* C = coef + (long long)node * stride;
  for (int p = threadIdx.x; p < far_block(nt, kind); p += kCoefThreads) {
    double v = 0.0;
    if (p < cnt) {
      const HarmCoef q = hc[p];
      for (int k = (q.s + 1) / 2; q.l + 2 * k < nt; k++)
        v = fma(s_e[k][q.s], s_a[harm_index(q.l, q.m, q.part, k)], v);
      for (int j = 3; j < 2 * (q.l + q.s); j += 2) v *= j;  // (2(l + s) - 1)!!
    } else if (p == cnt) {
      v = ldexp(1.0, he);
    }
    C[p] = (T)v;
  }
}

// The far field of one target group g (the CTA's whole work for that group).  Bound by the
// FP64 / FP32 pipe and issue: 244 instructions a pair (nterms 9, screened) where the
// reference's recurrence took 1,333 (FP64) and 1,118 (FP32); 324 against 738 and 683 with
// delta > 0.  2M clustered, theta = 0.7, 181 M pairs, before / now: FP64 screened 17.2 / 4.1
// ms, Coulomb (delta = 0.005) 11.0 / 5.4, screened regularised 17.2 / 7.0; mixed 9.1 / 2.6,
// 6.1 / 3.2, 9.1 / 4.2; mixed against FP64 (relative L2, screened) 1.91e-7 / 1.78e-7.
// Shared memory: per warp an accumulator row, one cluster's coefficients and a packed target list
// (a kernel running several orders sizes the coefficients for the largest).  bar: one
// mbarrier per warp, phase: this warp's count of its completed copies.  Returns false (in
// every thread) if a warp's bounded wait for its coefficients gave up: the error flag is
// set, the warp has waited (bounded again) for that copy, and the group's result is not
// valid.
template <int NT, int KIND, class T, int NW>
__device__ __forceinline__ bool far_group(const FarArgs& a, int g, int c0, uint64_t* bar, unsigned& phase) {
  constexpr int CNT = far_count(NT, KIND);
  constexpr int TP = far_block(NT, KIND);
  extern __shared__ __align__(16) unsigned char sm[];
  const int rows = a.rows;
  const int ROW = WarpAcc<T>::words * rows;
  T* msb = reinterpret_cast<T*>(sm);  // per warp a slot of a.stride elements
  T* accb = msb + NW * a.stride;
  unsigned short* tlb = reinterpret_cast<unsigned short*>(accb + NW * ROW);

  const int gc = a.g_tcount[g], t0 = a.g_tstart[g] + c0, tc = min(gc - c0, a.chunk);
  const int W = (gc + 31) >> 5, w0 = c0 >> 5, wn = (tc + 31) >> 5;  // words of the group, the chunk
  const long long e0 = a.off[g], e1 = e0 + a.cnt[g], m0 = a.moff[g];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const double *cx = a.tx + t0, *cy = a.ty + t0, *cz = a.tz + t0;
  for (int i = tid; i < NW * ROW; i += 32 * NW) accb[i] = T(0);
  unsigned short* tl = tlb + w * rows;
  T* row = accb + w * ROW;
  T* M = msb + w * a.stride;
  const T* coef = reinterpret_cast<const T*>(a.coef);
  const SysEval* se = a.sys + a.g_sys[g];
  const T tadd = (T)se->far_add, tk = (T)se->kappa;
  const double sign = se->far_sign;
  bool failed = false;
  // Each warp takes a contiguous run of the group's entries holding about 1/NW of its
  // (target, cluster) pairs: the entries whose exclusive prefix P of target counts has
  // w C <= NW P < (w + 1) C, C the group's total (cut, from the list builder).  The entries' costs vary widely, so the
  // round-robin deal this replaces left warps idle at the group's closing barrier.  The
  // split depends on the lists only, so results stay deterministic.
  long long e = e0 + warp_uniform(a.cut[g * NW + w]);
  const long long ee = e0 + warp_uniform(w + 1 < NW ? a.cut[g * NW + w + 1] : (int)(e1 - e0));
  __syncthreads();  // the rows are zero
  for (; e < ee; e++) {
    const int node = a.node[e];
    // The cluster's coefficients, its whole block (TP values, 16-byte aligned in global and
    // shared memory), by one TMA bulk copy into the warp's slot while the warp packs the
    // entry's targets.  The previous entry's reads of the slot ended at the __syncwarp
    // closing its loop.
    if (lane == 0) {
      fence_proxy_async();
      mbar_expect_tx(&bar[w], TP * (unsigned)sizeof(T));
      tma_load_1d(M, coef + (long long)node * a.stride, TP * (unsigned)sizeof(T), &bar[w]);
    }
    const unsigned wd = lane < wn ? a.mask[m0 + (e - e0) * W + w0 + lane] : 0u;
    int cnt = a.tgt[e];
    const double4 c = a.nodec[node];
    const bool all = cnt == gc;  // a cluster accepted by the whole group needs no list
    if (all) cnt = tc;
    else {
      if (tc < gc) cnt = __reduce_add_sync(0xffffffffu, __popc(wd));
      pack_list(wd, wn, tl);
    }
    const bool landed = __all_sync(0xffffffffu, mbar_wait(&bar[w], phase & 1));
    phase++;
    if (!landed) {
      if (lane == 0) {
        atomicOr(a.err, 8);
        mbar_wait(&bar[w], (phase - 1) & 1);
      }
      __syncwarp();
      failed = true;
      break;
    }
    const T H = M[CNT];
    for (int r = lane; r < cnt; r += 32) {
      const int i = all ? r : tl[r];
      const T dx = (T)(cx[i] - c.x), dy = (T)(cy[i] - c.y), dz = (T)(cz[i] - c.z);
      const T r2 = dx * dx + dy * dy + dz * dz;
      T v;
      if constexpr (KIND == 0) v = Harmonics<NT>::template hc<T>(dx, dy, dz, r2, tadd, tk, H, M);
      else if constexpr (KIND == FAR_SCREENED) v = Harmonics<NT>::template hs<T>(dx, dy, dz, r2, tadd, tk, H, M);
      else if constexpr (KIND == FAR_REG) v = Harmonics<NT>::template rc<T>(dx, dy, dz, r2, tadd, tk, H, M);
      else v = Harmonics<NT>::template rs<T>(dx, dy, dz, r2, tadd, tk, H, M);
      WarpAcc<T>::add(row, rows, i, v);
    }
    __syncwarp();
  }
  if (__syncthreads_or(failed)) return false;
  for (int i = tid; i < tc; i += 32 * NW) {
    double s = 0.0;
    for (int q = 0; q < NW; q++) s += WarpAcc<T>::get(accb + q * ROW, rows, i);
    a.out[t0 + i] = sign * s;
  }
  return true;
}

// One mbarrier per warp for the coefficient copies, initialised before the kernel's first
// __syncthreads.
template <int NW>
__device__ __forceinline__ void far_bars_init(uint64_t* bar) {
  if (threadIdx.x == 0) {
    for (int k = 0; k < NW; k++) mbar_init(&bar[k], 1);
    fence_mbar_init();
  }
}

// One launch class: CTA (b, k) takes chunk k of group order[b].  A target's sum is the same
// whatever the chunks: its entries are shared out to the warps by the whole group's work.
template <int NT, int KIND, class T, int NW>
__global__ void __launch_bounds__(32 * NW, far_blocks(NT)) k_far(FarArgs a) {
  __shared__ uint64_t bar[NW];
  const int g = a.order[blockIdx.x], c0 = blockIdx.y * a.chunk;
  if (c0 >= a.g_tcount[g]) return;  // (the whole CTA)
  far_bars_init<NW>(bar);
  unsigned phase = 0;
  far_group<NT, KIND, T, NW>(a, g, c0, bar, phase);
}

// Persistent work queue over the groups of every class: each CTA takes the next item
// (a group, in the given order) from a device counter until none is left, and runs the
// far field of that group's system (its nterms and kernel) -- the same device code, in the
// same order within the group, as k_far, so the results are identical.  No CTA waits for
// another; the counter is the only shared state.
template <class T, int NW>
__global__ void __launch_bounds__(32 * NW, 2) k_far_queue(FarArgs a, int count, int* head) {
  __shared__ int s_item;
  __shared__ uint64_t bar[NW];
  far_bars_init<NW>(bar);
  unsigned phase = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(head, 1);
    __syncthreads();
    const int item = s_item;
    __syncthreads();  // every thread has read s_item before it is overwritten
    if (item >= count) return;
    const int g = a.order[item];
    const SysEval* se = a.sys + a.g_sys[g];
    bool ok = true;
    switch (se->nterms * 4 + se->far_kind) {
#define FK(N, K) \
  case 4 * N + K: ok = far_group<N, K, T, NW>(a, g, 0, bar, phase); break;
#define FQ(N) FK(N, 0) FK(N, 1) FK(N, 2) FK(N, 3)
      FQ(1) FQ(2) FQ(3) FQ(4) FQ(5) FQ(6) FQ(7) FQ(8) FQ(9) FQ(10)
#undef FQ
#undef FK
      default:
        break;
    }
    if (!ok) return;  // a bounded wait gave up (every thread saw it): take no more items
    __syncthreads();  // the group's last reads of shared memory precede the next group's writes
  }
}

// ---- fields -------------------------------------------------------------------------------

// Far field of the vector fields: the regularised Coulomb field of treetaylorforce (KIND 0 or
// FAR_REG) and the screened 2-D field of shielded_treetaylorforce (KIND FAR_SCREENED), as the
// gradients of the potentials' polynomials (gen_harmonics.py).  A CTA takes a chunk of a
// group's targets (32 to 256, Lists::field_chunk), so that the three rows of FP64 sums a warp keeps stay small: the
// recurrence kernel that this replaces had rows for a whole group of 1024, 130 KB, and so four
// warps a multiprocessor.  Entries are shared out to the warps as in far_group (by the work of
// the whole group), and rows are summed in warp order.  Bound by the FP64 / FP32 pipe: 1,252
// flops a pair (nterms 9, delta > 0) against the recurrence's 3,455.  Before / now, FP64 with delta,
// without, mixed, screened, ms: 2M clustered, nterms 9: 32.3 / 11.3, 32.2 / 7.3, 27.3 / 7.1, 41.8 /
// 10.3; 150k, 9: 1.14 / 0.44, 1.14 / 0.29, 0.99 / 0.29, 1.47 / 0.39; 20k, 6: 0.145 / 0.077, 0.144 /
// 0.070, 0.119 / 0.064, 0.152 / 0.082.  Mixed against FP64, 2M: 3.4e-7 / 1.9e-7.
// CTAs of eight warps per SM: two (128 registers) hold every order without spills; three (80)
// do up to nterms 4, 230 -> 198 us on 100k in leaves of 100, but cost 50k, nterms 7, 165 -> 183.
// (One CTA, 166 registers: 2M 13.3 ms.)
constexpr int field_blocks(int nt) { return nt <= 4 ? 3 : 2; }

template <int NT, int KIND, class T>
__global__ void __launch_bounds__(32 * NWP, field_blocks(NT)) k_far_field(FarArgs a) {
  constexpr int NW = NWP;
  constexpr int CNT = far_count(NT, KIND);
  constexpr int TP = far_block(NT, KIND);
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ uint64_t bar[NW];
  const int g = a.order[blockIdx.x], c0 = blockIdx.y * a.chunk;
  const int t0 = a.g_tstart[g] + c0, gc = a.g_tcount[g], tc = min(gc - c0, a.chunk);
  if (tc <= 0) return;  // (the whole CTA)
  far_bars_init<NW>(bar);
  const int rows = a.rows;
  double* accb = reinterpret_cast<double*>(sm);  // [NW][3][rows]
  T* msb = reinterpret_cast<T*>(accb + NW * 3 * rows);
  unsigned short* tlb = reinterpret_cast<unsigned short*>(msb + NW * a.stride);
  const int W = (gc + 31) >> 5, w0 = c0 >> 5, wn = (tc + 31) >> 5;
  const long long e0 = a.off[g], e1 = e0 + a.cnt[g], m0 = a.moff[g];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const double *cx = a.tx + t0, *cy = a.ty + t0, *cz = a.tz + t0;
  for (int i = tid; i < NW * 3 * rows; i += 32 * NW) accb[i] = 0.0;
  double* row = accb + w * 3 * rows;
  T* M = msb + w * a.stride;
  unsigned short* tl = tlb + w * rows;
  const T* coef = reinterpret_cast<const T*>(a.coef);
  const SysEval* se = a.sys + a.g_sys[g];
  const T tadd = (T)se->far_add, tk = (T)se->kappa;
  long long e = e0 + warp_uniform(a.cut[g * NW + w]);
  const long long ee = e0 + warp_uniform(w + 1 < NW ? a.cut[g * NW + w + 1] : (int)(e1 - e0));
  __syncthreads();  // the rows are zero, the barriers ready
  bool failed = false;
  unsigned phase = 0;
  for (; e < ee; e++) {
    const int node = a.node[e];
    if (lane == 0) {
      fence_proxy_async();
      mbar_expect_tx(&bar[w], TP * (unsigned)sizeof(T));
      tma_load_1d(M, coef + (long long)node * a.stride, TP * (unsigned)sizeof(T), &bar[w]);
    }
    const unsigned wd = lane < wn ? a.mask[m0 + (e - e0) * W + w0 + lane] : 0u;
    const bool all = a.tgt[e] == gc;
    const int cnt = all ? tc : __reduce_add_sync(0xffffffffu, __popc(wd));
    const double4 c = a.nodec[node];
    if (!all && cnt) pack_list(wd, wn, tl);
    const bool landed = __all_sync(0xffffffffu, mbar_wait(&bar[w], phase & 1));
    phase++;
    if (!landed) {
      if (lane == 0) {
        atomicOr(a.err, 8);
        mbar_wait(&bar[w], (phase - 1) & 1);
      }
      __syncwarp();
      failed = true;
      break;
    }
    const T H = M[CNT];
    for (int r = lane; r < cnt; r += 32) {
      const int i = all ? r : tl[r];
      const T dx = (T)(cx[i] - c.x), dy = (T)(cy[i] - c.y), dz = (T)(cz[i] - c.z);
      const T r2 = dx * dx + dy * dy + dz * dz;
      T fx, fy, fz;
      if constexpr (KIND == 0) Harmonics<NT>::template ghc<T>(dx, dy, dz, r2, tadd, tk, H, M, fx, fy, fz);
      else if constexpr (KIND == FAR_REG) Harmonics<NT>::template grc<T>(dx, dy, dz, r2, tadd, tk, H, M, fx, fy, fz);
      else Harmonics<NT>::template ghs<T>(dx, dy, dz, r2, tadd, tk, H, M, fx, fy, fz);
      if constexpr (KIND == FAR_SCREENED) {  // the curl: (d phi / dy, -d phi / dx)
        row[i] -= (double)fy;
        row[rows + i] += (double)fx;
      } else {
        row[i] += (double)fx;
        row[rows + i] += (double)fy;
        row[2 * rows + i] += (double)fz;
      }
    }
    __syncwarp();
  }
  if (__syncthreads_or(failed)) return;
  for (int i = tid; i < tc; i += 32 * NW) {
    double sx = 0, sy = 0, sz = 0;
    for (int q = 0; q < NW; q++) {
      sx += accb[(q * 3 + 0) * rows + i];
      sy += accb[(q * 3 + 1) * rows + i];
      sz += accb[(q * 3 + 2) * rows + i];
    }
    a.out[t0 + i] = sx;
    a.out_y[t0 + i] = sy;
    a.out_z[t0 + i] = sz;
  }
}

// The regularised Coulomb field with the systems' kernel orders (FP64): the reference's
// recurrences (gen_farfield.py) on the moments themselves.
template <int NT>
__global__ void __launch_bounds__(32 * NWF) k_far_force_korder(FarArgs a) {
  using T = double;
  constexpr int TT = num_terms(NT);
  constexpr int TP = FarField<NT>::kPadded;
  constexpr int NW = NWF;
  extern __shared__ __align__(16) unsigned char sm[];
  double* cx = reinterpret_cast<double*>(sm);
  double* cy = cx + kGroupMax;
  double* cz = cy + kGroupMax;
  unsigned short* tlb = reinterpret_cast<unsigned short*>(cz + kGroupMax);
  double* accb = reinterpret_cast<double*>(tlb + NW * kGroupMax);  // [NW][3][kGroupMax]
  T* msb = reinterpret_cast<T*>(accb + NW * 3 * kGroupMax);         // moments, one per warp

  const int g = a.order[blockIdx.x];
  const int t0 = a.g_tstart[g], tc = a.g_tcount[g];
  const int W = (tc + 31) >> 5;
  const long long e0 = a.off[g], e1 = e0 + a.cnt[g], m0 = a.moff[g];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int i = tid; i < tc; i += 32 * NW) {
    cx[i] = a.tx[t0 + i]; cy[i] = a.ty[t0 + i]; cz[i] = a.tz[t0 + i];
  }
  for (int i = tid; i < NW * 3 * kGroupMax; i += 32 * NW) accb[i] = 0.0;
  __syncthreads();
  unsigned short* tl = tlb + w * kGroupMax;
  double* row = accb + w * 3 * kGroupMax;
  const SysEval* se = a.sys + a.g_sys[g];
  const T tadd = (T)se->far_add, tdel = (T)se->near_del;
  const int korder = se->kernel_order;
  for (long long e = e0 + w; e < e1; e += NW) {
    const unsigned wd = lane < W ? a.mask[m0 + (e - e0) * W + lane] : 0u;
    const int cnt = __reduce_add_sync(0xffffffffu, __popc(wd));
    pack_list(wd, W, tl);
    const int node = a.node[e];
    const double4 c = a.nodec[node];
    T* M = msb + w * TP;
    const double* mn = a.mom + a.mom_off[node];
    for (int k = lane; k < TP; k += 32) M[k] = k < TT ? (T)mn[FarField<NT>::canon(k)] : T(0);
    __syncwarp();
    for (int r = lane; r < cnt; r += 32) {
      const int i = tl[r];
      const T dx = (T)(cx[i] - c.x), dy = (T)(cy[i] - c.y), dz = (T)(cz[i] - c.z);
      const T rs = dx * dx + dy * dy + dz * dz + tadd;
      T fx = 0, fy = 0, fz = 0;
      FarField<NT>::template force_korder<T>(dx, dy, dz, rs, tdel, korder, M, fx, fy, fz);
      row[i] += (double)fx;
      row[kGroupMax + i] += (double)fy;
      row[2 * kGroupMax + i] += (double)fz;
    }
    __syncwarp();
  }
  __syncthreads();
  for (int i = tid; i < tc; i += 32 * NW) {
    double sx = 0, sy = 0, sz = 0;
    for (int q = 0; q < NW; q++) {
      sx += accb[q * 3 * kGroupMax + i];
      sy += accb[q * 3 * kGroupMax + kGroupMax + i];
      sz += accb[q * 3 * kGroupMax + 2 * kGroupMax + i];
    }
    a.out[t0 + i] = sx;
    a.out_y[t0 + i] = sy;
    a.out_z[t0 + i] = sz;
  }
}

template <class K>
void set_smem(K kernel, size_t bytes) {
  ensure_smem_attr(reinterpret_cast<const void*>(kernel), (int)bytes);
}

template <class T, int NW>
size_t far_smem(const FarArgs& a) {
  return NW * ((size_t)a.stride * sizeof(T) + (size_t)a.rows * (WarpAcc<T>::words * sizeof(T) + sizeof(unsigned short)));
}
constexpr size_t kFarSmemMax =
    NWP * ((far_block(kNtermsMax, FAR_REG) + kGroupMax) * sizeof(double) + kGroupMax * sizeof(unsigned short));

template <int NT, int KIND, class T, int NW>
void launch_far(const FarArgs& a, int ng, int chunks, cudaStream_t s) {
  set_smem(k_far<NT, KIND, T, NW>, kFarSmemMax);
  count_launch(), k_far<NT, KIND, T, NW><<<dim3(ng, chunks), 32 * NW, far_smem<T, NW>(a), s>>>(a);
}

template <int NT>
void launch_korder(const FarArgs& a, int ng, cudaStream_t s) {
  const size_t bytes = force_smem(FarField<NT>::kPadded * sizeof(double));
  set_smem(k_far_force_korder<NT>, bytes);
  count_launch(), k_far_force_korder<NT><<<ng, 32 * NWF, bytes, s>>>(a);
}

template <class T>
constexpr size_t field_smem(int stride, int rows) {
  return NWP * (3 * (size_t)rows * sizeof(double) + (size_t)stride * sizeof(T) + (size_t)rows * sizeof(unsigned short));
}

template <int NT, int KIND, class T>
void launch_field(const FarArgs& a, int ng, int chunks, cudaStream_t s) {
  set_smem(k_far_field<NT, KIND, T>, field_smem<double>(far_block(kNtermsMax, FAR_REG), kFieldChunk));
  count_launch(), k_far_field<NT, KIND, T><<<dim3(ng, chunks), 32 * NWP, field_smem<T>(a.stride, a.rows), s>>>(a);
}

FarArgs far_args(Tree* t, Lists* L, const EvalPlan& P, const double* tx, const double* ty,
                 const double* tz) {
  FarArgs a{};
  a.g_tstart = L->g_tstart.p;
  a.g_tcount = L->g_tcount.p;
  a.tx = tx; a.ty = ty; a.tz = tz;
  a.off = L->far_off.p;
  a.cnt = L->far_cnt.p;
  a.moff = L->far_moff.p;
  a.node = L->far_node.p;
  a.mask = L->far_mask.p;
  a.nodec = t->nodec.p;
  a.mom = t->mom64.p;
  a.mom_off = t->mom_off.p;
  a.err = t->ctx->dev_err();
  a.tgt = L->far_tgt.p;
  a.cut = L->far_cut.p;
  a.sys = P.sys.p;
  a.g_sys = L->g_sys.p;
  return a;
}

}  // namespace

template <class T, int NW>
void launch_far_queue(Ctx* c, const FarArgs& a, int count, int* head, cudaStream_t s) {
  const size_t bytes = far_smem<T, NW>(a);
  set_smem(k_far_queue<T, NW>, kFarSmemMax);
  int per_sm = 0;
  BIT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_far_queue<T, NW>, 32 * NW, bytes));
  const int grid = std::max(1, std::min(count, c->num_sms * std::max(per_sm, 1)));
  count_launch(), k_far_queue<T, NW><<<grid, 32 * NW, bytes, s>>>(a, count, head);
}

// Every node's coefficients for this plan's systems, at one stride (the largest system's
// block).  The buffer is sized in doubles whatever the precision, so that a tree evaluated
// in both (iterative refinement, whose matvecs are replayed as CUDA graphs on fixed
// buffers) keeps one buffer.
template <class T>
void far_coefs(Tree* t, const EvalPlan& P, FarArgs& a, cudaStream_t s) {
  a.stride = 0;
  for (const SysEval& se : P.h_sys) a.stride = std::max(a.stride, far_block(se.nterms, se.far_kind));
  t->far_coef.ensure(t->ctx, (size_t)a.stride * t->numtree);
  a.coef = t->far_coef.p;
  count_launch(), k_far_coefs<T><<<t->numtree, kCoefThreads, 0, s>>>(
      t->node_sys.p, P.sys.p, t->nodec.p, t->mom64.p, t->mom_off.p, reinterpret_cast<T*>(t->far_coef.p),
      a.stride);
  BIT_CHECK_LAUNCH();
}

// The work-queue form is used for plans of several classes when the context allows it;
// the queue takes every group in decreasing-work order (L->order).
bool use_queue(const Ctx* c, const std::vector<LaunchClass>& classes) {
  return c->work_queue && classes.size() > 1;
}

int* queue_head(Ctx* c, int which, cudaStream_t s) {
  c->queue_heads.ensure(c, 2);
  BIT_CUDA(cudaMemsetAsync(c->queue_heads.p + which, 0, sizeof(int), s));
  return c->queue_heads.p + which;
}

// One launch per (nterms, kind) class, each over its groups (P.far_ord + begin), or one
// work queue over them all.
void eval_far(Tree* t, Lists* L, const EvalPlan& P, const double* tx, const double* ty,
              const double* tz, double* out) {
  FarArgs a = far_args(t, L, P, tx, ty, tz);
  a.out = out;
  a.chunk = kGroupMax;
  a.rows = L->max_targets;
  cudaStream_t s = t->ctx->stream;
  const bool f32 = P.f32;
  if (f32) far_coefs<float>(t, P, a, s);
  else far_coefs<double>(t, P, a, s);
  if (use_queue(t->ctx, P.far_classes)) {
    int count = 0;
    for (const LaunchClass& k : P.far_classes) count += k.count;
    a.order = L->order.p;
    int* head = queue_head(t->ctx, 0, s);
    if (f32) launch_far_queue<float, NWP>(t->ctx, a, count, head, s);
    else launch_far_queue<double, NWP>(t->ctx, a, count, head, s);
    BIT_CHECK_LAUNCH();
    return;
  }
  a.chunk = L->far_chunk;
  a.rows = std::min(L->max_targets, a.chunk);
  const int chunks = (L->max_targets + a.chunk - 1) / a.chunk;
  for (const LaunchClass& k : P.far_classes) {
    a.order = P.far_ord + k.begin;
    const int ng = k.count;
    switch (k.nterms * 4 + k.kind) {
#define FK(N, K)                                             \
  case 4 * N + K:                                            \
    if (f32) launch_far<N, K, float, NWP>(a, ng, chunks, s);         \
    else launch_far<N, K, double, NWP>(a, ng, chunks, s);            \
    break;
#define CASE(N) FK(N, 0) FK(N, 1) FK(N, 2) FK(N, 3)
      CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10)
#undef CASE
#undef FK
      default:
        fail(BIT_ERR_STATE, "moments not computed");
    }
    BIT_CHECK_LAUNCH();
  }
}

void eval_far_force(Tree* t, Lists* L, const EvalPlan& P, double* fx, double* fy, double* fz) {
  FarArgs a = far_args(t, L, P, t->sx.p, t->sy.p, t->sz.p);
  a.out = fx; a.out_y = fy; a.out_z = fz;
  cudaStream_t s = t->ctx->stream;
  const bool f32 = P.f32;
  // field kind of the plan: 1 Coulomb (kernel order from each system), 2 screened curl
  const bool curl = P.force == 2;
  bool korder = false;
  for (const SysEval& se : P.h_sys) korder |= se.kernel_order > 0;
  if (f32 && (curl || korder)) fail(BIT_ERR_INVALID_ARGUMENT, "this field is FP64 only");
  if (!korder) {
    if (f32) far_coefs<float>(t, P, a, s);
    else far_coefs<double>(t, P, a, s);
  }
  a.chunk = L->field_chunk;
  a.rows = std::min(L->max_targets, a.chunk);
  const int chunks = (L->max_targets + a.chunk - 1) / a.chunk;
  for (const LaunchClass& k : P.far_classes) {
    a.order = P.far_ord + k.begin;
    const int ng = k.count;
    switch (k.nterms) {
#define CASE(N)                                                                            \
  case N:                                                                                  \
    if (korder) launch_korder<N>(a, ng, s);                                                \
    else if (curl) launch_field<N, FAR_SCREENED, double>(a, ng, chunks, s);                \
    else if (f32 && k.kind) launch_field<N, FAR_REG, float>(a, ng, chunks, s);             \
    else if (f32) launch_field<N, 0, float>(a, ng, chunks, s);                             \
    else if (k.kind) launch_field<N, FAR_REG, double>(a, ng, chunks, s);                   \
    else launch_field<N, 0, double>(a, ng, chunks, s);                                     \
    break;
      CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8) CASE(9) CASE(10)
#undef CASE
      default:
        fail(BIT_ERR_STATE, "moments not computed");
    }
    BIT_CHECK_LAUNCH();
  }
}

}  // namespace bit
