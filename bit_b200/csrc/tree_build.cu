// GPU tree build: the reference's aspect-ratio bisection tree (treemake,
// src/tree3d.cpp:1345-1551), level by level.
//
// Nodes of one level are consecutive indices [a, b); their children become [b, c) in
// parent order, which is the reference's breadth-first numbering.  Inside a node the
// reference runs a short sequential program of up to seven bisections (treedivide,
// src/tree3d.cpp:1163-1304), each needing the member count and bounding box of both
// halves of the slot it splits (min/max are order independent, so the result is exact).
//
// A node of up to 57,344 (114,688) members is one cluster's work (k_node_split: one to sixteen CTAs
// by its size): the members stay in shared memory through the whole program, and go to
// the children's ranges in one stable scatter, members in ascending original index (the
// reference's member order).  The level's last CTA scans the child counts, k_make_children
// appends the children and sorts out which of them are to be split, all from device-side
// level records, so the host launches four levels at a time and then looks.
//
// Larger nodes (the first levels of a large tree) are split by all SMs: a pass over all their
// members relabels by each node's last bisection and reduces counts and bounding boxes of the
// next (block reduction + atomics), and the CTA that finishes a node's last chunk takes the
// program's next step.  Members carry a slot label; a stable counting scatter follows.
//
// Field arithmetic (midpoints, aspect ratios, sqradius) is the reference's, with no FMA
// contraction.
//
// Bound by latency: launches, and in a node's CTA its scans and reductions, one bisection after
// the other.  With the passes for every node (18 launches and a round trip a level), before /
// now: 2k uniform in leaves of 50 744 / 172 us, 10k, 200: 693 / 183, 50k clustered, 300: 1,663 / 412,
// 100k, 500: 1,845 / 500, 200k, 500: 2,105 / 689, 2M, 1000: 4,149 / 2,130, 48 systems 1,279 / 535.  With
// one CTA up to 16,384 members that read them from L2 at every bisection: 10k 320, 100k 1,190.
// Doing the bisection in hand and a foreseen one in one pass (four passes for seven) gave
// nothing: a pass's own scan and reduction take the time, not its barriers.
#include <algorithm>
#include <climits>
#include <cstring>

#include <cooperative_groups.h>

#include "common.cuh"

namespace bit {

namespace {

namespace cg = cooperative_groups;

constexpr int CH = 2048;  // members per chunk (one block)
constexpr int TB = 256;   // threads per block
// Nodes that a cluster of CTAs splits with its members in shared memory, by size: one CTA of
// up to 3,584 members (two such CTAs an SM), four of those, eight or sixteen of 7,168.  Larger
// nodes take all SMs; so do those of the last class where larger ones are there to take along:
// it is used for trees and forests whose roots all fit it (a build of 100k clustered particles in
// leaves of 500 580 -> 500 us, of 48 systems of up to 100k 705 -> 535; with a larger root the
// passes are made in any case).
constexpr int kClasses = 4;
constexpr int kClassCtas[kClasses] = {1, 4, 8, 16};
constexpr int kClassRows[kClasses] = {7, 7, 14, 14};  // members of a thread
constexpr int ST = 512;                               // threads of a CTA
__host__ __device__ constexpr int class_members(int c) {
  return (c == 0 ? 1 : c == 1 ? 4 : c == 2 ? 8 : 16) * (c >= 2 ? 14 : 7) * ST;
}
static_assert(CH % TB == 0, "a chunk is a whole number of block strides");

__device__ __forceinline__ unsigned long long okey(double v) {
  long long b = __double_as_longlong(v);
  if (b == (long long)0x8000000000000000ULL) b = 0;  // -0.0 -> +0.0
  return b >= 0 ? ((unsigned long long)b | 0x8000000000000000ULL) : ~(unsigned long long)b;
}
__device__ __forceinline__ double okey_inv(unsigned long long k) {
  long long b = (k & 0x8000000000000000ULL) ? (long long)(k & 0x7FFFFFFFFFFFFFFFULL)
                                            : (long long)(~k);
  return __longlong_as_double(b);
}

// treeinit (src/tree3d.cpp:1045-1073)
__device__ void box_fields(double* f, double x0, double x1, double y0, double y1, double z0,
                           double z1) {
  double x = dmul(0.5, dadd(x1, x0)), y = dmul(0.5, dadd(y1, y0)), z = dmul(0.5, dadd(z1, z0));
  f[0] = x0; f[1] = x1; f[2] = y0; f[3] = y1; f[4] = z0; f[5] = z1;
  f[6] = x; f[7] = y; f[8] = z;
  f[9] = fabs(__ddiv_rn(dsub(x1, x0), dsub(y1, y0)));
  f[10] = fabs(__ddiv_rn(dsub(x1, x0), dsub(z1, z0)));
  f[11] = fabs(__ddiv_rn(dsub(y1, y0), dsub(z1, z0)));
  x = dsub(x1, x); y = dsub(y1, y); z = dsub(z1, z);
  f[12] = dadd(dadd(dmul(x, x), dmul(y, y)), dmul(z, z));
}

// box_fields by a warp, lanes 0..2 an axis and a quotient each; bb: smallest and (negated) largest
// coordinate of each axis.
__device__ void warp_box_fields(double* f, const double* bb) {
  const int lane = threadIdx.x & 31, a = lane < 3 ? lane : 0;
  const double lo = bb[2 * a], hi = -bb[2 * a + 1];
  const double mid = dmul(0.5, dadd(hi, lo)), ext = dsub(hi, lo), half = dsub(hi, mid), sq = dmul(half, half);
  const double ey = __shfl_sync(0xffffffffu, ext, 1), ez = __shfl_sync(0xffffffffu, ext, 2);
  const double ex = __shfl_sync(0xffffffffu, ext, 0);
  const double s1 = __shfl_sync(0xffffffffu, sq, 1), s2 = __shfl_sync(0xffffffffu, sq, 2);
  if (lane < 3) {
    f[2 * lane] = lo;
    f[2 * lane + 1] = hi;
    f[6 + lane] = mid;
    f[9 + lane] = fabs(__ddiv_rn(lane == 2 ? ey : ex, lane == 0 ? ey : ez));
    if (lane == 0) f[12] = dadd(dadd(sq, s1), s2);
  }
}

// What a split leaves for k_make_children: the child slots and the order of children[].
struct NodeOut {
  int nchild;
  int order[8], slot_n[8];
  double slot_f[8][13];
};

// One level of the tree, on the device (a ring of kLevels records).
constexpr int kLevels = 8;
struct Level {
  int a, b;            // its nodes
  int nact;            // nodes to split, numbered in no particular order
  int nsmall[kClasses], nbig;  // of those, by class
  int arrive;          // CTAs of the level's k_node_split launches that are done
};
struct Ctl {
  Level lv[kLevels];
  int cur;             // the first level whose children have not been made
  int stop;            // the node arrays are full: nothing runs until they have grown
  int err;             // 1 NaN, 2 a node that cannot be split, 4 / 8 consistency checks
};

// treemake's per-node program (src/tree3d.cpp:1412-1545), resumable at its bisections: slots
// are relative to the first free node index, order[] receives the children in recorded order.
struct Program {
  int pc, j, k, xc, yc, ind2, nchild, nchild2;
  int dir, src, c1, c2;  // the bisection to do: slot src (-1: the node) into c1 and c2
  int n[8], order[8];    // the slots' members
};

__device__ __forceinline__ void program_init(Program& g) {
  g.pc = g.nchild = g.nchild2 = 0;
  for (int s = 0; s < 8; s++) g.n[s] = 0;
}

// Go on after the bisection in hand, which made `made` non-empty halves (the first call: none
// in hand); P: the node's box, f: the slots' boxes.  True: the next bisection is in hand;
// false: the program is done.
__device__ bool program_next(Program& g, const double* P, const double (*f)[13], int made, double lim,
                             int maxmemb) {
  auto zsplit = [&](int s) { return f[s][10] < lim && f[s][11] < lim && g.n[s] > maxmemb; };
  auto bisect = [&](int pc, int dir, int src, int c1, int c2) {
    g.pc = pc; g.dir = dir; g.src = src; g.c1 = c1; g.c2 = c2;
    return true;
  };
  auto second = [&] {  // a second half is a child of its own
    if (made == 2) g.order[g.nchild++] = g.ind2++;
    return made == 2;
  };
  bool in_k = false;
  switch (g.pc) {
    case 0:
      if (P[9] > lim && P[10] > lim) return bisect(1, 0, -1, 0, 1);
      if (P[9] < lim && P[11] > lim) return bisect(5, 1, -1, 0, 1);
      return bisect(7, 2, -1, 0, 1);
    case 1:  // x done
    case 5:  // y done, no x
      g.xc = g.ind2 = made;
      g.j = 0;
      break;
    case 2:  // y of slot j done
      g.yc = made;
      second();
      g.k = 0;
      in_k = true;
      break;
    case 3:  // z of slot t done
      if (second()) g.nchild2++;
      g.k++;
      in_k = true;
      break;
    case 4:  // z of slot j done, no y
    case 6:
      second();
      g.j++;
      break;
    default:  // z only
      for (int j = 0; j < made; j++) g.order[g.nchild++] = j;
      return false;
  }
  if (g.pc >= 5) {
    for (; g.j < g.xc; g.j++) {
      g.order[g.nchild++] = g.j;
      if (zsplit(g.j)) return bisect(6, 2, g.j, g.j, g.ind2);
    }
    return false;
  }
  for (;;) {
    if (in_k) {
      for (; g.k < g.yc; g.k++) {
        // the reference's numtree+j+k*(nchild2+1) (src/tree3d.cpp:1460), as written
        const int t = g.j + g.k * (g.nchild2 + 1);
        if (t >= 8 || t >= g.ind2) continue;  // never-created slot: nummemb == 0
        if (zsplit(t)) return bisect(3, 2, t, t, g.ind2);
      }
      in_k = false;
      g.j++;
    }
    if (g.j >= g.xc) return false;
    g.order[g.nchild++] = g.j;
    if (f[g.j][9] < lim && f[g.j][11] > lim && g.n[g.j] > maxmemb) return bisect(2, 1, g.j, g.j, g.ind2);
    if (zsplit(g.j)) return bisect(4, 2, g.j, g.j, g.ind2);
    g.j++;
  }
}

// A large node's split: its program, and the bisections its next pass relabels by and reduces.
struct Divide {
  int dir, src, c1, c2;
  double mid;
};
struct SplitState {
  Program g;
  int has_cur, has_prev;
  Divide cur, prev;  // prev.c2: where the second half went
};

struct SplitAcc {
  int cnt[2];
  unsigned long long mn[2][3], mx[2][3];
};

__device__ void acc_reset(SplitAcc* a) {
  for (int h = 0; h < 2; h++) {
    a->cnt[h] = 0;
    for (int d = 0; d < 3; d++) { a->mn[h][d] = ~0ULL; a->mx[h][d] = 0ULL; }
  }
}

template <class T>
__device__ __forceinline__ T warp_min(T v) {
  for (int o = 16; o; o >>= 1) { T w = __shfl_xor_sync(0xffffffffu, v, o); v = w < v ? w : v; }
  return v;
}
template <class T>
__device__ __forceinline__ T warp_max(T v) {
  for (int o = 16; o; o >>= 1) { T w = __shfl_xor_sync(0xffffffffu, v, o); v = w > v ? w : v; }
  return v;
}
__device__ __forceinline__ int warp_sum(int v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The particles into tree order (the identity, to begin with) and the bounding box of each
// system's (its root, src/tree3d.cpp:1385-1403); flags NaNs.  grid.y = system, grid.x =
// blocks striding over that system.
__global__ void k_root_bbox(const int* sys_start, const int* sys_n, const double* x,
                            const double* y, const double* z, int* perm, double* sx, double* sy_,
                            double* sz, SplitAcc* acc, Ctl* ctl) {
  const int sy = blockIdx.y;
  const int i0 = sys_start[sy], i1 = i0 + sys_n[sy];
  unsigned long long mn[3] = {~0ULL, ~0ULL, ~0ULL}, mx[3] = {0, 0, 0};
  int bad = 0;
  for (int i = i0 + blockIdx.x * blockDim.x + threadIdx.x; i < i1; i += gridDim.x * blockDim.x) {
    double v[3] = {x[i], y[i], z[i]};
    perm[i] = i;
    sx[i] = v[0]; sy_[i] = v[1]; sz[i] = v[2];
    for (int d = 0; d < 3; d++) {
      if (isnan(v[d])) bad = 1;
      unsigned long long k = okey(v[d]);
      mn[d] = k < mn[d] ? k : mn[d];
      mx[d] = k > mx[d] ? k : mx[d];
    }
  }
  for (int d = 0; d < 3; d++) {
    mn[d] = warp_min(mn[d]);
    mx[d] = warp_max(mx[d]);
  }
  bad = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    for (int d = 0; d < 3; d++) {
      atomicMin(&acc[sy].mn[0][d], mn[d]);
      atomicMax(&acc[sy].mx[0][d], mx[d]);
    }
    if (bad) atomicOr(&ctl->err, 1);
  }
}

__global__ void k_acc_reset(SplitAcc* acc, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) acc_reset(&acc[i]);
}

// The lists of the nodes to split, by level parity.
struct Lists2 {
  int* small[kClasses][2];
  int* big[2];
};

// Node `node` of level lev (its record L) joins the list it belongs to; act: its number among
// the nodes to split, or -1; small: the largest node that a cluster takes.
__device__ __forceinline__ void enlist(int node, int cnt, int maxmemb, Level* L, int lev,
                                       const Lists2& ls, int* act, int* nch, int small) {
  nch[node] = 0;
  if (cnt <= maxmemb) {
    act[node] = -1;
    return;
  }
  act[node] = atomicAdd(&L->nact, 1);
  if (cnt > small) {
    ls.big[lev & 1][atomicAdd(&L->nbig, 1)] = node;
    return;
  }
  const int c = cnt <= class_members(0) ? 0 : cnt <= class_members(1) ? 1 : cnt <= class_members(2) ? 2 : 3;
  ls.small[c][lev & 1][atomicAdd(&L->nsmall[c], 1)] = node;
}

__global__ void k_root_init(int nsys, const int* sys_start, const int* sys_n, const int* sys_maxmemb,
                            const SplitAcc* acc, int* nummemb, int* start, int* children,
                            double* fields, int* node_sys, Ctl* ctl, Lists2 ls, int* act, int* nch, int small) {
  const int sy = blockIdx.x * blockDim.x + threadIdx.x;
  if (sy >= nsys) return;
  double f[13];
  const SplitAcc* A = &acc[sy];
  box_fields(f, okey_inv(A->mn[0][0]), okey_inv(A->mx[0][0]), okey_inv(A->mn[0][1]),
             okey_inv(A->mx[0][1]), okey_inv(A->mn[0][2]), okey_inv(A->mx[0][2]));
  for (int k = 0; k < 13; k++) fields[13LL * sy + k] = f[k];
  nummemb[sy] = sys_n[sy]; start[sy] = sys_start[sy];
  node_sys[sy] = sy;
  for (int c = 0; c < 8; c++) children[8LL * sy + c] = -1;
  if (sy == 0) ctl->lv[0].b = nsys;
  enlist(sy, sys_n[sy], sys_maxmemb[sy], &ctl->lv[0], 0, ls, act, nch, small);
}

struct Arrays {
  int *nummemb, *start, *children, *node_sys, *act, *nch, *cscan;
  double* fields;
  int* perm;
  double *sx, *sy, *sz;
  int* perm2;
  double *sx2, *sy2, *sz2;
  const int* sys_maxmemb;
  NodeOut* out;
  Ctl* ctl;
  Lists2 ls;
  double lim;
  int cap, small;
};

// ---- nodes of one cluster -------------------------------------------------------------------
constexpr int SW = ST / 32;  // warps of a CTA

struct NodeShared {
  Program g;
  double pf[13], f[8][13];      // the node's box, the slots'
  double red[SW][14];           // per warp: combine's values of both halves
  double part[2][14], all[14];  // the CTA's (by parity of the bisection), the node's
  int wcnt[SW][8], tot[8];      // members of each slot, per warp and in the CTA
  int made;
};

// Value v = 7 h + q of a bisection: q = 2 d the smallest coordinate of axis d in half h, 2 d + 1
// the largest's negative, 6 the count.
__device__ __forceinline__ double combine(int v, double a, double b) {
  return v % 7 == 6 ? a + b : (b < a ? b : a);
}
template <class T>
__device__ __forceinline__ void least(T& a, T b) { a = b < a ? b : a; }
// The warp's least of each of v[0..11], by halves: lane l is left with that of value
// 6 (l >> 4) + 3 (l >> 3 & 1) + (l >> 1 & 3) in v[0] (l >> 1 & 3 < 3).  13 exchanges, where twelve
// butterflies make 60, and the exchanges bounded a bisection.
template <class T>
__device__ __forceinline__ void warp_least12(T (&v)[12]) {
  const int lane = threadIdx.x & 31;
  auto halve = [&](int o, int n) {  // v[0..2n): the lanes of bit o keep the second n
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < 6; q++)
      if (q < n) {
        const T a = v[q], b = v[q + n], r = __shfl_xor_sync(0xffffffffu, up ? a : b, o);
        v[q] = up ? b : a;
        least(v[q], r);
      }
  };
  halve(16, 6);
  halve(8, 3);
  v[3] = v[2];
  halve(4, 2);
  halve(2, 1);
  least(v[0], __shfl_xor_sync(0xffffffffu, v[0], 1));
}

// Split every node of class C at level lev: a cluster of CTAs holds a node's members in shared
// memory, each thread its own (a warp a contiguous run), with the slot labels in nibbles of a
// register.  A bisection is a pass over the thread's members, a reduction over the warp, the
// CTA and (through distributed shared memory) the cluster, and one thread's step of the
// program, which every CTA takes for itself.  The members then go to the children's ranges in
// order, in place: all of them were read before any is written.  The level's last CTA, of the
// `total` of its launches, scans the child counts.
template <int C>
__global__ void __launch_bounds__(ST) k_node_split(Arrays A, int lev, int total) {
  constexpr int CS = kClassCtas[C], ROWS = kClassRows[C];
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ NodeShared N;
  __shared__ int s_last;
  double* xs = reinterpret_cast<double*>(sm);
  double* ys = xs + ROWS * ST;
  double* zs = ys + ROWS * ST;
  int* ps = reinterpret_cast<int*>(zs + ROWS * ST);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = CS > 1 ? (int)cluster.block_rank() : 0;
  Ctl* ctl = A.ctl;
  if (ctl->stop) return;
  Level* lv = &ctl->lv[lev % kLevels];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  const int count = lv->nsmall[C];  // (not ctl->err: a cluster's CTAs have to agree)
  int par = 0;
  for (int k = blockIdx.x / CS; k < count; k += gridDim.x / CS) {
    const int node = A.ls.small[C][lev & 1][k];
    const int s0 = A.start[node], cnt = A.nummemb[node], maxmemb = A.sys_maxmemb[A.node_sys[node]];
    if (tid < 13) N.pf[tid] = A.fields[13LL * node + tid];
    if (tid == 0) program_init(N.g);
    // this CTA's members, this warp's run of them
    const int per = (cnt + CS - 1) / CS;
    const int c0 = min(rank * per, cnt), c1 = min(c0 + per, cnt);
    const int run = (c1 - c0 + ST - 1) / ST * 32;
    const int r0 = min(c0 + w * run, c1), r1 = min(r0 + run, c1), rows = run / 32;
    for (int i = 0; i < rows; i++) {
      const int e = r0 + 32 * i + lane;
      if (e < r1) {
        ps[i * ST + tid] = A.perm[s0 + e];
        // + 0.0: a -0.0 enters the boxes as +0.0, as the large nodes' ordered keys have it
        xs[i * ST + tid] = A.sx[s0 + e];
        ys[i * ST + tid] = A.sy[s0 + e];
        zs[i * ST + tid] = A.sz[s0 + e];
      }
    }
    unsigned long long lab = ~0ULL;  // 15: the node itself
    __syncthreads();
    if (tid == 0) N.made = program_next(N.g, N.pf, N.f, 0, A.lim, maxmemb) ? 0 : -1;
    __syncthreads();
    while (N.made >= 0) {
      const int dir = N.g.dir, src = N.g.src;
      const double mid = (src < 0 ? N.pf : N.f[src])[6 + dir];
      const unsigned want = src < 0 ? 15u : (unsigned)src;
      double v[12];
#pragma unroll
      for (int q = 0; q < 12; q++) v[q] = inf;
      int n0 = 0, n1 = 0;
      unsigned up = 0;
      const double* cs = dir == 0 ? xs : (dir == 1 ? ys : zs);
      for (int i = 0; i < rows; i++) {
        if (r0 + 32 * i + lane >= r1 || ((unsigned)(lab >> (4 * i)) & 15u) != want) continue;
        const int o = i * ST + tid;
        const double x = xs[o] + 0.0, y = ys[o] + 0.0, z = zs[o] + 0.0;
        if (cs[o] <= mid) {
          n0++;
          least(v[0], x); least(v[1], -x); least(v[2], y); least(v[3], -y); least(v[4], z); least(v[5], -z);
        } else {
          up |= 1u << i;
          n1++;
          least(v[6], x); least(v[7], -x); least(v[8], y); least(v[9], -y); least(v[10], z); least(v[11], -z);
        }
      }
      n0 = __reduce_add_sync(0xffffffffu, n0);
      n1 = __reduce_add_sync(0xffffffffu, n1);
      warp_least12(v);
      if (!(lane & 1) && (lane & 6) != 6) N.red[w][7 * (lane >> 4) + 3 * ((lane >> 3) & 1) + (lane & 6) / 2] = v[0];
      if (lane == 0) N.red[w][6] = n0;
      if (lane == 16) N.red[w][13] = n1;
      __syncthreads();
      if (w < 14) {  // warp q: value q over the CTA's warps
        double x = N.red[lane & (SW - 1)][w];
#pragma unroll
        for (int o = SW / 2; o; o >>= 1) x = combine(w, x, __shfl_xor_sync(0xffffffffu, x, o));
        if (lane == 0) (CS > 1 ? N.part[par] : N.all)[w] = x;
      }
      if constexpr (CS > 1) {
        cluster.sync();
        if (w < 14) {
          double x = cluster.map_shared_rank(&N.part[par][0], lane & (CS - 1))[w];
#pragma unroll
          for (int o = CS / 2; o; o >>= 1) x = combine(w, x, __shfl_xor_sync(0xffffffffu, x, o));
          if (lane == 0) N.all[w] = x;
        }
        par ^= 1;  // (a CTA past the next barrier has read these values)
      }
      __syncthreads();
      const bool any0 = N.all[6] > 0.0, any1 = N.all[13] > 0.0;
      const int d0 = N.g.c1, d1 = any0 ? N.g.c2 : N.g.c1;
      __syncthreads();  // every thread has read the bisection in hand
      if (w < 2 && (w ? any1 : any0)) {  // a half's fields, one warp each, a lane an axis
        const int slot = w ? d1 : d0;
        warp_box_fields(N.f[slot], &N.all[7 * w]);
        if (lane == 0) N.g.n[slot] = (int)N.all[7 * w + 6];
      }
      for (int i = 0; i < rows; i++)
        if (((unsigned)(lab >> (4 * i)) & 15u) == want)
          lab = (lab & ~(15ULL << (4 * i))) | ((unsigned long long)((up >> i) & 1u ? d1 : d0) << (4 * i));
      __syncthreads();
      if (tid == 0) {
        const int made = (int)any0 + (int)any1;
        N.made = program_next(N.g, N.pf, N.f, made, A.lim, maxmemb) ? made : -1;
      }
      __syncthreads();
    }
    const int nchild = N.g.nchild;
    if (nchild < 2) {  // one child == the node itself: never terminates
      if (tid == 0) atomicOr(&ctl->err, 2);
      if (CS > 1) cluster.sync();
      else __syncthreads();
      continue;
    }
    // stable scatter: members of each slot per warp and CTA, then every member's place
    unsigned mine = 0;  // lane s: this warp's members of slot s
    for (int i = 0; i < rows; i++) {
      const unsigned l = r0 + 32 * i + lane < r1 ? (unsigned)(lab >> (4 * i)) & 15u : 15u;
      for (int s = 0; s < nchild; s++) {
        const unsigned m = __ballot_sync(0xffffffffu, l == (unsigned)s);
        if (lane == s) mine += __popc(m);
      }
    }
    if (lane < 8) N.wcnt[w][lane] = lane < nchild ? mine : 0;
    __syncthreads();
    if (tid < 8) {
      int t = 0;
      for (int q = 0; q < SW; q++) t += N.wcnt[q][tid];
      N.tot[tid] = t;
    }
    if (CS > 1) cluster.sync();  // (and every CTA of the cluster holds its members)
    else __syncthreads();
    int next = s0;  // lane s: where this warp's next member of slot s goes
    if (lane < nchild) {
      for (int s = 0; s < lane; s++) next += N.g.n[s];
      if constexpr (CS > 1)
        for (int r = 0; r < rank; r++) next += cluster.map_shared_rank(&N.tot[0], r)[lane];
      for (int q = 0; q < w; q++) next += N.wcnt[q][lane];
    }
    for (int i = 0; i < rows; i++) {
      const bool in = r0 + 32 * i + lane < r1;
      const unsigned l = in ? (unsigned)(lab >> (4 * i)) & 15u : 15u;
      int dst = __shfl_sync(0xffffffffu, next, l & 7);
      for (int s = 0; s < nchild; s++) {
        const unsigned m = __ballot_sync(0xffffffffu, l == (unsigned)s);
        if (l == (unsigned)s) dst += __popc(m & lt);
        if (lane == s) next += __popc(m);
      }
      if (in) {
        const int o = i * ST + tid;
        A.perm[dst] = ps[o]; A.sx[dst] = xs[o]; A.sy[dst] = ys[o]; A.sz[dst] = zs[o];
      }
    }
    if (rank == 0) {
      NodeOut* O = &A.out[A.act[node]];
      if (tid < 13 * nchild) (&O->slot_f[0][0])[tid] = (&N.f[0][0])[tid];
      if (tid < 8) {
        O->slot_n[tid] = tid < nchild ? N.g.n[tid] : 0;
        O->order[tid] = tid < nchild ? N.g.order[tid] : -1;
      }
      if (tid == 0) {
        O->nchild = nchild;
        A.nch[node] = nchild;
      }
    }
    if (CS > 1) cluster.sync();  // the cluster's reads of each other's counts are done
    else __syncthreads();
  }
  // the level's last CTA: where each node's children begin
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&lv->arrive, 1) == total - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int a = lv->a, b = lv->b;
  int* ws = &N.wcnt[0][0];
  int carry = b;
  for (int base = a; base < b; base += ST) {
    const int i = base + tid;
    const int v = i < b ? __ldcg(A.nch + i) : 0;
    int s = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    if (lane == 31) ws[w] = s;
    __syncthreads();
    int before = carry, all = 0;
    for (int q = 0; q < SW; q++) {
      if (q < w) before += ws[q];
      all += ws[q];
    }
    if (i < b) A.cscan[i] = before + s - v;
    carry += all;
    __syncthreads();
  }
  if (tid == 0) {
    Level* nx = &ctl->lv[(lev + 1) % kLevels];
    nx->a = b;
    nx->b = __ldcg(&ctl->err) ? b : carry;  // (another CTA may have set it)
    Level z{};
    ctl->lv[(lev + 2) % kLevels] = z;
  }
}

// The class's members in shared memory.
template <int C>
constexpr size_t split_smem() { return (size_t)kClassRows[C] * ST * (3 * sizeof(double) + sizeof(int)); }

// CTAs for at most `nodes` nodes of class C.
template <int C>
int split_ctas(const Ctx* c, long long nodes) {
  const int per_sm = C >= 2 ? 1 : 2;
  const long long fit = std::max(1, c->num_sms * per_sm / kClassCtas[C]);
  return (int)(std::max(1LL, std::min(nodes, fit)) * kClassCtas[C]);
}
template <int C>
void launch_split(const Arrays& A, int lev, int ctas, int total, cudaStream_t s) {
  ensure_smem_attr(reinterpret_cast<const void*>(k_node_split<C>), (int)split_smem<C>());
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(ST);
  cfg.dynamicSmemBytes = split_smem<C>();
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kClassCtas[C];
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  count_launch();
  BIT_CUDA(cudaLaunchKernelEx(&cfg, k_node_split<C>, A, lev, total));
}

// The sixteen-CTA class needs room for such a cluster (a size past the portable eight).
bool clusters_of_16(Ctx* c) {
  if (c->clusters16 < 0) {
    auto* f = reinterpret_cast<const void*>(k_node_split<3>);
    ensure_smem_attr(f, (int)split_smem<3>());
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(ST);
    cfg.dynamicSmemBytes = split_smem<3>();
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 16;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    const bool ok = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, f, &cfg) == cudaSuccess;
    if (!ok) cudaGetLastError();  // (the eight-CTA class and the passes do without it)
    c->clusters16 = ok && n > 0;
  }
  return c->clusters16 > 0;
}

// One level's classes, the larger ones on the context's side streams: their nodes are disjoint,
// none fills the chip, and one after the other they took 144 us a level of 100k particles
// where together they take the longest's 53.  They have the context's stream's priority: its caller
// chose that for all of a build.  The side streams' work ends with this object.
struct SplitFork {
  Ctx* c;
  cudaStream_t s;
  int n;  // side streams in use
  SplitFork(Ctx* c_, cudaStream_t s_, int n_) : c(c_), s(s_), n(n_) {
    if (n == 0) return;
    for (int k = 0; k < n; k++)
      if (!c->side[k]) {
        int priority = 0;
        BIT_CUDA(cudaStreamGetPriority(s, &priority));
        BIT_CUDA(cudaStreamCreateWithPriority(&c->side[k], cudaStreamNonBlocking, priority));
        BIT_CUDA(cudaEventCreateWithFlags(&c->side_ev[k], cudaEventDisableTiming));
      }
    if (!c->fork_ev) BIT_CUDA(cudaEventCreateWithFlags(&c->fork_ev, cudaEventDisableTiming));
    BIT_CUDA(cudaEventRecord(c->fork_ev, s));
    for (int k = 0; k < n; k++) BIT_CUDA(cudaStreamWaitEvent(c->side[k], c->fork_ev, 0));
  }
  ~SplitFork() {
    for (int k = 0; k < n; k++) {
      cudaEventRecord(c->side_ev[k], c->side[k]);
      cudaStreamWaitEvent(s, c->side_ev[k], 0);
    }
  }
};
void split_level(Ctx* c, const Arrays& A, int lev, int top, long long n, long long actl, cudaStream_t s) {
  const int g0 = split_ctas<0>(c, actl), g1 = top >= 1 ? split_ctas<1>(c, n / class_members(0) + 1) : 0,
            g2 = top >= 2 ? split_ctas<2>(c, n / class_members(1) + 1) : 0,
            g3 = top >= 3 ? split_ctas<3>(c, n / class_members(2) + 1) : 0, all = g0 + g1 + g2 + g3;
  const SplitFork f(c, s, top);
  if (top >= 3) launch_split<3>(A, lev, g3, all, c->side[2]);
  if (top >= 2) launch_split<2>(A, lev, g2, all, c->side[1]);
  if (top >= 1) launch_split<1>(A, lev, g1, all, c->side[0]);
  launch_split<0>(A, lev, g0, all, s);
}

// The children of level lev's nodes, one warp per node: their records, and the lists of the
// next level's nodes to split.
__global__ void __launch_bounds__(256) k_make_children(Arrays A, int lev) {
  Ctl* ctl = A.ctl;
  if (ctl->stop || ctl->err) return;
  const Level* lv = &ctl->lv[lev % kLevels];
  Level* nx = &ctl->lv[(lev + 1) % kLevels];
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  const int lane = threadIdx.x & 31;
  const int a = lv->a, b = lv->b;
  if (a == b) return;  // past the last level
  if (nx->b > A.cap) {
    if (first) ctl->stop = 1;  // (read by the kernels that follow this one)
    return;
  }
  for (int p = a + (blockIdx.x * blockDim.x + threadIdx.x) / 32; p < b; p += gridDim.x * blockDim.x / 32) {
    if (A.act[p] < 0) continue;
    const NodeOut* O = &A.out[A.act[p]];
    const int nchild = O->nchild, base = A.cscan[p], sys = A.node_sys[p];
    const int n = lane < 8 ? O->slot_n[lane] : 0;
    int off = n;
    for (int o = 1; o < 8; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o) off += t;
    }
    off -= n;
    for (int i = lane; i < 13 * nchild; i += 32) A.fields[13LL * base + i] = (&O->slot_f[0][0])[i];
    for (int i = lane; i < 8 * nchild; i += 32) A.children[8LL * base + i] = -1;
    if (lane < 8) A.children[8LL * p + lane] = lane < nchild ? base + O->order[lane] : -1;
    if (lane < nchild) {
      const int node = base + lane;
      A.nummemb[node] = n;
      A.start[node] = A.start[p] + off;
      A.node_sys[node] = sys;
      enlist(node, n, A.sys_maxmemb[sys], nx, lev + 1, A.ls, A.act, A.nch, A.small);
    }
  }
  if (first) ctl->cur = lev + 1;
}

// ---- nodes of more members: all SMs ---------------------------------------------------------
// The large node's next bisection, or, its program done, what k_make_children needs.
__device__ void plan_divide(const Arrays& A, int node, SplitState* S, int made) {
  NodeOut* O = &A.out[A.act[node]];
  const double* P = A.fields + 13LL * node;
  S->has_cur = program_next(S->g, P, O->slot_f, made, A.lim, A.sys_maxmemb[A.node_sys[node]]);
  if (S->has_cur) {
    const Program& g = S->g;
    S->cur.dir = g.dir; S->cur.src = g.src; S->cur.c1 = g.c1; S->cur.c2 = g.c2;
    S->cur.mid = (g.src < 0 ? P : O->slot_f[g.src])[6 + g.dir];
    return;
  }
  if (S->g.nchild < 2) {  // one child == the node itself: never terminates
    atomicOr(&A.ctl->err, 2);
    S->g.nchild = 0;
  }
  O->nchild = S->g.nchild;
  A.nch[node] = S->g.nchild;
  for (int c = 0; c < 8; c++) {
    O->order[c] = c < S->g.nchild ? S->g.order[c] : -1;
    O->slot_n[c] = c < S->g.nchild ? S->g.n[c] : 0;
  }
}

// The large nodes of the level (list), numbered li = 0 .. nbig - 1.
__global__ void k_big_init(Arrays A, int nbig, const int* list, SplitState* st, SplitAcc* acc, int* nchunk,
                           int* done) {
  int li = blockIdx.x * blockDim.x + threadIdx.x;
  if (li >= nbig) return;
  acc_reset(&acc[li]);
  nchunk[li] = (A.nummemb[list[li]] + CH - 1) / CH;
  done[li] = 0;
  SplitState* S = &st[li];
  program_init(S->g);
  S->has_prev = 0;
  plan_divide(A, list[li], S, 0);
}

// Exclusive scan of a small int array in one block; total in out[n].
__global__ void k_scan_small(const int* in, int* out, int n) {
  __shared__ int ws[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int base = 0; base < n; base += blockDim.x) {
    int i = base + threadIdx.x;
    int v = i < n ? in[i] : 0;
    int s = v;
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    if (lane == 31) ws[w] = s;
    __syncthreads();
    if (w == 0) {
      int t = lane < nw ? ws[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        int u = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += u;
      }
      if (lane < nw) ws[lane] = t;
    }
    __syncthreads();
    int pre = carry + (w ? ws[w - 1] : 0) + s - v;
    if (i < n) out[i] = pre;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = pre + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry;
}

__global__ void k_fill_chunks(int nbig, const int* list, const int* start, const int* cbeg, int2* chunks) {
  const int li = blockIdx.x, s = start[list[li]];
  for (int c = cbeg[li] + threadIdx.x; c < cbeg[li + 1]; c += blockDim.x)
    chunks[c] = make_int2(li, s + (c - cbeg[li]) * CH);
}

__device__ __forceinline__ double coord(int dir, const double* sx, const double* sy,
                                        const double* sz, int e) {
  return dir == 0 ? sx[e] : (dir == 1 ? sy[e] : sz[e]);
}

// One bisection step for every large node of the level (decide = 0: the level's final pass,
// which only relabels): apply the previous step's
// relabel, then reduce counts / bounding boxes of both halves of the current step.  The
// CTA that finishes a node's last chunk then makes the node's decision for the next step.
// 6 CTAs per SM as without the decision (40 registers); whatever the call to decide_node
// needs beyond that is spilled on the deciding thread's path only
__global__ void __launch_bounds__(TB, 6)
    k_split_pass(const __grid_constant__ Arrays A, const int2* chunks, const int* nch, const int* list,
                 const int* nchunk, int* done, signed char* __restrict__ lab, SplitState* st, SplitAcc* acc,
                 int decide) {
  const double* __restrict__ sx = A.sx;
  const double* __restrict__ sy = A.sy;
  const double* __restrict__ sz = A.sz;
  if ((int)blockIdx.x >= *nch) return;  // the grid is sized from a bound
  const int2 ck = chunks[blockIdx.x];
  const SplitState* S = &st[ck.x];
  const int hp = S->has_prev, hc = S->has_cur;
  if (!hp && !hc) return;  // (its decision would change nothing)
  const Divide pv = S->prev, cu = S->cur;
  const int pc2 = pv.c2;
  const int node = list[ck.x];
  const int e1 = min(ck.y + CH, A.start[node] + A.nummemb[node]);
  int cnt[2] = {0, 0};
  unsigned long long v[12];  // per half and axis: the smallest key, the largest's complement
#pragma unroll
  for (int q = 0; q < 12; q++) v[q] = ~0ULL;
  // this thread's members e = ck.y + tid + k TB: every label first, then the unrolled
  // loop, so the members' loads overlap instead of waiting one after the other
  constexpr int PER = CH / TB;
  signed char lb[PER];
#pragma unroll
  for (int k = 0; k < PER; k++) {
    const int e = ck.y + threadIdx.x + k * TB;
    lb[k] = e < e1 ? lab[e] : (signed char)-128;  // no slot has label -128
  }
#pragma unroll
  for (int k = 0; k < PER; k++) {
    const int e = ck.y + threadIdx.x + k * TB;
    int l = lb[k];
    if (l == -128) continue;
    if (hp && l == pv.src) {
      l = (coord(pv.dir, sx, sy, sz, e) <= pv.mid) ? pv.c1 : pc2;
      lab[e] = (signed char)l;
    }
    if (hc && l == cu.src) {
      const bool h = !(coord(cu.dir, sx, sy, sz, e) <= cu.mid);
      const double x[3] = {sx[e], sy[e], sz[e]};
      cnt[h]++;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const unsigned long long k = okey(x[d]);
        if (h) {
          least(v[6 + 2 * d], k);
          least(v[7 + 2 * d], ~k);
        } else {
          least(v[2 * d], k);
          least(v[2 * d + 1], ~k);
        }
      }
    }
  }
  // warp (by halves: a build of 2M 2,465 -> 2,130 us, of 800k 935 -> 842), then CTA reductions;
  // one set of global atomics per CTA (min / max / sum are
  // order-independent, so the result is exact whatever the order)
  constexpr int NW = TB / 32;
  __shared__ int s_c[NW][2];
  __shared__ unsigned long long s_v[NW][12];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int h = 0; h < 2; h++) {
    const int c = __reduce_add_sync(0xffffffffu, cnt[h]);
    if (lane == 0) s_c[w][h] = c;
  }
  warp_least12(v);
  if (!(lane & 1) && (lane & 6) != 6) s_v[w][6 * (lane >> 4) + 3 * ((lane >> 3) & 1) + (lane & 6) / 2] = v[0];
  __syncthreads();
  if (hc && threadIdx.x < 2 * 7) {  // thread (h, q): q = 0..5 smallest / largest of an axis, 6 count
    const int h = threadIdx.x / 7, q = threadIdx.x % 7;
    int c = 0;
    for (int k = 0; k < NW; k++) c += s_c[k][h];
    if (c > 0) {
      if (q == 6) {
        atomicAdd(&acc[ck.x].cnt[h], c);
      } else {
        unsigned long long m = ~0ULL;
        for (int k = 0; k < NW; k++) least(m, s_v[k][6 * h + q]);
        if (q & 1) atomicMax(&acc[ck.x].mx[h][q >> 1], ~m);
        else atomicMin(&acc[ck.x].mn[h][q >> 1], m);
      }
    }
  }
  if (!decide) return;
  // The CTA that completes the node's chunk count (its atomics, and every other chunk's, are
  // visible after the fences) records the bisection and plans the next.  The sums arrived as
  // atomics in L2 from other CTAs; __ldcg reads them there.
  __shared__ int s_last;
  __threadfence();  // this thread's atomics, before the count that may complete the node
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&done[ck.x], 1) == nchunk[ck.x] - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  SplitState* D = &st[ck.x];
  SplitAcc* R = &acc[ck.x];
  if (hc) {
    const int n0 = __ldcg(&R->cnt[0]), n1 = __ldcg(&R->cnt[1]);
    const int c2 = n0 > 0 ? cu.c2 : cu.c1;
    if (threadIdx.x % 32 == 0 && threadIdx.x < 64) {  // a half's fields, one warp each
      const int h = threadIdx.x / 32, c = h ? c2 : cu.c1;
      if (h ? n1 : n0) {
        double bb[6];
        for (int q = 0; q < 3; q++) {
          bb[2 * q] = okey_inv(__ldcg(&R->mn[h][q]));
          bb[2 * q + 1] = okey_inv(__ldcg(&R->mx[h][q]));
        }
        box_fields(A.out[A.act[node]].slot_f[c], bb[0], bb[1], bb[2], bb[3], bb[4], bb[5]);
        D->g.n[c] = h ? n1 : n0;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      D->prev = cu;
      D->prev.c2 = c2;
      D->has_prev = 1;
      acc_reset(R);
      plan_divide(A, node, D, (n0 > 0) + (n1 > 0));
    }
  } else if (threadIdx.x == 0) {
    D->has_prev = 0;  // (relabelled above; nothing is left to do)
  }
  if (threadIdx.x == 0) done[ck.x] = 0;
}

__global__ void k_scatter_count(const int2* chunks, const int* nch, const int* list, const int* start, const int* nummemb,
                                const signed char* lab, int* cc) {
  if ((int)blockIdx.x >= *nch) return;  // the grid is sized from a bound
  const int2 ck = chunks[blockIdx.x];
  const int node = list[ck.x];
  const int e1 = min(ck.y + CH, start[node] + nummemb[node]);
  __shared__ int s[8];
  if (threadIdx.x < 8) s[threadIdx.x] = 0;
  __syncthreads();
  int c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int e = ck.y + threadIdx.x; e < e1; e += TB) {
    int l = lab[e];
#pragma unroll
    for (int v = 0; v < 8; v++) c[v] += (l == v);
  }
#pragma unroll
  for (int v = 0; v < 8; v++) {
    int t = warp_sum(c[v]);
    if ((threadIdx.x & 31) == 0 && t) atomicAdd(&s[v], t);
  }
  __syncthreads();
  if (threadIdx.x < 8) cc[blockIdx.x * 8 + threadIdx.x] = s[threadIdx.x];
}

// Per node (one block): destination offset of each chunk's members of each child slot,
// an exclusive scan over the node's chunks of the per-slot counts, 8 slots at once.
__global__ void __launch_bounds__(TB) k_scatter_offsets(const int* list, const int* start, const int* cbeg,
                                                        const int* cc, int* coff,
                                                        const SplitState* st, int* err) {
  const int li = blockIdx.x;
  const Program* S = &st[li].g;
  constexpr int NW = TB / 32;
  __shared__ int s_base[8], s_carry[8], s_warp[NW][8];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) {
    int acc = 0;
    for (int v = 0; v < 8; v++) { s_base[v] = start[list[li]] + acc; acc += v < S->nchild ? S->n[v] : 0; s_carry[v] = 0; }
  }
  __syncthreads();
  const int c0 = cbeg[li], c1 = cbeg[li + 1];
  for (int cb = c0; cb < c1; cb += TB) {
    const int c = cb + tid;
    int val[8], inc[8];
    for (int v = 0; v < 8; v++) {
      val[v] = c < c1 ? cc[c * 8 + v] : 0;
      inc[v] = val[v];
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc[v], o);
        if (lane >= o) inc[v] += t;
      }
    }
    if (lane == 31)
      for (int v = 0; v < 8; v++) s_warp[w][v] = inc[v];
    __syncthreads();
    if (c < c1)
      for (int v = 0; v < 8; v++) {
        int before = s_carry[v];
        for (int q = 0; q < w; q++) before += s_warp[q][v];
        coff[c * 8 + v] = s_base[v] + before + inc[v] - val[v];
      }
    __syncthreads();
    if (tid < 8)
      for (int q = 0; q < NW; q++) s_carry[tid] += s_warp[q][tid];
    __syncthreads();
  }
  if (tid < S->nchild && s_carry[tid] != S->n[tid]) atomicOr(err, 8);
}

// Stable scatter of each chunk's members to their child's range (order kept).
__global__ void __launch_bounds__(TB) k_scatter(const int2* chunks, const int* nch, const int* list, const int* start,
                                                const int* nummemb, const signed char* __restrict__ lab,
                                                const int* coff, const int* __restrict__ perm,
                                                const double* __restrict__ sx,
                                                const double* __restrict__ sy,
                                                const double* __restrict__ sz, int* __restrict__ perm2,
                                                double* __restrict__ sx2, double* __restrict__ sy2,
                                                double* __restrict__ sz2) {
  if ((int)blockIdx.x >= *nch) return;  // the grid is sized from a bound
  const int2 ck = chunks[blockIdx.x];
  const int node = list[ck.x];
  const int e1 = min(ck.y + CH, start[node] + nummemb[node]);
  __shared__ int wcnt[TB / 32][8];
  __shared__ int run[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < 8) run[threadIdx.x] = coff[blockIdx.x * 8 + threadIdx.x];
  __syncthreads();
  const unsigned lt = (1u << lane) - 1u;
  for (int t0 = ck.y; t0 < e1; t0 += TB) {
    int e = t0 + threadIdx.x;
    int l = e < e1 ? lab[e] : -2;
    // the member's record loads while its rank among the block's members is formed
    int pv = 0;
    double xv = 0.0, yv = 0.0, zv = 0.0;
    if (l >= 0) { pv = perm[e]; xv = sx[e]; yv = sy[e]; zv = sz[e]; }
    int my_rank = 0;
    for (int v = 0; v < 8; v++) {
      unsigned m = __ballot_sync(0xffffffffu, l == v);
      if (l == v) my_rank = __popc(m & lt);
      if (lane == 0) wcnt[w][v] = __popc(m);
    }
    __syncthreads();
    if (l >= 0) {
      int dst = run[l] + my_rank;
      for (int q = 0; q < w; q++) dst += wcnt[q][l];
      perm2[dst] = pv;
      sx2[dst] = xv;
      sy2[dst] = yv;
      sz2[dst] = zv;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
      int tot = 0;
      for (int q = 0; q < TB / 32; q++) tot += wcnt[q][threadIdx.x];
      run[threadIdx.x] += tot;
    }
    __syncthreads();
  }
}

// (restrict: the two copies never overlap, so a thread's members' loads need not wait
// for its earlier stores)
__global__ void k_copy_back(const int2* chunks, const int* nch, const int* list, const int* start, const int* nummemb,
                            const int* __restrict__ perm2, const double* __restrict__ sx2,
                            const double* __restrict__ sy2, const double* __restrict__ sz2,
                            int* __restrict__ perm, double* __restrict__ sx,
                            double* __restrict__ sy, double* __restrict__ sz) {
  if ((int)blockIdx.x >= *nch) return;  // the grid is sized from a bound
  const int2 ck = chunks[blockIdx.x];
  const int node = list[ck.x];
  const int e1 = min(ck.y + CH, start[node] + nummemb[node]);
#pragma unroll
  for (int e = ck.y + threadIdx.x; e < e1; e += TB) {
    perm[e] = perm2[e]; sx[e] = sx2[e]; sy[e] = sy2[e]; sz[e] = sz2[e];
  }
}

// Per node (one warp): the packed forms the traversal and the near field read, and a leaf's
// number at each of its members.
__global__ void __launch_bounds__(256) k_finish_nodes(int numtree, const double* fields, const int* children,
                                                      const int* nummemb, const int* start, double4* nodec,
                                                      float4* nodeh, int2* kids, int* leaf_of) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x & 31;
  if (i >= numtree) return;
  // a node's children are consecutive indices (children[] holds them in the reference's own
  // order), so one int2 gives the traversal all of them: (first, count); a leaf is (-1, nummemb)
  const int* ch = children + 8LL * i;
  if (ch[0] == -1)
    for (int e = start[i] + lane; e < start[i] + nummemb[i]; e += 32) leaf_of[e] = i;
  if (lane) return;
  int base = ch[0], cnt = 0;
  for (int c = 0; c < 8 && ch[c] != -1; c++) {
    base = min(base, ch[c]);
    cnt++;
  }
  kids[i] = cnt ? make_int2(base, cnt) : make_int2(-1, nummemb[i]);
  const double* f = fields + 13LL * i;
  nodec[i] = make_double4(f[6], f[7], f[8], f[12]);
  // half extents about the midpoint, rounded up to FP32 (a box the members are inside of)
  const double hx = fmax(f[1] - f[6], f[6] - f[0]), hy = fmax(f[3] - f[7], f[7] - f[2]),
               hz = fmax(f[5] - f[8], f[8] - f[4]);
  nodeh[i] = make_float4(__double2float_ru(hx), __double2float_ru(hy), __double2float_ru(hz), 0.f);
}

__global__ void k_iperm(int n, const int* perm, int* iperm) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) iperm[perm[e]] = e;
}

}  // namespace

template <class T>
void DBuf<T>::grow(Ctx* ctx, size_t count, size_t keep, cudaStream_t s) {
  if (count <= n && p) return;
  T* q = static_cast<T*>(dev_alloc(ctx, count * sizeof(T)));
  if (p && keep) BIT_CUDA(cudaMemcpyAsync(q, p, keep * sizeof(T), cudaMemcpyDeviceToDevice, s));
  BIT_CUDA(cudaStreamSynchronize(s));
  release();
  p = q;
  n = count;
  c = ctx;
}
template struct DBuf<int>;
template struct DBuf<double>;

void tree_build(Tree* t, const double* x, const double* y, const double* z) {
  Ctx* c = t->ctx;
  cudaStream_t s = c->stream;
  const int n = t->n;
  const int nsys = t->nsys;
  // systems: particle ranges and leaf sizes (one system unless the caller made a forest)
  if ((int)t->h_sys_start.size() != nsys) {
    t->h_sys_start.assign(1, 0);
    t->h_sys_n.assign(1, n);
    t->h_sys_maxmemb.assign(1, t->maxmemb);
  }
  t->sys_start.ensure(c, nsys);
  t->sys_n.ensure(c, nsys);
  t->sys_maxmemb.ensure(c, nsys);
  BIT_CUDA(cudaMemcpyAsync(t->sys_start.p, t->h_sys_start.data(), nsys * sizeof(int), cudaMemcpyHostToDevice, s));
  BIT_CUDA(cudaMemcpyAsync(t->sys_n.p, t->h_sys_n.data(), nsys * sizeof(int), cudaMemcpyHostToDevice, s));
  BIT_CUDA(cudaMemcpyAsync(t->sys_maxmemb.p, t->h_sys_maxmemb.data(), nsys * sizeof(int), cudaMemcpyHostToDevice, s));
  t->perm.ensure(c, n);
  t->sx.ensure(c, n); t->sy.ensure(c, n); t->sz.ensure(c, n);
  DBuf<int> perm2; DBuf<double> sx2, sy2, sz2;
  perm2.ensure(c, n); sx2.ensure(c, n); sy2.ensure(c, n); sz2.ensure(c, n);
  // nodes: an estimate, grown when it is short; nodes to split at one level: more than maxmemb
  // members each
  long long capl = 64, actl = 1;
  int most = 0;  // members of the largest node to split
  for (int k = 0; k < nsys; k++) {
    const int m = t->h_sys_maxmemb[k];
    capl += 16LL * (t->h_sys_n[k] / std::max(m, 1) + 1) + 8;
    actl += t->h_sys_n[k] / (m + 1LL);
    if (t->h_sys_n[k] > m) most = std::max(most, t->h_sys_n[k]);
  }
  const int small_node = most <= class_members(3) && clusters_of_16(c) ? class_members(3) : class_members(2);
  const bool big = most > small_node;
  int cap = (int)std::min<long long>(capl, 1LL << 30);
  DBuf<int> act, nch, cscan, small, big0, big1;
  DBuf<NodeOut> out;
  DBuf<Ctl> ctl;
  t->nummemb.ensure(c, cap); t->start.ensure(c, cap); t->children.ensure(c, 8LL * cap);
  t->fields.ensure(c, 13LL * cap); t->node_sys.ensure(c, cap);
  act.ensure(c, cap); nch.ensure(c, cap); cscan.ensure(c, cap);
  small.ensure(c, 2 * kClasses * actl);
  big0.ensure(c, n / class_members(2) + 1); big1.ensure(c, n / class_members(2) + 1);
  out.ensure(c, actl);
  ctl.ensure(c, 1);
  BIT_CUDA(cudaMemsetAsync(ctl.p, 0, sizeof(Ctl), s));
  static_assert(sizeof(Ctl) <= 64 * sizeof(long long), "the control block fits the pinned read-back area");
  Ctl* h = reinterpret_cast<Ctl*>(c->h_pinned);

  Arrays A{};
  A.perm = t->perm.p; A.sx = t->sx.p; A.sy = t->sy.p; A.sz = t->sz.p;
  A.perm2 = perm2.p; A.sx2 = sx2.p; A.sy2 = sy2.p; A.sz2 = sz2.p;
  A.sys_maxmemb = t->sys_maxmemb.p;
  A.out = out.p;
  A.ctl = ctl.p;
  for (int k = 0; k < kClasses; k++)
    for (int p = 0; p < 2; p++) A.ls.small[k][p] = small.p + (2 * k + p) * actl;
  A.ls.big[0] = big0.p;
  A.ls.big[1] = big1.p;
  A.lim = 1.0 / std::sqrt(2.0);  // src/tree3d.cpp:1371
  A.small = small_node;
  auto point_at_nodes = [&] {
    A.nummemb = t->nummemb.p; A.start = t->start.p; A.children = t->children.p;
    A.node_sys = t->node_sys.p; A.fields = t->fields.p;
    A.act = act.p; A.nch = nch.p; A.cscan = cscan.p;
    A.cap = cap;
  };
  point_at_nodes();

  DBuf<SplitAcc> acc;
  acc.ensure(c, nsys);
  count_launch(), k_acc_reset<<<grid_for(nsys, 128), 128, 0, s>>>(acc.p, nsys);
  {
    const unsigned per = std::max(1u, std::min<unsigned>(grid_for(n / nsys + 1, 256), 4 * c->num_sms / nsys + 1));
    count_launch(), k_root_bbox<<<dim3(per, nsys), 256, 0, s>>>(t->sys_start.p, t->sys_n.p, x, y, z, t->perm.p,
                                                                t->sx.p, t->sy.p, t->sz.p, acc.p, ctl.p);
  }
  count_launch(), k_root_init<<<grid_for(nsys, 128), 128, 0, s>>>(
      nsys, t->sys_start.p, t->sys_n.p, t->sys_maxmemb.p, acc.p, t->nummemb.p, t->start.p, t->children.p,
      t->fields.p, t->node_sys.p, ctl.p, A.ls, act.p, nch.p, small_node);
  BIT_CHECK_LAUNCH();

  const unsigned gsplit = (unsigned)std::max(1LL, std::min(actl, 2LL * c->num_sms));
  // the largest class a system's root may be in: the first levels launch no more
  int top = 0;
  while (top + 1 < kClasses && most > class_members(top) && class_members(top + 1) <= small_node) top++;
  auto sync_ctl = [&] {
    BIT_CUDA(cudaMemcpyAsync(h, ctl.p, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    BIT_CUDA(cudaStreamSynchronize(s));
    if (h->err & 1) fail(BIT_ERR_INVALID_ARGUMENT, "particle coordinates contain NaN");
    if (h->err & 2)
      fail(BIT_ERR_DEGENERATE,
           "a node with more than maxmemb members cannot be split (coincident particles); "
           "the reference's treemake would not terminate");
    if (h->err & 12) fail(BIT_ERR_CUDA, "internal tree-build consistency check failed");
  };
  auto make_children = [&](int lev) {
    const int lo = lev == h->cur ? h->lv[lev % kLevels].b - h->lv[lev % kLevels].a : 0;
    const unsigned grid = std::max(gsplit, std::min(grid_for(lo, 8), 4u * c->num_sms));
    count_launch(), k_make_children<<<grid, 256, 0, s>>>(A, lev);
  };
  DBuf<signed char> lab;
  DBuf<SplitState> st;
  DBuf<int> nchunk, cbeg, cc, coff, done;
  DBuf<int2> chunks;
  int cur = 0;
  h->cur = -1;
  if (big) sync_ctl();
  int nbig = big ? h->lv[0].nbig : 0;
  while (true) {
    if (nbig > 0) {
      const int* list = A.ls.big[cur & 1];
      lab.ensure(c, n);
      st.ensure(c, nbig);
      acc.ensure(c, nbig);
      nchunk.ensure(c, nbig);
      cbeg.ensure(c, nbig + 1);
      done.ensure(c, nbig);
      BIT_CUDA(cudaMemsetAsync(lab.p, -1, n, s));  // members start unlabelled
      const unsigned gl = grid_for(nbig, 128);
      count_launch(), k_big_init<<<gl, 128, 0, s>>>(A, nbig, list, st.p, acc.p, nchunk.p, done.p);
      count_launch(), k_scan_small<<<1, 1024, 0, s>>>(nchunk.p, cbeg.p, nbig);
      // The chunk count stays on the device (cbeg[nbig]): the chunk kernels run on a grid
      // sized from its bound, n / CH + one partial chunk per node, and CTAs past it return.
      const int* nchk = cbeg.p + nbig;
      const int nch_total = (int)std::min<long long>((long long)n / CH + nbig + 1, INT_MAX);
      chunks.ensure(c, nch_total);
      cc.ensure(c, 8LL * nch_total);
      coff.ensure(c, 8LL * nch_total);
      count_launch(), k_fill_chunks<<<nbig, 128, 0, s>>>(nbig, list, t->start.p, cbeg.p, chunks.p);
      for (int step = 0; step < 8; step++)  // 7 bisection steps at most, then the last relabel
        count_launch(), k_split_pass<<<nch_total, TB, 0, s>>>(A, chunks.p, nchk, list, nchunk.p, done.p, lab.p,
                                                              st.p, acc.p, step < 7);
      count_launch(), k_scatter_count<<<nch_total, TB, 0, s>>>(chunks.p, nchk, list, t->start.p, t->nummemb.p, lab.p, cc.p);
      count_launch(), k_scatter_offsets<<<nbig, TB, 0, s>>>(list, t->start.p, cbeg.p, cc.p, coff.p, st.p, &ctl.p->err);
      count_launch(), k_scatter<<<nch_total, TB, 0, s>>>(chunks.p, nchk, list, t->start.p, t->nummemb.p, lab.p, coff.p,
                                                         t->perm.p, t->sx.p, t->sy.p, t->sz.p, perm2.p, sx2.p,
                                                         sy2.p, sz2.p);
      count_launch(), k_copy_back<<<nch_total, TB, 0, s>>>(chunks.p, nchk, list, t->start.p, t->nummemb.p, perm2.p,
                                                           sx2.p, sy2.p, sz2.p, t->perm.p, t->sx.p, t->sy.p, t->sz.p);
    }
    // Without large nodes, four levels before the next look (a level past the last costs two
    // empty launches).
    const int batch = nbig > 0 ? 1 : 4;
    for (int k = 0; k < batch; k++) {
      split_level(c, A, cur + k, top, n, actl, s);
      make_children(cur + k);
    }
    BIT_CHECK_LAUNCH();
    sync_ctl();
    while (h->stop) {  // the node arrays are full: grow them, and go on where it stopped
      const int have = h->lv[h->cur % kLevels].b, need = h->lv[(h->cur + 1) % kLevels].b;
      const int ncap = std::max(2 * cap, need + 64);
      t->nummemb.grow(c, ncap, have, s); t->start.grow(c, ncap, have, s);
      t->children.grow(c, 8LL * ncap, 8LL * have, s); t->fields.grow(c, 13LL * ncap, 13LL * have, s);
      t->node_sys.grow(c, ncap, have, s);
      act.grow(c, ncap, have, s); nch.grow(c, ncap, have, s); cscan.grow(c, ncap, have, s);
      cap = ncap;
      point_at_nodes();
      BIT_CUDA(cudaMemsetAsync(&ctl.p->stop, 0, sizeof(int), s));
      make_children(h->cur);
      BIT_CHECK_LAUNCH();
      sync_ctl();
    }
    cur = h->cur;
    const Level& L = h->lv[cur % kLevels];
    if (L.a == L.b) break;
    nbig = L.nbig;
    // children are no larger than their parents
    while (nbig == 0 && top > 0 && L.nsmall[top] == 0) top--;
  }
  const int b = h->lv[cur % kLevels].a;
  t->numtree = b;
  t->depth = cur;
  t->cap = cap;
  t->nodec.ensure(c, b);
  t->nodeh.ensure(c, b);
  t->kids.ensure(c, b);
  t->leaf_of.ensure(c, n);
  t->iperm.ensure(c, n);
  t->pstart.ensure(c, b);
  count_launch(), k_finish_nodes<<<grid_for(b, 8), 256, 0, s>>>(b, t->fields.p, t->children.p, t->nummemb.p,
                                                               t->start.p, t->nodec.p, t->nodeh.p, t->kids.p,
                                                               t->leaf_of.p);
  count_launch(), k_iperm<<<grid_for(n, 256), 256, 0, s>>>(n, t->perm.p, t->iperm.p);
  BIT_CHECK_LAUNCH();
  tree_sync_host(t);
  // leaves in member order: leaf l's FP32 sources begin at record (start + l) / 2, which
  // leaves every leaf whole records of two
  std::vector<int> leaves, ps(b, 0);
  for (int i = 0; i < b; i++)
    if (t->h_children[8LL * i] == -1) leaves.push_back(i);
  std::sort(leaves.begin(), leaves.end(), [&](int p, int q) { return t->h_start[p] < t->h_start[q]; });
  t->nleaves = (int)leaves.size();
  for (int l = 0; l < t->nleaves; l++) ps[leaves[l]] = (int)(((unsigned)t->h_start[leaves[l]] + (unsigned)l) >> 1);
  BIT_CUDA(cudaMemcpyAsync(t->pstart.p, ps.data(), b * sizeof(int), cudaMemcpyHostToDevice, s));
  BIT_CUDA(cudaStreamSynchronize(s));
  t->gen++;
  t->has_moments = false;
  t->plists.valid = false;
  t->plists.alt_valid = false;
}

template struct DBuf<signed char>;
template struct DBuf<SplitState>;
template struct DBuf<SplitAcc>;
template struct DBuf<int2>;
template struct DBuf<NodeOut>;
template struct DBuf<Ctl>;

void tree_sync_host(Tree* t) {
  const int b = t->numtree;
  t->h_nummemb.resize(b); t->h_start.resize(b); t->h_children.resize(8LL * b);
  t->h_fields.resize(13LL * b); t->h_node_sys.resize(b);
  copy_d2h_batch(t->ctx, {{t->h_nummemb.data(), t->nummemb.p, b * sizeof(int)},
                          {t->h_start.data(), t->start.p, b * sizeof(int)},
                          {t->h_children.data(), t->children.p, 8LL * b * sizeof(int)},
                          {t->h_fields.data(), t->fields.p, 13LL * b * sizeof(double)},
                          {t->h_node_sys.data(), t->node_sys.p, b * sizeof(int)}});
  t->h_sys_leaf_sqr.assign(t->nsys, 0.0);
  for (int i = 0; i < b; i++)
    if (t->h_children[8LL * i] == -1) {
      double& m = t->h_sys_leaf_sqr[t->h_node_sys[i]];
      m = std::max(m, t->h_fields[13LL * i + 12]);
    }
}

}  // namespace bit
