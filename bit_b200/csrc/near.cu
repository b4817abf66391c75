// Near field of the potentials: the leaf direct sums of treepotential / shielded_treepot
// (src/tree3d.cpp:4737-4774, 3539-3623), one CTA per item: a target group, or one of the
// equal parts a heavy group's work is cut into.
//
// A group's near work is the sum over its near entries (source leaf, bitmask over the
// group's targets) of targets x sources.  The CTA's warps share it out by source: entry
// after entry, source after source, each warp takes the contiguous run that holds 1/8 of the
// group's pair steps, so that all finish together without meeting at a barrier per tile, and
// every lane of a warp reads the same source (one shared-memory wavefront a load).  For each
// entry of its run a warp packs the targets that need the leaf into a list, streams its
// sources through two of its own shared-memory tiles by TMA bulk copies (the next tile lands
// while this one is consumed), and takes the targets 64 at a time, two per lane, so that one
// source load serves two pairs and four pairs are in flight; the last few targets of a list
// share a source among several lanes.  Sums go to the warp's own accumulator row; rows are
// added in warp order at the end.  Everything follows from the lists alone, so results do
// not depend on timing.
//
// FP64: bound by the FP64 pipe (12 operations a Coulomb pair, 25 a screened one; the kernel
// this replaces, one target a thread and a barrier per tile, was held up by shared-memory
// wavefronts).  Mixed: by the MUFU (one or two a pair) and issue.  Before / now, ms, default
// settings: 2M clustered (leaves of 1000, theta = 0.7, 8.6 G pairs) FP64 screened 20.7 / 17.0,
// Coulomb 13.4 / 7.4, mixed 6.0 / 5.4 and 3.6 / 3.4; 100k, theta = 0.15 (1.6 G pairs): 10.8 / 3.1,
// 6.5 / 1.3, mixed 2.26 / 1.12, 1.72 / 0.57; 300k uniform in leaves of 100: 1.17 / 0.48, 0.75 / 0.28,
// mixed 0.68 / 0.30, 0.50 / 0.25; 20k in leaves of 500 0.71 / 0.12, 0.41 / 0.06, 0.20 / 0.07, 0.16 /
// 0.04.  Eight warps a CTA: four are 5% faster in the
// mixed 2M case and up to 50% slower on 20k.
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "fp64math.cuh"
#include "near.cuh"
#include "tma.cuh"

namespace bit {

namespace {

constexpr int NW = 8;  // warps per CTA

// Every listed target against one tile; sums into the warp's row.
template <int KER, bool EPS, bool SELF, bool UF>
__device__ __forceinline__ void tile64(const Range64& r, const double* cx, const double* cy,
                                       const double* cz, const unsigned short* tl, bool all, int cnt,
                                       int own0, double* row) {
  const int lane = threadIdx.x & 31;
  const NearSteps st = near_steps(cnt);
  for (int b = 0; b < st.full; b++) {
    const int r0 = 64 * b + lane, r1 = r0 + 32;
    const bool v1 = r1 < cnt;  // (a partial last block holds more than 48: r0 is a target)
    const int i0 = all ? r0 : tl[r0], i1 = v1 ? (all ? r1 : tl[r1]) : i0;
    double p0, p1;
    two64<KER, EPS, SELF, UF>(r, cx[i0], cy[i0], cz[i0], cx[i1], cy[i1], cz[i1], i0 + own0, i1 + own0, p0, p1);
    row[i0] += p0;
    if (v1) row[i1] += p1;
  }
  int base = 64 * st.full;
  if (st.one) {
    const int i = all ? base + lane : tl[base + lane];
    row[i] += one64<KER, EPS, SELF, UF>(r, cx[i], cy[i], cz[i], i + own0, 0, 1);
    base += 32;
  }
  if (st.tail) {
    const int sh = near_tail_shift(st.tail), slot = lane >> sh, slice = lane & ((1 << sh) - 1);
    const bool v = slot < st.tail;
    const int r0 = base + (v ? slot : 0);
    const int i = all ? r0 : tl[r0];
    double p = one64<KER, EPS, SELF, UF>(r, cx[i], cy[i], cz[i], i + own0, slice, 1 << sh);
    for (int o = 1 << sh >> 1; o; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
    if (v && slice == 0) row[i] += p;
  }
  __syncwarp();
}

// -------------------------------------------------------------------------------- FP32 pairs
// Mixed precision: sources in FP32 relative to their leaf's centre, two to a 32-byte record
// (x0 x1 y0 y1 z0 z1 q0 q1), the target's offset from that centre formed in FP64 and rounded
// once.  Differences, squares and sums run on packed pairs of sources (f32x2: one issue slot
// for two), 1/r and 2^x on the MUFU.
struct Range32 {
  const ulonglong2* rec;  // the tile: two vectors per record of two sources
  int n;                  // its sources (the last record may be half empty: charge 0)
  float del, kl2, thr;    // kl2 = -kappa log2(e); pairs below thr are close (near.cuh)
};

// A target against one record.  M_WATCH: also the least r^2, from which the caller sees that a
// close pair was among them; M_CAREFUL: the target's own source (index o), the empty half and
// close pairs add nothing, and `close` tells that there was a close one.  Only the differences
// and r^2 are packed: what follows the MUFU stays scalar, since gathering its results into
// pairs costs a move each.
enum { M_PLAIN = 0, M_WATCH = 1, M_CAREFUL = 2 };
template <int KER, int MODE>
__device__ __forceinline__ void pair32(const Range32& r, int k, f32x2 nx, f32x2 ny, f32x2 nz, int o,
                                       float2& acc, float& least, bool& close) {
  const ulonglong2 u = r.rec[2 * k], v = r.rec[2 * k + 1];
  const f32x2 dx = add2(u.x, nx), dy = add2(u.y, ny), dz = add2(v.x, nz);
  float2 f = unpack2(fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, pack2(r.del, r.del)))));
  float2 q = unpack2(v.y);
  if (MODE == M_WATCH) least = fminf(least, fminf(f.x, f.y));
  if (MODE == M_CAREFUL) {
    const bool in0 = 2 * k != o, in1 = 2 * k + 1 != o && 2 * k + 1 < r.n;
    const bool c0 = f.x < r.thr, c1 = f.y < r.thr;
    close |= (in0 && c0) || (in1 && c1);
    if (!in0 || c0) { q.x = 0.f; f.x = 1.f; }
    if (!in1 || c1) { q.y = 0.f; f.y = 1.f; }
  }
  const float i0 = rsqrt_approx(f.x), i1 = rsqrt_approx(f.y);
  if (KER == BIT_KERNEL_COULOMB) {
    acc.x = fmaf(q.x, i0, acc.x);
    acc.y = fmaf(q.y, i1, acc.y);
  } else {
    acc.x = fmaf(q.x * i0, ex2_approx(f.x * i0 * r.kl2), acc.x);
    acc.y = fmaf(q.y * i1, ex2_approx(f.y * i1 * r.kl2), acc.y);
  }
}

struct Target32 {
  f32x2 nx, ny, nz;  // minus the offset from the leaf's centre, twice
  int own;           // tile index of its own source
  __device__ Target32(float x, float y, float z, int o)
      : nx(pack2(-x, -x)), ny(pack2(-y, -y)), nz(pack2(-z, -z)), own(o) {}
};

template <int KER, int MODE>
__device__ __forceinline__ void two32(const Range32& r, const Target32& a, const Target32& b, float& p0,
                                      float& p1, bool& c0, bool& c1) {
  float2 s0{0.f, 0.f}, s1{0.f, 0.f}, t0{0.f, 0.f}, t1{0.f, 0.f};
  float m0 = HUGE_VALF, m1 = HUGE_VALF;
  const int nr = (r.n + 1) >> 1;
  int k = 0;
#pragma unroll 1
  for (; k + 1 < nr; k += 2) {
    pair32<KER, MODE>(r, k, a.nx, a.ny, a.nz, a.own, s0, m0, c0);
    pair32<KER, MODE>(r, k, b.nx, b.ny, b.nz, b.own, t0, m1, c1);
    pair32<KER, MODE>(r, k + 1, a.nx, a.ny, a.nz, a.own, s1, m0, c0);
    pair32<KER, MODE>(r, k + 1, b.nx, b.ny, b.nz, b.own, t1, m1, c1);
  }
  if (k < nr) {
    pair32<KER, MODE>(r, k, a.nx, a.ny, a.nz, a.own, s0, m0, c0);
    pair32<KER, MODE>(r, k, b.nx, b.ny, b.nz, b.own, t0, m1, c1);
  }
  p0 = (s0.x + s0.y) + (s1.x + s1.y);
  p1 = (t0.x + t0.y) + (t1.x + t1.y);
  if (MODE == M_WATCH) {
    c0 = m0 < r.thr;
    c1 = m1 < r.thr;
  }
}

// One target against records k, k + step, ...
template <int KER, int MODE>
__device__ __forceinline__ float one32(const Range32& r, const Target32& a, int k, int step, bool& c) {
  float2 s0{0.f, 0.f}, s1{0.f, 0.f};
  float m = HUGE_VALF;
  const int nr = (r.n + 1) >> 1;
#pragma unroll 1
  for (; k + step < nr; k += 2 * step) {
    pair32<KER, MODE>(r, k, a.nx, a.ny, a.nz, a.own, s0, m, c);
    pair32<KER, MODE>(r, k + step, a.nx, a.ny, a.nz, a.own, s1, m, c);
  }
  if (k < nr) pair32<KER, MODE>(r, k, a.nx, a.ny, a.nz, a.own, s0, m, c);
  if (MODE == M_WATCH) c = m < r.thr;
  return (s0.x + s0.y) + (s1.x + s1.y);
}

// Every listed target against one tile of leaf `entry` (centre c, half extents hb); compensated
// sums into the warp's row (rows values, then rows errors).  own0: the tile index of target
// 0's own source if the leaf holds targets of the group (SELF).  A warp takes the careful loop
// in its own leaf (without close pairs: where the tile holds the own source of one of its
// targets), and where the watching loop, taken within the close distance of the leaf's box, has
// met a close pair (rare; the pairs that both loops add are the same, bit for bit).  2M clustered
// in leaves of 1000, us: the careful loop in all these places, screened 5761, regularised 5018,
// Coulomb with a delta past the close distance 3571; as it is 5401, 4875, 3375; watching in the
// own leaf too 5640, 4873, 3375 (a close pair in 40% of its tiles).
template <int KER, bool SELF>
__device__ __forceinline__ void tile32(const NearArgs& a, const Range32& r, const double* cx,
                                       const double* cy, const double* cz, double4 c, float4 hb,
                                       const unsigned short* tl, bool all, int cnt, int own0, float* row,
                                       int rows, int t0, int g, long long e, int toff) {
  const int lane = threadIdx.x & 31;
  const NearSteps st = near_steps(cnt);
  auto target = [&](int i) {
    return Target32((float)(cx[i] - c.x), (float)(cy[i] - c.y), (float)(cz[i] - c.z), SELF ? i + own0 : -1);
  };
  auto near_box = [&](const Target32& t) {
    return box_d2(unpack2(t.nx).x, unpack2(t.ny).x, unpack2(t.nz).x, hb) < r.thr;
  };
  auto own_in = [&](const Target32& t) { return (unsigned)t.own < (unsigned)r.n; };
  auto one = [&](const Target32& t, int k, int step, bool& cl) {
    float p = 0.f;
    bool careful = SELF && (r.thr > 0.f || __any_sync(0xffffffffu, own_in(t)));
    if (!careful) {
      if (SELF || !__any_sync(0xffffffffu, near_box(t))) return one32<KER, M_PLAIN>(r, t, k, step, cl);
      p = one32<KER, M_WATCH>(r, t, k, step, cl);
      careful = __any_sync(0xffffffffu, cl);
      cl = false;
    }
    return careful ? one32<KER, M_CAREFUL>(r, t, k, step, cl) : p;
  };
  auto add = [&](int i, float p, bool close) {
    two_sum(row[i], row[rows + i], p);
    if (close) record_close(a, t0 + i, g, e, toff);
  };
  for (int b = 0; b < st.full; b++) {
    const int r0 = 64 * b + lane, r1 = r0 + 32;
    const bool v1 = r1 < cnt;  // (a partial last block holds more than 48: r0 is a target)
    const int i0 = all ? r0 : tl[r0], i1 = v1 ? (all ? r1 : tl[r1]) : i0;
    const Target32 x = target(i0), y = target(i1);
    float p0, p1;
    bool c0 = false, c1 = false;
    bool careful = SELF && (r.thr > 0.f || __any_sync(0xffffffffu, own_in(x) || own_in(y)));
    if (!careful) {
      // (in the own leaf no pair can be close here)
      if (!SELF && __any_sync(0xffffffffu, near_box(x) || near_box(y))) {
        two32<KER, M_WATCH>(r, x, y, p0, p1, c0, c1);
        careful = __any_sync(0xffffffffu, c0 || c1);
        c0 = c1 = false;
      } else {
        two32<KER, M_PLAIN>(r, x, y, p0, p1, c0, c1);
      }
    }
    if (careful) two32<KER, M_CAREFUL>(r, x, y, p0, p1, c0, c1);
    add(i0, p0, c0);
    if (v1) add(i1, p1, c1);
  }
  int base = 64 * st.full;
  if (st.one) {
    const int i = all ? base + lane : tl[base + lane];
    const Target32 x = target(i);
    bool cl = false;
    const float p = one(x, 0, 1, cl);
    add(i, p, cl);
    base += 32;
  }
  if (st.tail) {
    const int sh = near_tail_shift(st.tail), slot = lane >> sh, slice = lane & ((1 << sh) - 1);
    const bool v = slot < st.tail;
    const int r0 = base + (v ? slot : 0);
    const int i = all ? r0 : tl[r0];
    const Target32 x = target(i);
    bool cl = false;
    float p = one(x, slice, 1 << sh, cl);
    int c = cl;
    for (int o = 1 << sh >> 1; o; o >>= 1) {
      p += __shfl_xor_sync(0xffffffffu, p, o);
      c |= __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (v && slice == 0) add(i, p, c != 0);
  }
  __syncwarp();
}

// -------------------------------------------------------------------------------- the item
// Shared memory of a CTA: the exponential's table (FP64 screened), per warp two source tiles,
// an accumulator row (a double, or a float and its error, per target) and a target list.
// Tiles are counted in 32-byte records: one FP64 source, two FP32 ones.
// A group's tiles are as large as its own rows leave room for beside a second CTA, so that its
// sums do not depend on the other groups of the launch.  At most 128 records: 64 / 96 / 128, FP64
// screened, FP64 Coulomb, mixed screened, mixed Coulomb, us: 2M in leaves of 1000 17223 / 17073 /
// 17032, 7530 / 7407 / 7370, 5921 / 5794 / 5757, 3765 / 3618 / 3569; 20k, 500: 367 / 363 / 361, 150 / 144
// / 140, 127 / 121 / 121, 88 / 82 / 82; 300k, 100: 516 / 477 / 478, 320 / 281 / 279, 295 / 295 / 295, 248 /
// 246 / 248.
struct Layout {
  int cap, tab;  // records of a tile at most; bytes of the table
  int seq;       // groups that take their parts in turn: where the sums of those done begin
  static __host__ __device__ int rows(int tc) { return (tc + 31) / 32 * 32; }
  template <bool F32>
  static __host__ __device__ int recs(int cap, int rows) {
    constexpr int room = (kSmemMax / 2 - 1024 - (F32 ? 0 : kExpTabBytes)) / NW;
    const int n = (room - rows * (int)(sizeof(double) + sizeof(unsigned short))) / (2 * kRec) / 16 * 16;
    return n < 16 ? 16 : (n < cap ? n : cap);
  }
  static __host__ __device__ size_t warp_bytes(int recs, int rows) {
    return 2 * (size_t)recs * kRec + (size_t)rows * (sizeof(double) + sizeof(unsigned short));
  }
  // for every group of up to `most` targets
  template <bool F32>
  size_t total(int most) const {
    size_t b = 0;
    for (int r = 32; r <= most; r += 32) b = std::max(b, warp_bytes(recs<F32>(cap, r), r));
    return tab + NW * b;
  }
};

// Part `part` of group g's work, of `parts`: the CTA's warps' sums into their rows.  Returns false
// (in every thread) if a warp's bounded wait for a tile gave up: the error flag is set, the
// warp has waited, bounded again, for its copies in flight, and the group's result is not
// valid.  phase: this warp's count of completed copies, over the items of a queue.
template <int KER, bool EPS, bool F32>
__device__ __forceinline__ bool near_part(const NearArgs& a, const Layout& L, int g, int part, int parts,
                                          uint64_t* bar, unsigned& phase) {
  constexpr int PER = F32 ? 2 : 1;  // sources of a record
  const int ROWS = Layout::rows(a.g_tcount[g]), RECS = Layout::recs<F32>(L.cap, ROWS);
  const int TILE = RECS * PER;
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const double2* tab = reinterpret_cast<const double2*>(sm) + (lane & (kExpTabCopies - 1));
  unsigned char* tiles0 = sm + L.tab;
  unsigned char* tiles = tiles0 + (size_t)w * 2 * RECS * kRec;
  double* rows = reinterpret_cast<double*>(tiles0 + NW * 2 * (size_t)RECS * kRec);
  double* row = rows + (size_t)w * ROWS;
  unsigned short* tl = reinterpret_cast<unsigned short*>(rows + (size_t)NW * ROWS) + (size_t)w * ROWS;

  const int t0 = a.g_tstart[g], tc = a.g_tcount[g];
  const SysEval* se = a.sys + a.g_sys[g];
  const int W = (tc + 31) >> 5;
  const long long e0 = a.off[g], e1 = e0 + a.cnt[g], m0 = a.moff[g];
  const double *cx = a.tx + t0, *cy = a.ty + t0, *cz = a.tz + t0;
  for (int i = tid; i < NW * ROWS; i += 32 * NW) rows[i] = 0.0;
  // this warp's run [T0, T1) of the group's work (all parts' warps share it), and the entry
  // it begins in: the last whose prefix is at most T0
  const long long tot = a.tot[g];
  const int nv = NW * parts, v = part * NW + w;
  const long long T0 = run_begin(tot, nv, v), T1 = run_begin(tot, nv, v + 1);
  long long P;
  long long e = run_entry(a.pre, e0, e1, T0, [&](long long k) { return near_work(a, k); }, P);
  long long d0 = T0 - P, d1 = T1 - P;  // the run, from where the entry's work begins
  __syncthreads();  // the rows are zero
  const double del = se->near_del;
  const ExpScale ks = exp_scale(se->kappa);
  const float kl2 = (float)(-se->kappa * 1.4426950408889634);  // -kappa log2(e)
  bool failed = false;
  for (; e < e1 && d1 > 0; e++) {
    const int node = a.node[e], ns = a.nummemb[node], cnt = a.tgt[e];
    const int wt = near_weight(cnt);
    const int ja = cut(d0, wt, ns), jb = cut(d1, wt, ns);
    d0 -= (long long)wt * ns;
    d1 -= (long long)wt * ns;
    if (ja >= jb) continue;
    const int s0 = a.start[node];
    const unsigned char* src = reinterpret_cast<const unsigned char*>(a.src) +
                               (size_t)(F32 ? a.pstart[node] : s0) * kRec;
    auto fetch = [&](int j, unsigned n) {  // the tile that begins at source j (even for FP32)
      if (lane == 0) {
        const int cnt_j = min(jb, (j / TILE + 1) * TILE) - j;
        const unsigned bytes = (unsigned)((cnt_j + PER - 1) / PER) * kRec;
        fence_proxy_async();
        mbar_expect_tx(&bar[2 * w + (n & 1)], bytes);
        tma_load_1d(tiles + (n & 1) * RECS * kRec, src + (size_t)(j / PER) * kRec, bytes,
                    &bar[2 * w + (n & 1)]);
      }
    };
    // the first tile streams in while the targets are packed
    fetch(ja, phase);
    const bool all = cnt == tc;
    if (!all) {
      const unsigned wd = lane < W ? a.mask[m0 + (e - e0) * W + lane] : 0u;
      pack_list(wd, W, tl);
    }
    // a particle target's own source is the leaf's source at its own sorted position
    const bool self = se->particles && s0 < t0 + tc && t0 < s0 + ns;
    Range32 r32;
    double4 c{};
    float4 hb{};
    if (F32) {
      c = a.nodec[node];
      hb = a.nodeh[node];
      r32.del = (float)del;
      r32.kl2 = kl2;
      // where del alone reaches the threshold no pair of this leaf can be close
      r32.thr = near_close_thr(c.w);
      if (!(r32.del < r32.thr)) r32.thr = 0.f;
    }
    for (int j = ja; j < jb;) {
      const int jn = min(jb, (j / TILE + 1) * TILE);
      if (jn < jb) fetch(jn, phase + 1);  // (its buffer's reads ended at the last __syncwarp)
      if (!__all_sync(0xffffffffu, mbar_wait(&bar[2 * w + (phase & 1)], (phase >> 1) & 1))) {
        if (lane == 0) {
          atomicOr(a.err, 2);
          mbar_wait(&bar[2 * w + (phase & 1)], (phase >> 1) & 1);
          if (jn < jb) mbar_wait(&bar[2 * w + ((phase + 1) & 1)], ((phase + 1) >> 1) & 1);
        }
        __syncwarp();
        failed = true;
        break;
      }
      const unsigned char* tile = tiles + (phase & 1) * RECS * kRec;
      phase++;
      const int own = t0 - s0 - j;
      if constexpr (F32) {
        r32.rec = reinterpret_cast<const ulonglong2*>(tile);
        r32.n = jn - j;
        float* row32 = reinterpret_cast<float*>(row);
        const int toff = j / TILE * TILE;
        if (self) tile32<KER, true>(a, r32, cx, cy, cz, c, hb, tl, all, cnt, own, row32, ROWS, t0, g, e, toff);
        else tile32<KER, false>(a, r32, cx, cy, cz, c, hb, tl, all, cnt, 0, row32, ROWS, t0, g, e, toff);
      } else {
        const Range64 r{reinterpret_cast<const double4*>(tile), jn - j, del, ks, tab};
        if (KER != BIT_KERNEL_COULOMB && se->underflow) {
          if (self) tile64<KER, EPS, true, true>(r, cx, cy, cz, tl, all, cnt, own, row);
          else tile64<KER, EPS, false, true>(r, cx, cy, cz, tl, all, cnt, 0, row);
        } else {
          if (self) tile64<KER, EPS, true, false>(r, cx, cy, cz, tl, all, cnt, own, row);
          else tile64<KER, EPS, false, false>(r, cx, cy, cz, tl, all, cnt, 0, row);
        }
      }
      j = jn;
    }
    if (failed) break;
  }
  return !__syncthreads_or(failed);
}

// An item.  Returns false as near_part does.  SEQ: without scratch a group's first item takes all of
// its parts, one after the other, and adds their sums in shared memory in the same order.
template <int KER, bool EPS, bool F32, bool SEQ>
__device__ __forceinline__ bool near_item(const NearArgs& a, const Layout& L, int2 item, uint64_t* bar,
                                          unsigned& phase) {
  __shared__ int s_last;
  extern __shared__ __align__(128) unsigned char sm[];
  const int g = item.x, part = item.y & 0xffff, parts = item.y >> 16, tid = threadIdx.x;
  if (SEQ && part) return true;
  const int t0 = a.g_tstart[g], tc = a.g_tcount[g], ROWS = Layout::rows(tc), W = (tc + 31) >> 5;
  const double* rows = reinterpret_cast<const double*>(
      sm + L.tab + NW * 2 * (size_t)Layout::recs<F32>(L.cap, ROWS) * kRec);
  auto warps_sum = [&](int i) {
    double s = 0.0;
    for (int q = 0; q < NW; q++) {
      const double* x = rows + (size_t)q * ROWS;
      if (F32) {
        const float* f = reinterpret_cast<const float*>(x);
        s += (double)f[i] + (double)f[ROWS + i];
      } else {
        s += x[i];
      }
    }
    return s;
  };
  double* seq = reinterpret_cast<double*>(sm + L.seq);
  bool ok = near_part<KER, EPS, F32>(a, L, g, part, parts, bar, phase);
  if (SEQ && parts > 1) {
    for (int q = 0;;) {
      for (int i = tid; i < tc; i += 32 * NW) seq[i] = (q ? seq[i] : 0.0) + warps_sum(i);
      __syncthreads();  // the rows are read
      if (!ok || ++q == parts) break;
      ok = near_part<KER, EPS, F32>(a, L, g, q, parts, bar, phase);
    }
  }
  // this item's sums: straight into the result, or the group's scratch, which the CTA that
  // completes the group adds up in part order (a failed item counts too; the host sets the counts
  // back when it reports the error)
  double* sum = a.part + a.part_off[g];
  if (!SEQ && parts > 1) {
    for (int i = tid; i < tc; i += 32 * NW) sum[(long long)part * tc + i] = warps_sum(i);
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      s_last = atomicAdd(&a.part_done[g], 1) == parts - 1;
      if (s_last) {
        a.part_done[g] = 0;
        __threadfence();
      }
    }
    __syncthreads();
    if (!s_last) return ok;
  }
  for (int i = tid; i < tc; i += 32 * NW) {
    double s = 0.0;
    if (SEQ && parts > 1) {
      s = seq[i];
    } else if (parts > 1) {
      for (int q = 0; q < parts; q++) s += __ldcg(sum + (long long)q * tc + i);
    } else {
      s = warps_sum(i);
    }
    double self = 0.0;
    const SysEval* se = a.sys + a.g_sys[g];
    if (se->self_term) {
      // the reference's self term, where the target's own leaf is one of its near entries;
      // added, not subtracted (src/tree3d.cpp:3596)
      const int leaf = a.leaf_of[t0 + i];
      const long long e0 = a.off[g], e1 = e0 + a.cnt[g], m0 = a.moff[g];
      for (long long k = e0; k < e1; k++)
        if (a.node[k] == leaf) {
          if ((a.mask[m0 + (k - e0) * W + (i >> 5)] >> (i & 31)) & 1u)
            self = a.src64[t0 + i].w * se->intg / (a.sw ? a.sw[t0 + i] : 1.0);
          break;
        }
    }
    a.out[t0 + i] += se->near_sign * s + self;
  }
  return ok;
}

// Two mbarriers a warp for its tiles, and the exponential's table, before the kernel's first
// __syncthreads.
__device__ __forceinline__ void near_init(const Layout& L, uint64_t* bar) {
  extern __shared__ __align__(128) unsigned char sm[];
  if (L.tab) exp_tab_fill(reinterpret_cast<double2*>(sm), threadIdx.x, 32 * NW);
  if (threadIdx.x == 0) {
    for (int k = 0; k < 2 * NW; k++) mbar_init(&bar[k], 1);
    fence_mbar_init();
  }
}

// One launch class: CTA b takes item b.
template <int KER, bool EPS, bool F32, bool SEQ>
__global__ void __launch_bounds__(32 * NW, 2) k_near(NearArgs a, Layout L) {
  __shared__ uint64_t bar[2 * NW];
  near_init(L, bar);
  unsigned phase = 0;
  near_item<KER, EPS, F32, SEQ>(a, L, a.items[blockIdx.x], bar, phase);
}

// Persistent work queue over the items of every class (as k_far_queue): the same device code
// per item, so the results are identical.
template <bool F32, bool SEQ>
__global__ void __launch_bounds__(32 * NW, 2) k_near_queue(NearArgs a, Layout L, int count, int* head) {
  __shared__ int s_item;
  __shared__ uint64_t bar[2 * NW];
  near_init(L, bar);
  unsigned phase = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(head, 1);
    __syncthreads();
    const int k = s_item;
    __syncthreads();  // every thread has read s_item before it is overwritten
    if (k >= count) return;
    const int2 item = a.items[k];
    const SysEval* se = a.sys + a.g_sys[item.x];
    bool ok;
    // (the mixed path applies the limit on r^2 in its FP64 pass over close pairs)
    const bool eps = !F32 && se->eps_check;
    if (se->kernel == BIT_KERNEL_COULOMB)
      ok = eps ? near_item<BIT_KERNEL_COULOMB, !F32, F32, SEQ>(a, L, item, bar, phase)
               : near_item<BIT_KERNEL_COULOMB, false, F32, SEQ>(a, L, item, bar, phase);
    else
      ok = eps ? near_item<BIT_KERNEL_SCREENED, !F32, F32, SEQ>(a, L, item, bar, phase)
               : near_item<BIT_KERNEL_SCREENED, false, F32, SEQ>(a, L, item, bar, phase);
    if (!ok) return;
    __syncthreads();  // the item's last reads of shared memory precede the next item's writes
  }
}

// FP64 sum of the close pairs that the mixed kernel left out (FP32 r^2 < thr, the target's
// own source excluded), one warp per recorded target: the recorded tiles in list order (two
// warps whose runs meet in a tile may both have recorded it), or, for a target with more
// records than slots, every near entry of its group that covers it (tiles without close pairs
// add nothing, so the sum is the same).  Lanes take the sources in a fixed order and the warp
// reduces in a fixed order, so the result does not depend on scheduling.
template <int KER, bool EPS>
__device__ double close_sum(const NearArgs& a, const SysEval* se, int t, int g, double x, double y,
                            double z) {
  const int lane = threadIdx.x & 31;
  const double sdel = se->near_del;
  const float del = (float)sdel;
  const int self = se->particles ? t : -1;  // sorted position of the target's own source
  double acc = 0.0;
  auto tile = [&](int node, int j0, int j1) {
    const double4 c = a.nodec[node];
    const float xt = (float)(x - c.x), yt = (float)(y - c.y), zt = (float)(z - c.z);
    const float thr = near_close_thr(c.w);
    const int s0 = a.start[node];
    const float* f = reinterpret_cast<const float*>(a.src) + 8 * (size_t)a.pstart[node];
    for (int j = j0 + lane; j < j1; j += 32) {
      const float* p = f + 8 * (j >> 1) + (j & 1);
      if (s0 + j != self && r2_32(xt, yt, zt, make_float4(p[0], p[2], p[4], 0.f), del) < thr)
        pair64<KER, EPS, false, true, 1>(x, y, z, a.src64[s0 + j], sdel, exp_scale(se->kappa), kExp2Tab64, false, acc);
    }
  };
  const int nrec = a.ccnt[t];
  if (nrec <= kCloseRec) {
    int2 r[kCloseRec];
    for (int k = 0; k < nrec; k++) r[k] = a.crec[(long long)t * kCloseRec + k];
    if (nrec == 2 && (r[1].x < r[0].x || (r[1].x == r[0].x && r[1].y < r[0].y))) {
      const int2 s = r[0];
      r[0] = r[1];
      r[1] = s;
    }
    for (int k = 0; k < nrec; k++) {
      if (k && r[k].x == r[k - 1].x && r[k].y == r[k - 1].y) continue;
      const int node = a.node[r[k].x];
      tile(node, r[k].y, min(r[k].y + 2 * Layout::recs<true>(a.cap, Layout::rows(a.g_tcount[g])), a.nummemb[node]));
    }
  } else {
    const int i = t - a.g_tstart[g], W = (a.g_tcount[g] + 31) >> 5;
    const long long e0 = a.off[g], e1 = e0 + a.cnt[g], m0 = a.moff[g];
    for (long long e = e0; e < e1; e++)
      if ((a.mask[m0 + (e - e0) * W + (i >> 5)] >> (i & 31)) & 1u) {
        const int node = a.node[e];
        tile(node, 0, a.nummemb[node]);
      }
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

__global__ void __launch_bounds__(256) k_close(NearArgs a) {
  const int lane = threadIdx.x & 31;
  const int n = *a.cn;
  for (int w = blockIdx.x * 8 + (threadIdx.x >> 5); w < n; w += gridDim.x * 8) {
    const int2 tg = a.clist[w];
    const int t = tg.x, g = tg.y;
    const SysEval* se = a.sys + a.g_sys[g];
    const double x = a.tx[t], y = a.ty[t], z = a.tz[t];
    double v;
    if (se->kernel == BIT_KERNEL_COULOMB)
      v = se->eps_check ? close_sum<BIT_KERNEL_COULOMB, true>(a, se, t, g, x, y, z)
                        : close_sum<BIT_KERNEL_COULOMB, false>(a, se, t, g, x, y, z);
    else
      v = se->eps_check ? close_sum<BIT_KERNEL_SCREENED, true>(a, se, t, g, x, y, z)
                        : close_sum<BIT_KERNEL_SCREENED, false>(a, se, t, g, x, y, z);
    if (lane == 0) a.out[t] += se->near_sign * v;
  }
}

template <bool F32, bool SEQ>
void launch_near(Tree* t, Lists* L, const EvalPlan& P, NearArgs& a) {
  Ctx* c = t->ctx;
  cudaStream_t s = c->stream;
  a.part = L->near_part.p;
  Layout lay;
  lay.tab = 0;
  for (const LaunchClass& k : P.near_classes)
    if (!F32 && k.kernel != BIT_KERNEL_COULOMB) lay.tab = kExpTabBytes;
  // a context's tile setting counts the records of a CTA's eight warps
  lay.cap = a.cap = c->near_tile ? std::min(128, std::max(32, c->near_tile / 8)) : 128;
  size_t bytes = lay.total<F32>(L->max_targets);
  lay.seq = (int)((bytes + 15) / 16 * 16);
  if (SEQ) bytes = lay.seq + L->max_targets * sizeof(double);
  if (c->work_queue && P.near_classes.size() > 1) {
    const int count = (int)L->h_items.size();
    a.items = L->items.p;
    ensure_smem_attr(reinterpret_cast<const void*>(k_near_queue<F32, SEQ>), kSmemMax - 1024);
    int per_sm = 0;
    BIT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_near_queue<F32, SEQ>, 32 * NW, bytes));
    const int grid = std::max(1, std::min(count, c->num_sms * std::max(per_sm, 1)));
    c->queue_heads.ensure(c, 2);
    BIT_CUDA(cudaMemsetAsync(c->queue_heads.p + 1, 0, sizeof(int), s));
    count_launch(), k_near_queue<F32, SEQ><<<grid, 32 * NW, bytes, s>>>(a, lay, count, c->queue_heads.p + 1);
    BIT_CHECK_LAUNCH();
    return;
  }
  for (const LaunchClass& k : P.near_classes) {
    a.items = P.near_it + k.ibegin;
    auto go = [&](auto kernel) {
      ensure_smem_attr(reinterpret_cast<const void*>(kernel), kSmemMax - 1024);
      count_launch(), kernel<<<k.icount, 32 * NW, bytes, s>>>(a, lay);
      BIT_CHECK_LAUNCH();
    };
    const bool eps = !F32 && k.eps;
    if (k.kernel == BIT_KERNEL_COULOMB) {
      if (eps) go(k_near<BIT_KERNEL_COULOMB, !F32, F32, SEQ>);
      else go(k_near<BIT_KERNEL_COULOMB, false, F32, SEQ>);
    } else {
      if (eps) go(k_near<BIT_KERNEL_SCREENED, !F32, F32, SEQ>);
      else go(k_near<BIT_KERNEL_SCREENED, false, F32, SEQ>);
    }
  }
}

}  // namespace

bool parts_in_turn(Ctx* c, Lists* L, DBuf<double>& part, size_t count) {
  if (part.n >= count) return false;
  if (count * sizeof(double) > ctx_room(c)) L->gstage.release();
  if (count * sizeof(double) > ctx_room(c)) return true;
  part.ensure(c, count);
  return false;
}

// One launch per (kernel, eps check) class over its items, or one work queue over all.
void eval_near(Tree* t, Lists* L, const EvalPlan& P, const double* tx, const double* ty,
               const double* tz, double* out) {
  Ctx* c = t->ctx;
  cudaStream_t s = c->stream;
  NearArgs a = near_args(t, L, P, tx, ty, tz);
  a.out = out;
  if (!P.f32) {
    if (parts_in_turn(c, L, L->near_part, L->part_total)) launch_near<false, true>(t, L, P, a);
    else launch_near<false, false>(t, L, P, a);
    return;
  }
  // Mixed: close pairs need r^2 < thr = max(sqradius / 1024, 2e-14) of some leaf, and the
  // FP32 r^2 is at least the system's del (a rounded sum of non-negative terms and del);
  // where del reaches the largest leaf threshold no pair can be close, and the records
  // and the FP64 pass are skipped.
  bool close_possible = false;
  for (size_t sy = 0; sy < P.h_sys.size(); sy++)
    close_possible |= (float)P.h_sys[sy].near_del < near_close_thr(t->h_sys_leaf_sqr[sy]);
  if (close_possible) {
    // close-pair records, cleared for this evaluation (k_close consumes them)
    const int nt = L->ntargets;
    if (L->nnear >= INT_MAX) fail(BIT_ERR_CAPACITY, "too many near entries");
    c->close_cnt.ensure(c, nt);
    c->close_rec.ensure(c, (size_t)nt * kCloseRec);
    c->close_list.ensure(c, nt);
    c->close_n.ensure(c, 1);
    BIT_CUDA(cudaMemsetAsync(c->close_cnt.p, 0, (size_t)nt * sizeof(int), s));
    BIT_CUDA(cudaMemsetAsync(c->close_n.p, 0, sizeof(int), s));
    a.ccnt = c->close_cnt.p;
    a.crec = c->close_rec.p;
    a.clist = c->close_list.p;
    a.cn = c->close_n.p;
  }
  if (parts_in_turn(c, L, L->near_part, L->part_total)) launch_near<true, true>(t, L, P, a);
  else launch_near<true, false>(t, L, P, a);
  if (close_possible) {
    count_launch(), k_close<<<c->num_sms * 4, 256, 0, s>>>(a);
    BIT_CHECK_LAUNCH();
  }
}

}  // namespace bit
