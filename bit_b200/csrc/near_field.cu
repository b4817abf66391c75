// Near field of the fields: the leaf direct sums of treeforce / shielded_treeforce
// (src/tree3d.cpp:923-967, 3378-3398), one CTA per target group.
//
// For each near entry (source leaf, bitmask over the group's targets) the CTA packs the
// targets that need the leaf into a dense list and splits the leaf's sources across 1..32
// threads per target, whichever keeps the most threads busy (partial sums combined by
// warp shuffles).  Source tiles are staged in shared memory by TMA bulk
// copies (cp.async.bulk with an mbarrier), double buffered so the next tile streams in
// while the current one is consumed; every thread then reads each source from shared
// memory, broadcast across the targets.  Accumulation per target is in shared memory in a
// fixed order, so results are deterministic.
//
// FP64 path: the reference's arithmetic.  Mixed path: sources in FP32 relative to their
// leaf centre, the target's offset from that centre formed in FP64 and rounded once; pairs
// too close for FP32 coordinates are summed in FP64.
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "fp64math.cuh"
#include "near.cuh"
#include "tma.cuh"

namespace bit {

namespace {

constexpr int NT = 256;  // threads per CTA

template <bool F32>
struct Prec;
// Source tile (records per TMA copy): the default, and the range a context may choose
// (bit_ctx_set_near_config); shared memory holds two tiles.
template <>
struct Prec<true> {
  using S = float4;
  using T = float;
  static constexpr int TILE = 1024, TILE_MIN = 256, TILE_MAX = 2048;
};
template <>
struct Prec<false> {
  using S = double4;
  using T = double;
  static constexpr int TILE = 512, TILE_MIN = 128, TILE_MAX = 1024;
};

// Field of eval_grad_kernel_reg (src/tree3d.cpp:73-97), KERNEL_ORDER = 0:
// q * (-(x_j - x) / (r * r^2)).
__device__ __forceinline__ void fpair(double x, double y, double z, double4 s, double del,
                                      double& ax, double& ay, double& az) {
  const double dx = s.x - x, dy = s.y - y, dz = s.z - z;
  const double rs = dx * dx + dy * dy + dz * dz + del;
  const double r = sqrt(rs);
  const double t = s.w / (r * rs);
  ax -= dx * t; ay -= dy * t; az -= dz * t;
}
// The same with the reference's KERNEL_ORDER family (eval_grad_kernel_reg,
// src/tree3d.cpp:80-91): 1/(r rs) plus korder terms, each the previous one times
// (l + 1/2)/l * del/rs.
__device__ __forceinline__ void fpair_order(double x, double y, double z, double4 s, double del,
                                            int korder, double& ax, double& ay, double& az) {
  const double dx = s.x - x, dy = s.y - y, dz = s.z - z;
  const double rs = dx * dx + dy * dy + dz * dz + del;
  const double r = sqrt(rs);
  double temp = 1.0 / (r * rs), f = temp;
  for (int l = 1; l <= korder; l++) {
    f = f * (l + 0.5) / l * del / rs;
    temp += f;
  }
  const double t = s.w * temp;
  ax -= dx * t; ay -= dy * t; az -= dz * t;
}
// Screened 2-D field of one pair (shielded_treeforce's leaf loop, src/tree3d.cpp:3384-3398):
// t = q e^{-kappa r} / r^2 (kappa + 1/r), fx -= dy t, fy += dx t, no del.
__device__ __forceinline__ void cpair(double x, double y, double z, double4 s, double kappa,
                                      double& ax, double& ay) {
  const double dx = x - s.x, dy = y - s.y, dz = z - s.z;
  const double rs = dx * dx + dy * dy + dz * dz;
  const double r = sqrt(rs);
  const double t = s.w * exp(-kappa * r) / rs * (kappa + 1 / r);
  ax -= dy * t; ay += dx * t;
}

template <class T>
__device__ __forceinline__ T shfl_sum(T v, int tpt) {
  for (int o = tpt >> 1; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Field of one pair, q (x - x_j) / r^3 (eval_grad_kernel_reg, src/tree3d.cpp:73-97,
// KERNEL_ORDER = 0); CHK as acc_pot.
template <bool CHK>
__device__ __forceinline__ void acc_force(float xt, float yt, float zt, float4 s, float del,
                                          float thr, float& ax, float& ay, float& az,
                                          bool& close) {
  const float dx = xt - s.x, dy = yt - s.y, dz = zt - s.z;
  float rs = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, del)));
  float q = s.w;
  if (CHK) {
    const bool cl = rs < thr;
    close |= cl;
    q = cl ? 0.f : q;
    rs = cl ? 1.f : rs;
  }
  const float ri = rsqrt_approx(rs);
  const float tq = q * ri * ri * ri;
  ax = fmaf(dx, tq, ax); ay = fmaf(dy, tq, ay); az = fmaf(dz, tq, az);
}

__device__ __forceinline__ void close_force(float xt, float yt, float zt, double x, double y,
                                         double z, const float4* fs, const double4* s64,
                                         int slice, int tpt, int ns, int selfj, float del,
                                         float thr, double del64, double& cx, double& cy,
                                         double& cz) {
  for (int j = slice; j < ns; j += tpt)
    if (j != selfj && r2_32(xt, yt, zt, fs[j], del) < thr) fpair(x, y, z, s64[j], del64, cx, cy, cz);
}

// Threads per target for an entry with cnt targets: the power of two (1..32, or up to a tuned
// cap) that keeps the most of the CTA's threads busy over the rounds of NT units (a larger
// split must win by 4% to be taken, since it adds a shuffle reduction and shortens each
// thread's run).
__device__ __forceinline__ int split_for(int cnt, int cap) {
  const int maxtp = cap > 0 ? cap : 32;
  int best = 1;
  float bu = 0.f;
  for (int tp = 1; tp <= maxtp; tp <<= 1) {
    const int units = cnt * tp;
    const int rounds = (units + NT - 1) / NT;
    const float util = (float)units / (float)(rounds * NT);
    if (util > bu + 0.04f) {
      bu = util;
      best = tp;
    }
  }
  return best;
}

// Shared-memory layout of one CTA: two source tiles of `tile` records, then the
// accumulators, the packed target list and the mbarriers (target
// coordinates are read through L1).
template <bool F32>
struct Smem {
  using S = typename Prec<F32>::S;
  static constexpr size_t acc = 3 * kGroupMax * sizeof(double);
  static constexpr size_t list = kGroupMax * sizeof(int);
  static constexpr size_t bars = 64;
  __host__ __device__ static size_t tiles(int tile) { return 2 * (size_t)tile * sizeof(S); }
  __host__ __device__ static size_t total(int tile) { return tiles(tile) + acc + list + bars; }
};

// The whole near field of group g, by the whole CTA.  If a bounded wait gave up, the error
// flag is set, and the CTA has waited, bounded again, for its copies in flight.
template <int KER, bool F32>
__device__ __forceinline__ void near_group(const NearArgs& a, int g) {
  using P = Prec<F32>;
  using S = typename P::S;
  using T = typename P::T;
  using L = Smem<F32>;
  const int TILE = a.tile;
  extern __shared__ __align__(128) unsigned char sm[];
  S* tiles = reinterpret_cast<S*>(sm);
  const double* cx = a.tx + 0;  // group targets, indexed t0 + i below
  const double* cy = a.ty + 0;
  const double* cz = a.tz + 0;
  unsigned char* rest = sm + L::tiles(TILE);
  double* accd = reinterpret_cast<double*>(rest);
  int* tl = reinterpret_cast<int*>(rest + L::acc);
  uint64_t* bar = reinterpret_cast<uint64_t*>(rest + L::acc + L::list);
  __shared__ int s_cnt;

  const int t0 = a.g_tstart[g], tc = a.g_tcount[g];
  const SysEval* se = a.sys + a.g_sys[g];
  const double sdel = se->near_del, skappa = se->kappa;
  const int W = (tc + 31) >> 5;
  const long long e0 = a.off[g], e1 = e0 + a.cnt[g];
  const long long m0 = a.moff[g];
  const int tid = threadIdx.x, lane = tid & 31;
  for (int k = tid; k < 3 * kGroupMax; k += NT) accd[k] = 0.0;
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (e0 < e1) {
    const S* src = reinterpret_cast<const S*>(a.src);
    const float del = (float)sdel;
    // job iterator: (entry e, first source of the tile in the entry's leaf)
    long long e = e0;
    int node = a.node[e];
    int j0 = a.start[node], jn = a.nummemb[node];
    int toff = 0;
    if (tid == 0) {
      const int cnt0 = min(TILE, jn);
      fence_proxy_async();
      mbar_expect_tx(&bar[0], cnt0 * (unsigned)sizeof(S));
      tma_load_1d(tiles, src + j0, cnt0 * (unsigned)sizeof(S), &bar[0]);
    }
    int k = 0, tpt = 1, cnt = 0;
    while (true) {
      const int buf = k & 1;
      const int ns = min(TILE, jn - toff);
      if (toff == 0 && tid < 32) {
        // pack the targets of this entry (warp 0)
        unsigned wd = lane < W ? a.mask[m0 + (e - e0) * W + lane] : 0u;
        const int c = __popc(wd);
        int pre = c;
        for (int o = 1; o < 32; o <<= 1) {
          int t = __shfl_up_sync(0xffffffffu, pre, o);
          if (lane >= o) pre += t;
        }
        int base = pre - c;
        while (wd) {
          const int b = __ffs(wd) - 1;
          wd &= wd - 1;
          tl[base++] = 32 * lane + b;
        }
        if (lane == 31) s_cnt = pre;
      }
      // the next job streams into the other buffer while this one is consumed
      long long ne = e;
      int noff = toff + TILE;
      if (noff >= jn) { ne = e + 1; noff = 0; }
      if (tid == 0 && ne < e1) {
        const int nd = a.node[ne];
        const int cntn = min(TILE, a.nummemb[nd] - noff);
        fence_proxy_async();
        mbar_expect_tx(&bar[buf ^ 1], cntn * (unsigned)sizeof(S));
        tma_load_1d(tiles + (buf ^ 1) * TILE, src + a.start[nd] + noff,
                    cntn * (unsigned)sizeof(S), &bar[buf ^ 1]);
      }
      // Every thread waits (bounded) for this job's tile; the barrier then combines the
      // outcomes, so the whole CTA takes the same branch.  On a timeout the CTA waits,
      // bounded again, for both copies it may still have in flight into its shared memory
      // before it returns, and the host reports the error flag.
      const bool landed = mbar_wait(&bar[buf], (k >> 1) & 1);
      if (__syncthreads_or(!landed)) {
        if (tid == 0) {
          atomicOr(a.err, 2);
          mbar_wait(&bar[buf], (k >> 1) & 1);
          if (ne < e1) mbar_wait(&bar[buf ^ 1], ((k + 1) >> 1) & 1);
        }
        __syncthreads();
        return;
      }
      if (toff == 0) {
        cnt = s_cnt;
        tpt = split_for(cnt, a.split);
      }
      const S* ts = tiles + buf * TILE;
      const double4 c = a.nodec[node];
      // Particle targets: target i's own source sits at its sorted position t0 + i, i.e.
      // at tile index i + selfbase, which is inside this tile only if the target is one
      // of the tile's sources.
      const int selfbase = se->particles ? (t0 - (j0 + toff)) : INT_MIN;
      const int units = cnt * tpt;
      const int lt = __ffs(tpt) - 1;
      // close-pair checks are needed only where a target comes within r_t of this leaf's box
      float thr = fmaxf((float)c.w * kCloseFrac, kThrMin);  // r_t^2 = sqradius / 1024
      // the FP32 r^2 is at least del (fmaf of non-negative squares onto del), so where del
      // reaches thr no pair of this tile can be close: thr = 0 keeps every warp on the
      // plain loop (no box distance is below 0), which is then exact
      if (!(del < thr)) thr = 0.f;
      const float4 hb = a.nodeh[node];
      const double4* s64 = a.src64 + j0 + toff;
      for (int u0 = 0; u0 < units; u0 += NT) {
        const int u = u0 + tid;
        const bool valid = u < units;
        const int slot = u >> lt, slice = u & (tpt - 1);
        const int i = valid ? tl[slot] : 0;
        const int selfj = selfbase == INT_MIN ? -1 : i + selfbase;
        const bool self_in = selfj >= 0 && selfj < ns && ((selfj - slice) & (tpt - 1)) == 0;
        // the target's own source in this lane's slice: sum around it
        const int je = self_in ? selfj : ns;
        {
          T fx = 0, fy = 0, fz = 0;
          if constexpr (F32) {
            const float4* fs = reinterpret_cast<const float4*>(ts);
            const float xt = (float)(cx[t0 + i] - c.x), yt = (float)(cy[t0 + i] - c.y),
                        zt = (float)(cz[t0 + i] - c.z);
            const bool chk = __any_sync(0xffffffffu, valid && box_d2(xt, yt, zt, hb) < thr);
            if (valid) {
              bool close = false;
              if (!chk) {
                for (int j = slice; j < je; j += tpt)
                  acc_force<false>(xt, yt, zt, fs[j], del, thr, fx, fy, fz, close);
                if (self_in)
                  for (int j = selfj + tpt; j < ns; j += tpt)
                    acc_force<false>(xt, yt, zt, fs[j], del, thr, fx, fy, fz, close);
              } else {
                for (int j = slice; j < je; j += tpt)
                  acc_force<true>(xt, yt, zt, fs[j], del, thr, fx, fy, fz, close);
                if (self_in)
                  for (int j = selfj + tpt; j < ns; j += tpt)
                    acc_force<true>(xt, yt, zt, fs[j], del, thr, fx, fy, fz, close);
              }
              if (close) {
                double qx = 0.0, qy = 0.0, qz = 0.0;
                close_force(xt, yt, zt, cx[t0 + i], cy[t0 + i], cz[t0 + i], fs, s64, slice, tpt,
                            ns, selfj, del, thr, sdel, qx, qy, qz);
                fx += (float)qx; fy += (float)qy; fz += (float)qz;
              }
            }
          } else {
            if (valid) {
              const double4* ds = reinterpret_cast<const double4*>(ts);
              const double x = cx[t0 + i], y = cy[t0 + i], z = cz[t0 + i];
              const int korder = se->kernel_order;
              if (KER == BIT_KERNEL_SCREENED) {
                for (int j = slice; j < ns; j += tpt)
                  if (j != selfj) cpair(x, y, z, ds[j], skappa, fx, fy);
              } else if (korder > 0) {
                for (int j = slice; j < ns; j += tpt)
                  if (j != selfj) fpair_order(x, y, z, ds[j], sdel, korder, fx, fy, fz);
              } else {
                for (int j = slice; j < ns; j += tpt)
                  if (j != selfj) fpair(x, y, z, ds[j], sdel, fx, fy, fz);
              }
            }
          }
          fx = shfl_sum(fx, tpt);
          fy = shfl_sum(fy, tpt);
          fz = shfl_sum(fz, tpt);
          if (valid && slice == 0) {
            accd[i] += (double)fx;
            accd[kGroupMax + i] += (double)fy;
            accd[2 * kGroupMax + i] += (double)fz;
          }
        }
      }
      __syncthreads();
      k++;
      if (ne >= e1) break;
      if (ne != e) {
        e = ne;
        node = a.node[e];
        j0 = a.start[node];
        jn = a.nummemb[node];
      }
      toff = noff;
    }
  }
  __syncthreads();
  for (int i = tid; i < tc; i += NT) {
    a.out[t0 + i] += accd[i];
    a.out_y[t0 + i] += accd[kGroupMax + i];
    a.out_z[t0 + i] += accd[2 * kGroupMax + i];
  }
}

// One launch class: CTA b takes group order[b].
template <int KER, bool F32>
__global__ void __launch_bounds__(NT) k_near_field(NearArgs a) {
  near_group<KER, F32>(a, a.order[blockIdx.x]);
}

template <int KER, bool F32>
void launch(const NearArgs& a, int ngroups, cudaStream_t s) {
  const size_t bytes = Smem<F32>::total(a.tile);
  ensure_smem_attr(reinterpret_cast<const void*>(k_near_field<KER, F32>),
                   (int)Smem<F32>::total(Prec<F32>::TILE_MAX));
  count_launch(), k_near_field<KER, F32><<<ngroups, NT, bytes, s>>>(a);
}

}  // namespace

NearArgs near_args(Tree* t, Lists* L, const EvalPlan& P, const double* tx, const double* ty,
                   const double* tz) {
  NearArgs a{};
  a.g_tstart = L->g_tstart.p;
  a.g_tcount = L->g_tcount.p;
  a.tx = tx; a.ty = ty; a.tz = tz;
  a.off = L->near_off.p;
  a.cnt = L->near_cnt.p;
  a.moff = L->near_moff.p;
  a.node = L->near_node.p;
  a.mask = L->near_mask.p;
  a.start = t->start.p;
  a.nummemb = t->nummemb.p;
  a.nodec = t->nodec.p;
  a.src = P.f32 ? (const void*)t->src32.p : (const void*)t->src64.p;
  a.src64 = t->src64.p;
  a.nodeh = t->nodeh.p;
  a.sw = t->has_weights ? t->sw.p : nullptr;
  a.sys = P.sys.p;
  a.g_sys = L->g_sys.p;
  a.err = t->ctx->dev_err();
  // the context's tile, clamped to the precision's range (0: the default)
  const int want = t->ctx->near_tile;
  const int lo = P.f32 ? Prec<true>::TILE_MIN : Prec<false>::TILE_MIN;
  const int hi = P.f32 ? Prec<true>::TILE_MAX : Prec<false>::TILE_MAX;
  a.tile = want == 0 ? (P.f32 ? Prec<true>::TILE : Prec<false>::TILE) : std::min(hi, std::max(lo, want));
  a.split = t->ctx->near_split;
  a.tgt = L->near_tgt.p;
  a.pre = L->near_pre.p;
  a.pstart = t->pstart.p;
  a.tot = L->near_tot.p;
  a.leaf_of = t->leaf_of.p;
  a.part = L->near_part.p;
  a.part_off = L->part_off.p;
  a.part_done = L->part_done.p;
  return a;
}

void eval_near_force(Tree* t, Lists* L, const EvalPlan& P, double* fx, double* fy, double* fz) {
  cudaStream_t s = t->ctx->stream;
  NearArgs a = near_args(t, L, P, t->sx.p, t->sy.p, t->sz.p);
  a.out = fx; a.out_y = fy; a.out_z = fz;
  // P.force: 1 the regularised Coulomb field (kernel order per system; FP64 beyond order
  // 0), 2 the screened 2-D field of shielded_treeforce (FP64)
  for (const LaunchClass& k : P.near_classes) {
    a.order = P.near_ord + k.begin;
    if (P.force == 2) {
      if (P.f32) fail(BIT_ERR_INVALID_ARGUMENT, "the screened field is FP64 only");
      launch<BIT_KERNEL_SCREENED, false>(a, k.count, s);
    } else if (P.f32) {
      launch<BIT_KERNEL_COULOMB, true>(a, k.count, s);
    } else {
      launch<BIT_KERNEL_COULOMB, false>(a, k.count, s);
    }
    BIT_CHECK_LAUNCH();
  }
}

}  // namespace bit
