// Near field of the fields: the leaf direct sums of treeforce / shielded_treeforce
// (src/tree3d.cpp:923-967, 3378-3398), with the work shared out as the potentials' (near.cu):
// one CTA per item and chunk of the group's targets, every warp a contiguous run of the group's
// sources, two targets a lane (mixed: one), its own tiles and accumulator rows (three, in FP64).
//
// FP64: the reference's sums, with 1/r^3 from one reciprocal square root: 16 FP64 operations a
// Coulomb pair, where a square root and a division took about 40.  Mixed: sources in FP32
// relative to their leaf centre, the target's offset from that centre formed in FP64 and
// rounded once, a tile's sums in FP32; pairs too close for FP32 coordinates are summed in FP64.
// Bound by the FP64 pipe, mixed by issue.  Before (a square root and a division, one target a
// thread, a barrier per tile) / now, ms: 2M clustered in leaves of 1000, theta = 0.7, FP64 Coulomb
// 24.2 / 11.0, mixed 7.6 / 6.1, screened 40.3 / 21.1; 100k uniform in leaves of 100 0.57 / 0.16, 0.47 /
// 0.11, 0.70 / 0.24; 50k in leaves of 300 1.03 / 0.20, 0.47 / 0.13, 1.50 / 0.33; 20k 0.33 / 0.08,
// 0.21 / 0.06, 0.42 / 0.10.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "fp64math.cuh"
#include "near.cuh"
#include "tma.cuh"

namespace bit {

namespace {

// Warps per CTA: with chunks of 256 targets, their three rows leave room for four CTAs an SM.
constexpr int NW = 4;
// The regularised Coulomb field, the same with the reference's KERNEL_ORDER family, the
// screened 2-D field.
enum { F_COULOMB = 0, F_ORDER = 1, F_CURL = 2 };

struct Field {
  double del, kappa;
  ExpScale k;
  const double2* tab;
  int korder;
};

// One pair's field in FP64, added to (ax, ay, az):
// F_COULOMB  q (x - x_j) / (r^2 + del)^(3/2) (eval_grad_kernel_reg, src/tree3d.cpp:73-97)
// F_ORDER    the same plus korder terms, each the previous one times (l + 1/2)/l del/rs
//            (src/tree3d.cpp:80-91)
// F_CURL     t (-dy, dx), t = q e^(-kappa r) / r^2 (kappa + 1/r) (src/tree3d.cpp:3384-3398)
// 1/r^3: with y the hardware seed of 1/r and e = 1 - rs y^2 (of the rounded y^2),
// y^3 (1 + 3/2 e + 15/8 e^2), an error of e^3 ~ 1e-17.
template <int FK, bool SELF, bool UF>
__device__ __forceinline__ void field64(double x, double y, double z, double4 s, const Field& f, bool own,
                                        double& ax, double& ay, double& az) {
  const double dx = x - s.x, dy = y - s.y, dz = z - s.z;
  double rs = fma(dx, dx, fma(dy, dy, fma(dz, dz, f.del))), q = s.w;
  if (SELF && own) {
    q = 0.0;
    rs = 1.0;
  }
  if constexpr (FK == F_ORDER) {
    double temp = 1.0 / (sqrt(rs) * rs), g = temp;
    for (int l = 1; l <= f.korder; l++) {
      g = g * (l + 0.5) / l * f.del / rs;
      temp += g;
    }
    const double t = q * temp;
    ax = fma(dx, t, ax); ay = fma(dy, t, ay); az = fma(dz, t, az);
  } else {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(rs));
    if constexpr (FK == F_COULOMB) {
      const double y2 = y0 * y0;
      const double e = fma(-rs, y2, 1.0);
      const double t = (q * y0) * y2 * fma(e, fma(e, 1.875, 1.5), 1.0);
      ax = fma(dx, t, ax); ay = fma(dy, t, ay); az = fma(dz, t, az);
    } else {
      const double u = rs * y0;
      const double e = fma(-u, y0, 1.0);
      const double ec = e * fma(e, 0.375, 0.5);
      const double ri = fma(y0, ec, y0);
      const double ex = exp_scaled<UF, kExpTabCopies>(fma(u, ec, u), f.k, f.tab);
      const double t = q * ex * (ri * ri) * (f.kappa + ri);
      ax = fma(-dy, t, ax); ay = fma(dx, t, ay);
    }
  }
}

struct Vec {
  double x, y, z;
};

// The field of a tile's sources j, j + step, ... by the plain formulas: where field64 leaves NaN
// (an r^2 past FP64's range counts as 0, one of 0 as infinite), and where a screened field grows
// with the distance (kappa < 0, which the entry points take) past exp_scaled's domain.
template <int FK>
__device__ __noinline__ Vec plain64(const double4* src, int n, double x, double y, double z, double del,
                                    double kappa, int o, int j, int step) {
  Vec p{0.0, 0.0, 0.0};
  for (; j < n; j += step) {
    if (j == o) continue;
    const double4 s = src[j];
    const double dx = x - s.x, dy = y - s.y, dz = z - s.z;
    const double rs = dx * dx + dy * dy + dz * dz + del, r = sqrt(rs);
    if (FK == F_CURL) {
      const double t = s.w * exp(-kappa * r) / rs * (kappa + 1 / r);
      p.x -= dy * t; p.y += dx * t;
    } else {
      const double t = s.w / (r * rs);
      p.x += dx * t; p.y += dy * t; p.z += dz * t;
    }
  }
  return p;
}

template <int FK, bool SELF, bool UF>
__device__ __forceinline__ void two64(const double4* src, int n, const Field& f, Vec s, Vec t, int o0, int o1,
                                      Vec& p, Vec& r) {
  p = r = Vec{0.0, 0.0, 0.0};
  Vec p1 = p, r1 = p;
  int j = 0;
#pragma unroll 1
  for (; j + 1 < n; j += 2) {
    const double4 a = src[j], b = src[j + 1];
    field64<FK, SELF, UF>(s.x, s.y, s.z, a, f, j == o0, p.x, p.y, p.z);
    field64<FK, SELF, UF>(t.x, t.y, t.z, a, f, j == o1, r.x, r.y, r.z);
    field64<FK, SELF, UF>(s.x, s.y, s.z, b, f, j + 1 == o0, p1.x, p1.y, p1.z);
    field64<FK, SELF, UF>(t.x, t.y, t.z, b, f, j + 1 == o1, r1.x, r1.y, r1.z);
  }
  if (j < n) {
    field64<FK, SELF, UF>(s.x, s.y, s.z, src[j], f, j == o0, p.x, p.y, p.z);
    field64<FK, SELF, UF>(t.x, t.y, t.z, src[j], f, j == o1, r.x, r.y, r.z);
  }
  p.x += p1.x; p.y += p1.y; p.z += p1.z;
  r.x += r1.x; r.y += r1.y; r.z += r1.z;
}

template <int FK, bool SELF, bool UF>
__device__ __forceinline__ Vec one64(const double4* src, int n, const Field& f, Vec s, int o, int j, int step) {
  Vec p{0.0, 0.0, 0.0}, q = p;
#pragma unroll 1
  for (; j + step < n; j += 2 * step) {
    field64<FK, SELF, UF>(s.x, s.y, s.z, src[j], f, j == o, p.x, p.y, p.z);
    field64<FK, SELF, UF>(s.x, s.y, s.z, src[j + step], f, j + step == o, q.x, q.y, q.z);
  }
  if (j < n) field64<FK, SELF, UF>(s.x, s.y, s.z, src[j], f, j == o, p.x, p.y, p.z);
  return Vec{p.x + q.x, p.y + q.y, p.z + q.z};
}

// Mixed: one target (offset from the leaf centre, negated and doubled) against records k,
// k + step, ...; careful: its own source, the empty half and close pairs add nothing.
struct Tile32 {
  const ulonglong2* rec;
  const double4* s64;  // the tile's sources in FP64
  int n;
  float del, thr;
};
template <bool CAREFUL>
__device__ __forceinline__ void field32(const Tile32& r, int k, f32x2 nx, f32x2 ny, f32x2 nz, int o, float& ax,
                                        float& ay, float& az, bool& close) {
  const ulonglong2 u = r.rec[2 * k], v = r.rec[2 * k + 1];
  const f32x2 dx = add2(u.x, nx), dy = add2(u.y, ny), dz = add2(v.x, nz);
  float2 f = unpack2(fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, pack2(r.del, r.del)))));
  float2 q = unpack2(v.y);
  if (CAREFUL) {
    const bool in0 = 2 * k != o, in1 = 2 * k + 1 != o && 2 * k + 1 < r.n;
    const bool c0 = f.x < r.thr, c1 = f.y < r.thr;
    close |= (in0 && c0) || (in1 && c1);
    if (!in0 || c0) { q.x = 0.f; f.x = 1.f; }
    if (!in1 || c1) { q.y = 0.f; f.y = 1.f; }
  }
  const float i0 = rsqrt_approx(f.x), i1 = rsqrt_approx(f.y);
  const float t0 = q.x * i0 * i0 * i0, t1 = q.y * i1 * i1 * i1;
  const float2 x = unpack2(dx), y = unpack2(dy), z = unpack2(dz);
  ax = fmaf(-x.x, t0, ax); ay = fmaf(-y.x, t0, ay); az = fmaf(-z.x, t0, az);
  ax = fmaf(-x.y, t1, ax); ay = fmaf(-y.y, t1, ay); az = fmaf(-z.y, t1, az);
}
template <bool CAREFUL>
__device__ __forceinline__ Vec sum32(const Tile32& r, double px, double py, double pz, float x, float y, float z,
                                     double del, int o, int k0, int step) {
  const f32x2 nx = pack2(-x, -x), ny = pack2(-y, -y), nz = pack2(-z, -z);
  const int nr = (r.n + 1) >> 1;
  float ax = 0.f, ay = 0.f, az = 0.f, bx = 0.f, by = 0.f, bz = 0.f;
  bool close = false;
  int k = k0;
#pragma unroll 1
  for (; k + step < nr; k += 2 * step) {
    field32<CAREFUL>(r, k, nx, ny, nz, o, ax, ay, az, close);
    field32<CAREFUL>(r, k + step, nx, ny, nz, o, bx, by, bz, close);
  }
  if (k < nr) field32<CAREFUL>(r, k, nx, ny, nz, o, ax, ay, az, close);
  Vec p{(double)(ax + bx), (double)(ay + by), (double)(az + bz)};
  if (CAREFUL && close) {  // this lane's close pairs, in FP64
    const float* f = reinterpret_cast<const float*>(r.rec);
    Field c{};
    c.del = del;
    for (k = k0; k < nr; k += step)
      for (int j = 2 * k; j < min(2 * k + 2, r.n); j++) {
        const float* s = f + 8 * (j >> 1) + (j & 1);
        if (j != o && r2_32(x, y, z, make_float4(s[0], s[2], s[4], 0.f), r.del) < r.thr)
          field64<F_COULOMB, false, false>(px, py, pz, r.s64[j], c, false, p.x, p.y, p.z);
      }
  }
  return p;
}

struct Layout {
  int recs, rows, tab;  // records of a tile, targets of a row, bytes of the exponential's table
  int chunk;            // targets of a CTA, at most
  int seq;              // no scratch: a group's first item takes the parts in turn, sums from here
  __host__ __device__ size_t warp_bytes() const {
    return 2 * (size_t)recs * kRec + (size_t)rows * (3 * sizeof(double) + sizeof(unsigned short));
  }
  __host__ __device__ size_t total() const { return tab + NW * warp_bytes(); }
};

// near_item of near.cu with three sums.  Field kinds per launch: FK.  SEQ as there.
template <int FK, bool F32, bool SEQ>
__global__ void __launch_bounds__(32 * NW, 4) k_near_field(NearArgs a, Layout L) {
  constexpr int PER = F32 ? 2 : 1;  // sources of a record
  __shared__ uint64_t bar[2 * NW];
  __shared__ int s_last;
  extern __shared__ __align__(128) unsigned char sm[];
  const int TILE = L.recs * PER;
  const int2 item = a.items[blockIdx.x];
  const int g = item.x, parts = item.y >> 16;
  int part = item.y & 0xffff;
  if (SEQ && part) return;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (L.tab) exp_tab_fill(reinterpret_cast<double2*>(sm), tid, 32 * NW);
  if (tid == 0) {
    for (int k = 0; k < 2 * NW; k++) mbar_init(&bar[k], 1);
    fence_mbar_init();
  }
  unsigned phase = 0;
  unsigned char* tiles0 = sm + L.tab;
  unsigned char* tiles = tiles0 + (size_t)w * 2 * L.recs * kRec;
  double* rows = reinterpret_cast<double*>(tiles0 + NW * 2 * (size_t)L.recs * kRec);
  double* row = rows + (size_t)w * 3 * L.rows;
  unsigned short* tl = reinterpret_cast<unsigned short*>(rows + (size_t)NW * 3 * L.rows) + (size_t)w * L.rows;

  const int gc = a.g_tcount[g], c0 = blockIdx.y * L.chunk, tc = min(gc - c0, L.chunk);
  if (tc <= 0) return;  // (the whole CTA)
  const int t0 = a.g_tstart[g] + c0, chunks = (gc + L.chunk - 1) / L.chunk;
  const SysEval* se = a.sys + a.g_sys[g];
  const int W = (gc + 31) >> 5, w0 = c0 >> 5, wn = (tc + 31) >> 5;  // words of the group, the chunk
  const long long e0 = a.off[g], e1 = e0 + a.cnt[g], m0 = a.moff[g];
  const double *cx = a.tx + t0, *cy = a.ty + t0, *cz = a.tz + t0;
  const long long tot = a.tot[g];
  Field f;
  f.del = se->near_del;
  f.kappa = se->kappa;
  f.k = exp_scale(se->kappa);
  f.tab = reinterpret_cast<const double2*>(sm) + (lane & (kExpTabCopies - 1));
  f.korder = se->kernel_order;
  auto warps_sum = [&](int d, int i) {
    double s = 0.0;
    for (int q = 0; q < NW; q++) s += rows[((size_t)q * 3 + d) * L.rows + i];
    return s;
  };
  double* seq = reinterpret_cast<double*>(sm + L.seq);
  for (;;) {  // once, or (SEQ) every part
    for (int i = tid; i < NW * 3 * L.rows; i += 32 * NW) rows[i] = 0.0;
    const int nv = NW * parts, v = part * NW + w;
    const long long T0 = run_begin(tot, nv, v), T1 = run_begin(tot, nv, v + 1);
    long long P;
    long long e = run_entry(a.pre, e0, e1, T0, [&](long long k) { return near_work(a, k); }, P);
    long long d0 = T0 - P, d1 = T1 - P;  // the run, from where the entry's work begins
    __syncthreads();  // the rows are zero, the table and the barriers are there
    bool failed = false;
    for (; e < e1 && d1 > 0; e++) {
      const int node = a.node[e], ns = a.nummemb[node], ec = a.tgt[e];
      const int wt = near_weight(ec);  // (the work is shared out by the whole group's)
      const int ja = cut(d0, wt, ns), jb = cut(d1, wt, ns);
      d0 -= (long long)wt * ns;
      d1 -= (long long)wt * ns;
      if (ja >= jb) continue;
      const bool all = ec == gc;
      const unsigned wd = !all && lane < wn ? a.mask[m0 + (e - e0) * W + w0 + lane] : 0u;
      const int cnt = all ? tc : __reduce_add_sync(0xffffffffu, __popc(wd));
      if (!cnt) continue;
      const int s0 = a.start[node];
      const unsigned char* src =
          reinterpret_cast<const unsigned char*>(a.src) + (size_t)(F32 ? a.pstart[node] : s0) * kRec;
      auto fetch = [&](int j, unsigned n) {
        if (lane == 0) {
          const int c = min(jb, (j / TILE + 1) * TILE) - j;
          const unsigned bytes = (unsigned)((c + PER - 1) / PER) * kRec;
          fence_proxy_async();
          mbar_expect_tx(&bar[2 * w + (n & 1)], bytes);
          tma_load_1d(tiles + (n & 1) * L.recs * kRec, src + (size_t)(j / PER) * kRec, bytes, &bar[2 * w + (n & 1)]);
        }
      };
      fetch(ja, phase);
      if (!all) pack_list(wd, wn, tl);
      const bool self = s0 < t0 + tc && t0 < s0 + ns;
      const double4 c = a.nodec[node];
      const float4 hb = a.nodeh[node];
      const NearSteps st = near_steps(cnt);
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
        const unsigned char* tile = tiles + (phase & 1) * L.recs * kRec;
        phase++;
        const int n = jn - j, own0 = t0 - s0 - j;
        auto add = [&](int i, const Vec& p) {
          row[i] += p.x;
          row[L.rows + i] += p.y;
          if (FK != F_CURL) row[2 * L.rows + i] += p.z;
        };
        if constexpr (F32) {
          Tile32 r{reinterpret_cast<const ulonglong2*>(tile), a.src64 + s0 + j, n, (float)f.del, near_close_thr(c.w)};
          if (!(r.del < r.thr)) r.thr = 0.f;
          auto sum = [&](int i, int k, int step) {
            const float x = (float)(cx[i] - c.x), y = (float)(cy[i] - c.y), z = (float)(cz[i] - c.z);
            return self || __any_sync(0xffffffffu, box_d2(x, y, z, hb) < r.thr)
                       ? sum32<true>(r, cx[i], cy[i], cz[i], x, y, z, f.del, self ? i + own0 : -1, k, step)
                       : sum32<false>(r, cx[i], cy[i], cz[i], x, y, z, f.del, -1, k, step);
          };
          for (int b = 0; b < cnt - 31; b += 32) {
            const int i = all ? b + lane : tl[b + lane];
            add(i, sum(i, 0, 1));
          }
          if (cnt & 31) {
            const int r0 = cnt & 31, sh = near_tail_shift(r0), slot = lane >> sh, slice = lane & ((1 << sh) - 1);
            const bool in = slot < r0;
            const int q = (cnt & ~31) + (in ? slot : 0), i = all ? q : tl[q];
            Vec p = sum(i, slice, 1 << sh);
            for (int o = 1 << sh >> 1; o; o >>= 1) {
              p.x += __shfl_xor_sync(0xffffffffu, p.x, o);
              p.y += __shfl_xor_sync(0xffffffffu, p.y, o);
              p.z += __shfl_xor_sync(0xffffffffu, p.z, o);
            }
            if (in && slice == 0) add(i, p);
          }
        } else {
          const double4* ds = reinterpret_cast<const double4*>(tile);
          const bool grows = FK == F_CURL && f.kappa < 0.0 && se->underflow;
          auto plain = [&](Vec& p, int i, int k, int step) {
            if (FK != F_ORDER && (grows || isnan(p.x)))  // (a pair's factor is NaN in all components)
              p = plain64<FK>(ds, n, cx[i], cy[i], cz[i], f.del, f.kappa, i + own0, k, step);
          };
          auto run = [&](auto S, auto U) {
            constexpr bool SELF = decltype(S)::value, UF = decltype(U)::value;
            for (int b = 0; b < st.full; b++) {
              const int r0 = 64 * b + lane, r1 = r0 + 32;
              const bool v1 = r1 < cnt;  // (a partial last block holds more than 48: r0 is a target)
              const int i0 = all ? r0 : tl[r0], i1 = v1 ? (all ? r1 : tl[r1]) : i0;
              Vec p, q;
              two64<FK, SELF, UF>(ds, n, f, Vec{cx[i0], cy[i0], cz[i0]}, Vec{cx[i1], cy[i1], cz[i1]}, i0 + own0,
                                  i1 + own0, p, q);
              plain(p, i0, 0, 1);
              plain(q, i1, 0, 1);
              add(i0, p);
              if (v1) add(i1, q);
            }
            int base = 64 * st.full;
            if (st.one) {
              const int i = all ? base + lane : tl[base + lane];
              Vec p = one64<FK, SELF, UF>(ds, n, f, Vec{cx[i], cy[i], cz[i]}, i + own0, 0, 1);
              plain(p, i, 0, 1);
              add(i, p);
              base += 32;
            }
            if (st.tail) {
              const int sh = near_tail_shift(st.tail), slot = lane >> sh, slice = lane & ((1 << sh) - 1);
              const bool in = slot < st.tail;
              const int r0 = base + (in ? slot : 0), i = all ? r0 : tl[r0];
              Vec p = one64<FK, SELF, UF>(ds, n, f, Vec{cx[i], cy[i], cz[i]}, i + own0, slice, 1 << sh);
              plain(p, i, slice, 1 << sh);
              for (int o = 1 << sh >> 1; o; o >>= 1) {
                p.x += __shfl_xor_sync(0xffffffffu, p.x, o);
                p.y += __shfl_xor_sync(0xffffffffu, p.y, o);
                p.z += __shfl_xor_sync(0xffffffffu, p.z, o);
              }
              if (in && slice == 0) add(i, p);
            }
          };
          // (the careful forms only where they can matter)
          if (FK == F_CURL && se->underflow) run(std::true_type{}, std::true_type{});
          else if (self) run(std::true_type{}, std::false_type{});
          else run(std::false_type{}, std::false_type{});
        }
        __syncwarp();
        j = jn;
      }
      if (failed) break;
    }
    __syncthreads();
    if (!SEQ || parts == 1) break;
    for (int i = tid; i < 3 * tc; i += 32 * NW) seq[i] = (part ? seq[i] : 0.0) + warps_sum(i / tc, i % tc);
    __syncthreads();  // the rows are read
    if (++part == parts) break;
  }
  // as near_item: straight into the result, or the group's scratch and then in part order
  double* sum = a.part + 3 * a.part_off[g];
  double* out[3] = {a.out, a.out_y, a.out_z};
  if (SEQ || parts == 1) {
    for (int i = tid; i < 3 * tc; i += 32 * NW)
      out[i / tc][t0 + i % tc] += parts == 1 ? warps_sum(i / tc, i % tc) : seq[i];
    return;
  }
  for (int i = tid; i < 3 * tc; i += 32 * NW)
    sum[((long long)part * 3 + i / tc) * gc + c0 + i % tc] = warps_sum(i / tc, i % tc);
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    s_last = atomicAdd(&a.part_done[g], 1) == parts * chunks - 1;
    if (s_last) {
      a.part_done[g] = 0;
      __threadfence();
    }
  }
  __syncthreads();
  if (!s_last) return;
  for (int i = tid; i < 3 * gc; i += 32 * NW) {
    double s = 0.0;
    for (int q = 0; q < parts; q++) s += __ldcg(sum + (long long)q * 3 * gc + i);
    out[i / gc][t0 - c0 + i % gc] += s;
  }
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
  a.src = P.f32 ? (const void*)t->src2.p : (const void*)t->src64.p;
  a.src64 = t->src64.p;
  a.nodeh = t->nodeh.p;
  a.sw = t->has_weights ? t->sw.p : nullptr;
  a.sys = P.sys.p;
  a.g_sys = L->g_sys.p;
  a.err = t->ctx->dev_err();
  a.tgt = L->near_tgt.p;
  a.pre = L->near_pre.p;
  a.pstart = t->pstart.p;
  a.tot = L->near_tot.p;
  a.leaf_of = t->leaf_of.p;
  a.part_off = L->part_off.p;
  a.part_done = L->part_done.p;
  return a;
}

void eval_near_force(Tree* t, Lists* L, const EvalPlan& P, double* fx, double* fy, double* fz) {
  Ctx* c = t->ctx;
  cudaStream_t s = c->stream;
  NearArgs a = near_args(t, L, P, t->sx.p, t->sy.p, t->sz.p);
  a.out = fx; a.out_y = fy; a.out_z = fz;
  // P.force: 1 the regularised Coulomb field (kernel order per system; FP64 beyond order
  // 0), 2 the screened 2-D field of shielded_treeforce (FP64)
  if (P.force == 2 && P.f32) fail(BIT_ERR_INVALID_ARGUMENT, "the screened field is FP64 only");
  bool korder = false;
  for (const SysEval& se : P.h_sys) korder |= se.kernel_order > 0;
  // the parts' scratch, three sums a target
  Layout lay;
  const bool seq = parts_in_turn(c, L, L->field_part, 3 * (size_t)L->part_total);
  a.part = L->field_part.p;
  lay.chunk = L->field_chunk;
  lay.rows = std::min(L->max_targets, lay.chunk);
  const int chunks = (L->max_targets + lay.chunk - 1) / lay.chunk;
  lay.tab = P.force == 2 ? kExpTabBytes : 0;
  lay.recs = c->near_tile ? std::min(128, std::max(32, c->near_tile / 8)) : 64;
  // four CTAs an SM if tiles of 32 do it
  while (lay.recs > 32 && lay.total() > kSmemMax / 4 - 1024) lay.recs -= 16;
  lay.seq = (int)((lay.total() + 15) / 16 * 16);
  const size_t bytes = seq ? lay.seq + 3 * lay.rows * sizeof(double) : lay.total();
  for (const LaunchClass& k : P.near_classes) {
    a.items = P.near_it + k.ibegin;
    auto go = [&](auto kernel) {
      ensure_smem_attr(reinterpret_cast<const void*>(kernel), kSmemMax - 1024);
      count_launch(), kernel<<<dim3(k.icount, chunks), 32 * NW, bytes, s>>>(a, lay);
      BIT_CHECK_LAUNCH();
    };
    auto run = [&](auto S) {
      constexpr bool SEQ = decltype(S)::value;
      if (P.force == 2) go(k_near_field<F_CURL, false, SEQ>);
      else if (P.f32) go(k_near_field<F_COULOMB, true, SEQ>);
      else if (korder) go(k_near_field<F_ORDER, false, SEQ>);
      else go(k_near_field<F_COULOMB, false, SEQ>);
    };
    if (seq) run(std::true_type{});
    else run(std::false_type{});
  }
}

}  // namespace bit
