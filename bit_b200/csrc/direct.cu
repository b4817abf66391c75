// FP64 direct sums at selected particle targets: the O(N^2) reference every treecode
// result is measured against (shielded_pot_particle_ds, src/tree3d.cpp:1966-2016, and the
// Coulomb / regularised-screened sums of the same form).  The target itself is skipped by
// index, as in the reference (`if (i != ind)`).
//
// Potentials: one CTA per (tile of up to 512 targets, chunk of sources), two targets a lane and
// the near field's pair arithmetic (near.cuh); with few targets the warps share the chunk's
// tiles out instead.  The chunks are as many as fill the SMs four times.  Bound by the FP64
// pipe (26 operations a screened pair); a call with 10,000 targets of 200,000 screened, host
// copies included: one target a thread with CUDA's square root, division and exponential,
// chunks of 16,384, 10.1 ms; now 4.3 ms.  Fields: one target a thread, chunks of 16,384.  Per-chunk partial sums are added per
// target in chunk order, so the result is deterministic.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "near.cuh"

namespace bit {

namespace {

constexpr int DT = 256;      // threads per CTA
constexpr int DS = 512;      // sources staged per tile
constexpr int DCH = 16384;   // sources per chunk (fields)

// Target p's sum over sources [j0, j1) of the tile at s0 by the plain formula: for sums that
// the pair arithmetic left NaN (a pair at distance 0, which the screened sum takes as infinite).
template <int KER>
__device__ __noinline__ double direct_plain(const double* x, const double* y, const double* z, const double* q,
                                            int j0, int j1, int p, double del, double kappa) {
  const double X = x[p], Y = y[p], Z = z[p];
  double acc = 0.0;
  for (int j = j0; j < j1; j++) {
    if (j == p) continue;
    const double dx = X - x[j], dy = Y - y[j], dz = Z - z[j];
    double r2 = dx * dx + dy * dy + dz * dz;
    if (KER != BIT_KERNEL_SCREENED) {
      r2 += del;
      if (!(r2 > kEpsNear)) continue;
    }
    const double r = sqrt(r2);
    acc += KER == BIT_KERNEL_COULOMB ? q[j] / r : q[j] * exp(-kappa * r) / r;
  }
  return acc;
}

// Chunks c0, c0 + 1, ... of `per` sources.  wt: warps with targets of their own (1, 2, 4, 8); the
// 8 / wt warps of one target set take a contiguous part of each tile each.
template <int KER, bool EPS>
__global__ void __launch_bounds__(DT, 2) k_direct(int n, const double* x, const double* y, const double* z,
                                                  const double* q, int m, const int* tg, double del,
                                                  double kappa, int per, int c0, int wt, double* part, int* err) {
  constexpr int PK = KER == BIT_KERNEL_COULOMB ? BIT_KERNEL_COULOMB : BIT_KERNEL_SCREENED;
  __shared__ double4 S[DS];
  __shared__ double2 tab[PK == BIT_KERNEL_COULOMB ? 1 : 64 * kExpTabCopies];
  __shared__ double red[DT / 32][64];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int slices = DT / 32 / wt, sl = w / wt;
  const int ti = blockIdx.x * 64 * wt + 64 * (w % wt) + lane;
  const int j0 = (c0 + blockIdx.y) * per, j1 = min(n, j0 + per);
  if (PK != BIT_KERNEL_COULOMB) exp_tab_fill(tab, tid, DT);
  int p[2];
  double X[2], Y[2], Z[2], acc[2] = {0.0, 0.0};
  for (int k = 0; k < 2; k++) {
    p[k] = ti + 32 * k < m ? tg[ti + 32 * k] : -1;
    if (p[k] >= n || p[k] < -1) {  // a target index outside the sources: flag it, sum nothing
      if (blockIdx.y == 0) atomicOr(err, 4);
      p[k] = -1;
    }
    X[k] = p[k] >= 0 ? x[p[k]] : 0.0;
    Y[k] = p[k] >= 0 ? y[p[k]] : 0.0;
    Z[k] = p[k] >= 0 ? z[p[k]] : 0.0;
  }
  Range64 r;
  r.del = KER == BIT_KERNEL_SCREENED ? 0.0 : del;
  r.k = exp_scale(kappa);
  r.tab = tab + (lane & (kExpTabCopies - 1));
  for (int s0 = j0; s0 < j1; s0 += DS) {
    const int cnt = min(DS, j1 - s0);
    __syncthreads();
    for (int k = tid; k < cnt; k += DT) S[k] = make_double4(x[s0 + k], y[s0 + k], z[s0 + k], q[s0 + k]);
    __syncthreads();
    const int lo = cnt * sl / slices, hi = cnt * (sl + 1) / slices;
    r.src = S + lo;
    r.n = hi - lo;
    const int o0 = p[0] - s0 - lo, o1 = p[1] - s0 - lo;  // the targets' own tile indices
    double a0, a1;
    if (__any_sync(0xffffffffu, (o0 >= 0 && o0 < r.n) || (o1 >= 0 && o1 < r.n)))
      two64<PK, EPS, true, true>(r, X[0], Y[0], Z[0], X[1], Y[1], Z[1], o0, o1, a0, a1);
    else
      two64<PK, EPS, false, true>(r, X[0], Y[0], Z[0], X[1], Y[1], Z[1], o0, o1, a0, a1);
    for (int k = 0; k < 2; k++) {
      double a = k ? a1 : a0;
      if (isnan(a) && p[k] >= 0) a = direct_plain<KER>(x, y, z, q, s0 + lo, s0 + hi, p[k], del, kappa);
      acc[k] += a;
    }
  }
  if (slices == 1) {
    for (int k = 0; k < 2; k++)
      if (ti + 32 * k < m) part[(long long)blockIdx.y * m + ti + 32 * k] = p[k] >= 0 ? acc[k] : 0.0;
    return;
  }
  for (int k = 0; k < 2; k++) red[w][lane + 32 * k] = p[k] >= 0 ? acc[k] : 0.0;
  __syncthreads();
  if (sl) return;
  for (int k = 0; k < 2; k++) {
    double a = 0.0;
    for (int s = 0; s < slices; s++) a += red[w + s * wt][lane + 32 * k];
    if (ti + 32 * k < m) part[(long long)blockIdx.y * m + ti + 32 * k] = a;
  }
}

// Field direct sums, force_particle_ds_reg (src/tree3d.cpp:298-330, with the KERNEL_ORDER
// family of eval_grad_kernel_reg, :73-97) and force_particle_ds_noreg (:182-213):
// sum over j != target of q_j G(x_j - x), G(d) = -d t, t = 1/(r rs) (+ korder terms) with
// rs = |d|^2 + del (REG) or t = 1/(rs sqrt(rs)) with rs = |d|^2.  Three partial sums per
// (chunk, target): part[(c * 3 + axis) * m + ti].
template <bool REG>
__global__ void __launch_bounds__(DT) k_direct_field(int n, const double* x, const double* y,
                                                     const double* z, const double* q, int m,
                                                     const int* tg, double del, int korder,
                                                     double* part, int* err) {
  __shared__ double4 S[DS];
  const int ti = blockIdx.x * DT + threadIdx.x;
  const int j0 = blockIdx.y * DCH, j1 = min(n, j0 + DCH);
  int p = ti < m ? tg[ti] : -1;
  if (p >= n || p < -1) {
    if (blockIdx.y == 0) atomicOr(err, 4);
    p = -1;
  }
  double X = 0, Y = 0, Z = 0;
  if (p >= 0) { X = x[p]; Y = y[p]; Z = z[p]; }
  double ax = 0.0, ay = 0.0, az = 0.0;
  for (int s0 = j0; s0 < j1; s0 += DS) {
    const int cnt = min(DS, j1 - s0);
    __syncthreads();
    for (int k = threadIdx.x; k < cnt; k += DT)
      S[k] = make_double4(x[s0 + k], y[s0 + k], z[s0 + k], q[s0 + k]);
    __syncthreads();
    if (p < 0) continue;
    const int self = p - s0;
    for (int k = 0; k < cnt; k++) {
      if (k == self) continue;
      const double4 s = S[k];
      const double dx = s.x - X, dy = s.y - Y, dz = s.z - Z;
      double t;
      if (REG) {
        const double rs = dx * dx + dy * dy + dz * dz + del;
        const double r = sqrt(rs);
        t = 1.0 / (r * rs);
        double f = t;
        for (int l = 1; l <= korder; l++) {
          f = f * (l + 0.5) / l * del / rs;
          t += f;
        }
      } else {
        const double rs = dx * dx + dy * dy + dz * dz;
        t = 1 / (rs * sqrt(rs));
      }
      ax += s.w * (-dx * t);
      ay += s.w * (-dy * t);
      az += s.w * (-dz * t);
    }
  }
  if (ti < m) {
    const long long b = (long long)blockIdx.y * 3 * m + ti;
    part[b] = ax;
    part[b + m] = ay;
    part[b + 2LL * m] = az;
  }
}

// out[i] = sign * sum over chunks of part[c][i], in chunk order; go_on: the sum of the chunks before
// is in out already
__global__ void k_direct_sum(int m, int nch, const double* part, bool go_on, double sign, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double s = go_on ? out[i] : 0.0;
  for (int c = 0; c < nch; c++) s += part[(long long)c * m + i];
  out[i] = sign * s;
}

// out[axis * m + i] = sum over chunks of part[(c * 3 + axis) * m + i], in chunk order
__global__ void k_direct_field_sum(int m, int nch, const double* part, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * m) return;
  const int axis = i / m, ti = i - axis * m;
  double s = 0.0;
  for (int c = 0; c < nch; c++) s += part[((long long)c * 3 + axis) * m + ti];
  out[i] = s;
}

}  // namespace

// All pointers on the device; out holds fx, fy, fz of the m targets (3 m doubles).
void direct_field(Ctx* c, int n, const double* x, const double* y, const double* z,
                  const double* q, int regularised, double del, int korder, int m,
                  const int* tg, double* out) {
  cudaStream_t s = c->stream;
  const int nch = (n + DCH - 1) / DCH;
  DBuf<double> part;
  part.ensure(c, (size_t)nch * 3 * m);
  const dim3 grid((m + DT - 1) / DT, nch);
  int* err = c->dev_err();
  if (regularised)
    count_launch(), k_direct_field<true><<<grid, DT, 0, s>>>(n, x, y, z, q, m, tg, del, korder, part.p, err);
  else
    count_launch(), k_direct_field<false><<<grid, DT, 0, s>>>(n, x, y, z, q, m, tg, del, korder, part.p, err);
  count_launch(), k_direct_field_sum<<<grid_for(3LL * m, 256), 256, 0, s>>>(m, nch, part.p, out);
  BIT_CHECK_LAUNCH();
}

// All pointers on the device.  The screened sum is negated (src/tree3d.cpp:2014).
void direct_potential(Ctx* c, int n, const double* x, const double* y, const double* z,
                      const double* q, const bit_eval_params& p, int m, const int* tg,
                      double* out) {
  cudaStream_t s = c->stream;
  int wt = 1;
  while (wt < DT / 32 && 64 * wt < m) wt *= 2;
  const int tiles = (m + 64 * wt - 1) / (64 * wt);
  // four CTAs a resident slot (two an SM), of at least a tile each
  const int want = std::max(1, std::min(4 * 2 * c->num_sms / tiles, (n + DS - 1) / DS));
  const int per = (n + want - 1) / want, nch = (n + per - 1) / per;
  // all chunks at once, or as many as the memory budget has room for: the sum goes on in chunk order
  const int at_once = (int)std::max<size_t>(1, std::min<size_t>(nch, ctx_room(c) / sizeof(double) / m));
  DBuf<double> part;
  part.ensure(c, (size_t)at_once * m);
  int* err = c->dev_err();
  const double sign = p.kernel == BIT_KERNEL_SCREENED ? -1.0 : 1.0;
  auto go = [&](auto kernel) {
    for (int c0 = 0; c0 < nch; c0 += at_once) {
      const int k = std::min(at_once, nch - c0);
      count_launch(), kernel<<<dim3(tiles, k), DT, 0, s>>>(n, x, y, z, q, m, tg, p.del, p.kappa, per, c0, wt, part.p, err);
      BIT_CHECK_LAUNCH();
      count_launch(), k_direct_sum<<<grid_for(m, 256), 256, 0, s>>>(m, k, part.p, c0 > 0, c0 + k < nch ? 1.0 : sign, out);
      BIT_CHECK_LAUNCH();
    }
  };
  // (where del alone keeps r^2 + del above the limit, no pair need check it)
  const bool eps = !(p.del > kEpsNear);
  switch (p.kernel) {
    case BIT_KERNEL_COULOMB:
      if (eps) go(k_direct<BIT_KERNEL_COULOMB, true>);
      else go(k_direct<BIT_KERNEL_COULOMB, false>);
      break;
    case BIT_KERNEL_SCREENED:
      go(k_direct<BIT_KERNEL_SCREENED, false>);
      break;
    default:
      if (eps) go(k_direct<BIT_KERNEL_SCREENED_REG, true>);
      else go(k_direct<BIT_KERNEL_SCREENED_REG, false>);
      break;
  }
}

}  // namespace bit
