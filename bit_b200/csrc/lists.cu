// Interaction lists: the MAC traversal of treepotential / shielded_treepot / treeforce
// (src/tree3d.cpp:4679-4778, 3448-3627, 851-971) for a whole group of targets at once.
//
// A group is up to 1024 consecutive targets (a run of consecutive small leaves, a leaf, or
// a chunk of one; for external points, 32 to 256 consecutive points in Morton order).  One CTA walks
// the tree for the group, with a 32-bit mask word per 32 targets.  At a node every active target
// evaluates the reference's acceptance test in FP64 without contraction
// (sqradius < acc * ((dx*dx + dy*dy + dz*dz + add) - sub)); the node becomes a far entry
// for the accepting targets, and the others descend into the children, or get a near entry at
// a leaf.  Entries carry the group's bitmask.  Restricted to one target, the entries are
// exactly those of its reference traversal.  In a forest the walk starts at the root of the
// group's system, with that system's MAC.
//
// k_lists is a persistent kernel whose CTAs take groups from a device counter and visit each
// group's nodes breadth first, which is by increasing index, up to 256 waiting nodes at a time:
// one thread per node tests the box of the group's targets, the warps test the nodes that this
// leaves open against the targets they hold (one mask word or up to four a warp), then
// one thread per node places its far or near entry and its children by prefix sums.  What the
// group has visited (its reject masks above all) stays in the CTA's own region of global
// memory; the CTA then reserves room in the global lists with one atomic per list and writes
// the entries out (a group's entries are contiguous and in the order of the visits; groups land
// in completion order, addressed by begin/count).
//
// The lists are written in place, into arrays sized from an estimate, and the regions from the
// group with the most visits of the previous build (of this tree, else the context's last build
// under the same MAC; a first build uses an allowance).  Where a group overflows its region, or
// a reservation runs past the arrays, the build is run again, with four times the room a group
// (up to every node of the tree), or with room for the totals that this run counted: the same
// lists, later.  A memory budget limits the regions to as many as fit beside the lists, down to one,
// and what is allocated after them may have their room (dev_alloc).
//
// Bound by issue and latency (tensor and FP64 pipes idle, everything in L1 and L2).  Walking
// depth first, one node at a time and a thread per target, against this; a whole build with its
// host part, us: 2M particles, leaves of 1000: 3200 -> 1250; 300k, leaves of 100: 3500 -> 750;
// 200k, 500: 517 -> 258; 50k, 300: 235 -> 140; 10k, 200: 117 -> 82.  Of that the box test took
// the kernel from 1310 to 545 (2M) and from 200 to 116 (200k): half of the issue slots went to
// tests whose outcome the group shares.
//
// Optionally the walk also evaluates a second MAC (another kernel's parameters, e.g. the
// Coulomb test's (r^2 + del) - del next to the screened r^2 - mac_del) at every (target,
// node) it visits.  If no decision differs, that MAC's own walk would take the same path
// and emit the same entries, so the lists serve both MACs bit for bit; one differing
// decision anywhere and they serve only their own.
#include <algorithm>
#include <climits>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "near.cuh"

namespace bit {

namespace {

constexpr long long kVisitsFirst = 768;  // first build: visits of a group
constexpr int kVisitWords = 7;           // of a visit's record, next to its mask words
constexpr int QT = 256;                  // threads of the builder
constexpr size_t kRegionBytes = 1u << 30;  // of all regions, one at least

struct ListArgs {
  const int *g_tstart, *g_tcount;
  const double *tx, *ty, *tz;
  const double4* nodec;
  const int2* kids;  // per node: (first child, count), a leaf (-1, members)
  const SysEval* sys;  // per system: MAC parameters
  const int* g_sys;    // per group: system (its root is node g_sys[g])
  // per group
  long long *far_off, *near_off, *far_moff, *near_moff;
  int *far_cnt, *near_cnt;
  unsigned long long* g_near;  // near pairs of each group
  // per entry: its targets.  How a group's work is shared out, far: per group the first entry of
  // each share (work: targets); near: for the entries whose index is a multiple of 32, the work
  // (near_weight x sources) of their group's entries before them, from which run_entry finds the
  // others', and per group that of all
  unsigned short *far_tgt, *near_tgt;
  int* far_cut;
  long long *near_pre, *near_tot;
  // lists
  int *far_node, *near_node;
  unsigned *far_mask, *near_mask;
  unsigned long long* totals;  // far entries, far words, near entries, near words
  unsigned long long* pairs;   // far pairs, near pairs
  int* err;                    // 1: a region overflowed, 2: the arrays did,
                               // 4: the alternative MAC disagreed somewhere
  unsigned long long cap[4];   // room in the four output arrays
  int has_alt;                 // also evaluate a second MAC and compare its decisions
  double alt_acc, alt_add, alt_sub;
  // each resident CTA's own region in global memory, `stage` words, the most
  // visits of any group (maximum), and the work counter over the ngroups groups
  unsigned* gstage;
  long long stage;
  unsigned long long* visits;
  int* head;
  int ngroups;
};

// The alternative MAC's decision for squared distance s and node sqradius w.
__device__ __forceinline__ bool alt_ok(const ListArgs& a, double s, double w) {
  return w < dmul(a.alt_acc, dsub(dadd(s, a.alt_add), a.alt_sub));
}

// How the work of group g's entries, whose targets are in place, is shared out: warp 0 the far list
// (from entry fo; tot: its targets, all told), warp 1 the near list (from no).  A far entry belongs
// to share w of kFarWarps where w tot <= kFarWarps P < (w + 1) tot, P the targets of those before.
__device__ __forceinline__ void group_shares(const ListArgs& a, int g, long long nf, long long fo, long long tot,
                                             long long nn, long long no) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w > 1) return;
  const long long n = w ? nn : nf;
  long long run = 0;
  int cut[kFarWarps] = {};
  for (long long b = 0; b < n; b += 32) {
    const long long k = b + lane;
    long long v = 0;
    if (k < n) v = w ? (long long)near_weight(a.near_tgt[no + k]) * a.kids[a.near_node[no + k]].y : a.far_tgt[fo + k];
    long long inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    const long long before = run + inc - v;
    if (w) {
      if (k < n && !((no + k) & 31)) a.near_pre[(no + k) >> 5] = before;
    } else {
#pragma unroll
      for (int q = 1; q < kFarWarps; q++)
        cut[q] += __popc(__ballot_sync(0xffffffffu, k < n && before * kFarWarps < q * tot));
    }
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane) return;
  if (w) a.near_tot[g] = run;
  else
    for (int q = 0; q < kFarWarps; q++) a.far_cut[g * kFarWarps + q] = cut[q];
}

// No CTA waits for another; the work counter is the only shared state.
__global__ void __launch_bounds__(QT, 4) k_lists(ListArgs a) {
  constexpr int QW = QT / 32;
  constexpr int MAXJ = 32 / QW;  // mask words of a warp, at most
  __shared__ int s_item, s_ac[QT], s_rc[QT], s_open[QT], s_nopen, s_nan;
  __shared__ long long s_ws[QW];
  __shared__ double s_part[QW][6], s_box[6];
  __shared__ unsigned long long s_pairs[2], s_base[4];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  unsigned* region = a.gstage + (size_t)blockIdx.x * (size_t)a.stage;
  bool differ = false;
  for (;;) {
    __syncthreads();  // the last group's reads of shared memory and of the region
    if (tid == 0) s_item = atomicAdd(a.head, 1);
    if (tid < 2) s_pairs[tid] = 0;
    if (tid == 0) s_nopen = s_nan = 0;
    __syncthreads();
    const int g = s_item;
    if (g >= a.ngroups) break;
    const int t0 = a.g_tstart[g], tc = a.g_tcount[g], W = (tc + 31) >> 5, root = a.g_sys[g];
    const double macc = a.sys[root].acc, madd = a.sys[root].mac_add, msub = a.sys[root].mac_sub;
    // visit v: its node; the visit whose reject row holds the targets that came here (-1: all),
    // and the one whose row holds those that it rejected (itself, unless all were); the numbers
    // it accepted and rejected; the visits that made far and near entries, in order; reject rows
    const int vcap = (int)min(a.stage / (W + kVisitWords), (long long)INT_MAX);
    int* vnode = reinterpret_cast<int*>(region);
    int *vrow = vnode + vcap, *vrej = vrow + vcap, *vac = vrej + vcap, *vrc = vac + vcap, *fref = vrc + vcap, *nref = fref + vcap;
    unsigned* R = reinterpret_cast<unsigned*>(nref + vcap);
    auto live = [&](int j) { return tc - 32 * j >= 32 ? 0xffffffffu : (1u << (tc - 32 * j)) - 1u; };
    // Up to four words: the warps share the nodes out (nsl of them to a word); more: each warp
    // takes every node for words w, w + 8, ...
    const int wp = W > 4 ? QW : (W > 2 ? 4 : W), nsl = QW / wp, j0 = w % wp, sl = w / wp;
    double x[MAXJ], y[MAXJ], z[MAXJ];
#pragma unroll
    for (int i = 0; i < MAXJ; i++) {
      const int k = 32 * (j0 + QW * i) + lane;
      const bool in = k < tc && (i == 0 || wp == QW);
      x[i] = in ? a.tx[t0 + k] : 0.0;
      y[i] = in ? a.ty[t0 + k] : 0.0;
      z[i] = in ? a.tz[t0 + k] : 0.0;
    }
    // the box of the group's targets
    {
      double b[6] = {HUGE_VAL, HUGE_VAL, HUGE_VAL, -HUGE_VAL, -HUGE_VAL, -HUGE_VAL};
      bool nan = false;
#pragma unroll
      for (int i = 0; i < MAXJ; i++) {
        if (!(32 * (j0 + QW * i) + lane < tc && (i == 0 || wp == QW))) continue;
        const double t[3] = {x[i], y[i], z[i]};
        for (int q = 0; q < 3; q++) {
          nan |= isnan(t[q]);
          b[q] = fmin(b[q], t[q]);
          b[3 + q] = fmax(b[3 + q], t[q]);
        }
      }
      for (int q = 0; q < 6; q++) {
        for (int o = 16; o; o >>= 1) {
          const double t = __shfl_xor_sync(0xffffffffu, b[q], o);
          b[q] = q < 3 ? fmin(b[q], t) : fmax(b[q], t);
        }
        if (lane == 0) s_part[w][q] = b[q];
      }
      if (nan) s_nan = 1;
      __syncthreads();
      if (tid < 6) {
        double t = s_part[0][tid];
        for (int q = 1; q < QW; q++) t = tid < 3 ? fmin(t, s_part[q][tid]) : fmax(t, s_part[q][tid]);
        s_box[tid] = t;
      }
    }
    if (tid == 0) {
      vnode[0] = root;
      vrow[0] = -1;
    }
    __syncthreads();
    int head = 0, tail = 1, nf = 0, nn = 0;
    unsigned long long fp = 0, np = 0;
    bool full = vcap < 1;
    while (head < tail && !full) {
      const int c = min(QT, tail - head);
      s_ac[tid] = s_rc[tid] = 0;
      // One thread per node tries the whole box first.  Every operation of the test rounds
      // monotonically, so the box's nearest point to the node bounds all targets' values from
      // below and its farthest corner from above: the decision is theirs, bit for bit.
      int verdict = 0;  // 1: all accept, -1: all reject, 0: open
      if (tid < c) {
        const double4 nd = a.nodec[vnode[head + tid]];
        const double n3[3] = {nd.x, nd.y, nd.z};
        double lo[3], hi[3];
        for (int q = 0; q < 3; q++) {
          const double d0 = dsub(s_box[q], n3[q]), d1 = dsub(s_box[3 + q], n3[q]);
          lo[q] = n3[q] >= s_box[q] ? (n3[q] <= s_box[3 + q] ? 0.0 : d1) : d0;
          hi[q] = fmax(fabs(d0), fabs(d1));
        }
        const double s0 = dadd(dadd(dmul(lo[0], lo[0]), dmul(lo[1], lo[1])), dmul(lo[2], lo[2]));
        const double s1 = dadd(dadd(dmul(hi[0], hi[0]), dmul(hi[1], hi[1])), dmul(hi[2], hi[2]));
        const bool all = nd.w < dmul(macc, dsub(dadd(s0, madd), msub));
        const bool any = nd.w < dmul(macc, dsub(dadd(s1, madd), msub));
        verdict = !s_nan && macc >= 0.0 && (all || !any) ? (all ? 1 : -1) : 0;
        if (a.has_alt && !(a.alt_acc >= 0.0 && alt_ok(a, s0, nd.w) == all && alt_ok(a, s1, nd.w) == any)) verdict = 0;
      }
      const unsigned open = __ballot_sync(0xffffffffu, tid < c && !verdict);
      int ob = 0;
      if (lane == 0 && open) ob = atomicAdd(&s_nopen, __popc(open));
      ob = __shfl_sync(0xffffffffu, ob, 0);
      if ((open >> lane) & 1u) s_open[ob + __popc(open & ((1u << lane) - 1u))] = tid;
      __syncthreads();
      for (int kk = sl; kk < s_nopen; kk += nsl) {
        const int k = s_open[kk], v = head + k, row = vrow[v];
        const double4 nd = a.nodec[vnode[v]];
        int na = 0, nr = 0;
#pragma unroll
        for (int i = 0; i < MAXJ; i++) {
          const int j = j0 + QW * i;
          if (j >= W || (i > 0 && wp != QW)) break;
          const unsigned m = row < 0 ? live(j) : R[(size_t)row * W + j];
          unsigned am = 0;
          if (m) {
            bool ok = false;
            if ((m >> lane) & 1u) {
              const double dx = dsub(x[i], nd.x), dy = dsub(y[i], nd.y), dz = dsub(z[i], nd.z);
              const double s = dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
              ok = nd.w < dmul(macc, dsub(dadd(s, madd), msub));
              if (a.has_alt) differ |= ok != alt_ok(a, s, nd.w);
            }
            am = __ballot_sync(0xffffffffu, ok);
          }
          if (lane == 0) R[(size_t)v * W + j] = m & ~am;
          na += __popc(am);
          nr += __popc(m & ~am);
        }
        if (lane == 0) {
          if (na) atomicAdd(&s_ac[k], na);
          if (nr) atomicAdd(&s_rc[k], nr);
        }
      }
      __syncthreads();
      // one thread per node: its entry and its children, by prefix sums (far | near | children)
      const int v = head + tid;
      int nacc = 0, nrej = 0, nch = 0;
      bool leaf = false;
      int2 kd{};
      if (tid == 0) s_nopen = 0;
      int rej = v;
      if (tid < c) {
        nacc = s_ac[tid];
        nrej = s_rc[tid];
        if (verdict) {
          const int row = vrow[v], cnt = row < 0 ? tc : vrc[row];
          nacc = verdict > 0 ? cnt : 0;
          nrej = cnt - nacc;
          rej = row;
        }
        vrej[v] = rej;
        if (nrej) {
          kd = a.kids[vnode[v]];
          leaf = kd.x < 0;
          nch = leaf ? 0 : kd.y;
        }
        vac[v] = nacc;
        vrc[v] = nrej;
      }
      const long long mine = (nacc > 0) | (long long)leaf << 21 | (long long)nch << 42;
      long long inc = mine;
      for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (lane == 31) s_ws[w] = inc;
      __syncthreads();
      long long before = 0, all = 0;
      for (int q = 0; q < QW; q++) {
        if (q < w) before += s_ws[q];
        all += s_ws[q];
      }
      before += inc - mine;
      constexpr long long F = (1 << 21) - 1;
      full = tail + (int)(all >> 42) > vcap;
      if (!full) {
        if (nacc) {
          fref[nf + (int)(before & F)] = v;
          fp += nacc;
        }
        if (leaf) {
          nref[nn + (int)((before >> 21) & F)] = v;
          np += (unsigned long long)nrej * kd.y;
        }
        const int cb = tail + (int)(before >> 42);
        for (int q = 0; q < nch; q++) {
          vnode[cb + q] = kd.x + q;
          vrow[cb + q] = rej;
        }
        head += c;
        tail += (int)(all >> 42);
        nf += (int)(all & F);
        nn += (int)((all >> 21) & F);
      }
      __syncthreads();  // the region's new records; the counts are read
    }
    if (tid == 0) atomicMax(a.visits, (unsigned long long)tail);
    if (full) {
      if (tid == 0) atomicOr(a.err, 1);
      continue;
    }
    for (int o = 16; o; o >>= 1) {
      fp += __shfl_xor_sync(0xffffffffu, fp, o);
      np += __shfl_xor_sync(0xffffffffu, np, o);
    }
    if (lane == 0) {
      if (fp) atomicAdd(&s_pairs[0], fp);
      if (np) atomicAdd(&s_pairs[1], np);
    }
    __syncthreads();
    if (tid == 0) {
      atomicAdd(&a.pairs[0], s_pairs[0]);
      atomicAdd(&a.pairs[1], s_pairs[1]);
      a.g_near[g] = s_pairs[1];
      s_base[0] = atomicAdd(&a.totals[0], (unsigned long long)nf);
      s_base[1] = atomicAdd(&a.totals[1], (unsigned long long)nf * W);
      s_base[2] = atomicAdd(&a.totals[2], (unsigned long long)nn);
      s_base[3] = atomicAdd(&a.totals[3], (unsigned long long)nn * W);
      // the arrays were sized from an estimate: past their end, the build is run again
      if (s_base[0] + nf > a.cap[0] || s_base[1] + (unsigned long long)nf * W > a.cap[1] ||
          s_base[2] + nn > a.cap[2] || s_base[3] + (unsigned long long)nn * W > a.cap[3]) {
        atomicOr(a.err, 2);
        s_base[0] = ~0ull;
      }
      a.far_off[g] = (long long)s_base[0];
      a.far_moff[g] = (long long)s_base[1];
      a.near_off[g] = (long long)s_base[2];
      a.near_moff[g] = (long long)s_base[3];
      a.far_cnt[g] = nf;
      a.near_cnt[g] = nn;
    }
    __syncthreads();
    if (s_base[0] == ~0ull) continue;
    const long long fo = (long long)s_base[0], fmo = (long long)s_base[1], no = (long long)s_base[2],
                    nmo = (long long)s_base[3];
    for (int k = tid; k < nf; k += QT) {
      const int v = fref[k];
      a.far_node[fo + k] = vnode[v];
      a.far_tgt[fo + k] = (unsigned short)vac[v];
    }
    for (int k = tid; k < nn; k += QT) {
      const int v = nref[k];
      a.near_node[no + k] = vnode[v];
      a.near_tgt[no + k] = (unsigned short)vrc[v];
    }
    // a warp per entry, a lane per word
    for (int k = w; k < nf + nn; k += QW) {
      const int v = k < nf ? fref[k] : nref[k - nf];
      if (lane < W) {
        auto row = [&](int q) { return q < 0 ? live(lane) : R[(size_t)q * W + lane]; };
        const unsigned r = vrc[v] ? row(vrej[v]) : 0u;
        if (k < nf) a.far_mask[fmo + (long long)k * W + lane] = row(vrow[v]) & ~r;
        else a.near_mask[nmo + (long long)(k - nf) * W + lane] = r;
      }
    }
    __syncthreads();  // the entries' nodes and targets
    group_shares(a, g, nf, fo, (long long)s_pairs[0], nn, no);
  }
  if (a.has_alt && __any_sync(0xffffffffu, differ) && lane == 0) atomicOr(a.err, 4);
}

}  // namespace

// Groups for particle targets.  G = 0: each leaf, in chunks of at most kGroupMax targets.
// G > 0: runs of consecutive leaves (in tree order, which keeps them spatially close:
// siblings and cousins) of one system, up to G targets together; a leaf larger than G is
// cut into chunks of G.  Packed small leaves share one traversal, one set of entries and
// the near field's source tiles, but each near entry then covers fewer targets; which is
// faster depends on the workload (bit_b200.autotune measures it).
static void particle_groups(Tree* t, int G, std::vector<int>& ts, std::vector<int>& tc,
                            std::vector<int>& sys) {
  if (G <= 0) {
    for (int i = 0; i < t->numtree; i++) {
      if (t->h_children[8LL * i] != -1) continue;
      const int st = t->h_start[i], en = st + t->h_nummemb[i];
      for (int e = st; e < en; e += kGroupMax) {
        ts.push_back(e);
        tc.push_back(std::min(kGroupMax, en - e));
        sys.push_back(t->h_node_sys[i]);
      }
    }
    return;
  }
  std::vector<int> leaves;
  for (int i = 0; i < t->numtree; i++)
    if (t->h_children[8LL * i] == -1) leaves.push_back(i);
  std::sort(leaves.begin(), leaves.end(),
            [&](int a, int b) { return t->h_start[a] < t->h_start[b]; });
  int cur0 = -1, curn = 0, cursys = -1;
  auto flush = [&] {
    if (curn > 0) {
      ts.push_back(cur0);
      tc.push_back(curn);
      sys.push_back(cursys);
    }
    curn = 0;
  };
  for (int i : leaves) {
    const int st = t->h_start[i], cnt = t->h_nummemb[i], sy = t->h_node_sys[i];
    if (cnt > G) {
      flush();
      for (int e = st; e < st + cnt; e += G) {
        ts.push_back(e);
        tc.push_back(std::min(G, st + cnt - e));
        sys.push_back(sy);
      }
      continue;
    }
    if (curn > 0 && (sy != cursys || curn + cnt > G || cur0 + curn != st)) flush();
    if (curn == 0) {
      cur0 = st;
      cursys = sy;
    }
    curn += cnt;
  }
  flush();
}

// Points per group: as few as make six groups a multiprocessor, in powers of two from a mask
// word to kPointGroup.  A small group shares less (traversal, coefficients, sources), but few
// groups leave the chip idle.  A whole call on 200k particles (nterms 9, screened, FP64), groups
// of 32 / 64 / 128 / 256, us: 300 points 516 / 711 / 1093 / 1739; 10k 635 / 721 / 844 / 1112;
// 27k 786 / 801 / 1006 / 1121; 40k 1008 / 922 / 1110 / 1271; 60k 1366 / 1155 / 1160 / 1416; 140k
// 3737 / 3232 / 3072 / 3002; 1M 22256 / 18659 / 17114 / 15959; other trees and kernels cross at
// 20k to 27k, 50k to 60k and 100k to 130k.
static int point_group(int m, int sms) {
  int size = 32;
  while (size < kPointGroup && m > 6LL * sms * size) size *= 2;
  return size;
}

// Targets of a CTA: `top`, or less where the groups' chunks of that size would be fewer than
// `enough`.
static int chunk_size(const std::vector<int>& tc, int top, long long enough) {
  for (int size = top; size > 32; size /= 2) {
    long long chunks = 0;
    for (int k : tc) chunks += (k + size - 1) / size;
    if (chunks >= enough) return size;
  }
  return 32;
}
// The potentials' far kernel (two CTAs of eight warps a multiprocessor): whole groups from 1.25
// chunks a multiprocessor.  A chunk reads its group's coefficients again.  Screened / with delta,
// FP64, chunks of 32 / 64 / 128 / 256 / 512 / whole groups, us: 20k in leaves of 500 (64 groups)
// 67, 76 / 55, 61 / 47, 60 / 54, 65 / 63, 77 / 63, 78; 50k, 1000 (64) 109, 122 / 74, 86 / 63, 77 / 63, 83 /
// 83, 102 / 112, 143; 10k, 200 (64) 44, 49 / 37, 43 / 41, 49 / 41, 49 / 43, 49 / 43, 49; 50k, 300 (260)
// 156, 178 / 119, 135 / 101, 120 / 95, 118 / 100, 127 / 102, 127; 200k, 500 (750) 698, 807 / 463, 552 / 337,
// 427 / 277, 362 / 246, 334 / 248, 339.
static int far_chunk(const std::vector<int>& tc, int sms) { return chunk_size(tc, kGroupMax, 5LL * sms / 4); }
// The fields' kernels, which keep three sums a target and warp: at most kFieldChunk, and from
// 2.5 chunks a multiprocessor.  Far + near, FP64 Coulomb field, chunks of 32 / 64 / 128 / 256, us:
// 2k in leaves of 500 61 / 78 / 96 / 132; 8k, 300: 100 / 108 / 136 / 197; 20k, 200: 168 / 153 / 180 /
// 186; 50k, 300: 460 / 388 / 392 / 485; 100k, 300: 854 / 667 / 587 / 600; 150k, 600: 1817 / 1361 / 1138 /
// 1045; 2M, 1000, ms: 42.8 / 31.0 / 25.2 / 22.3 (whole groups: 25.2).
static int field_chunk(const std::vector<int>& tc, int sms) { return chunk_size(tc, kFieldChunk, 5LL * sms / 2); }

// The near-field items, heaviest first: a group's near work in one item, or in up to kNearParts
// equal parts of at least `chunk` pairs each, whose sums meet in scratch (near_part).  A part
// packs its targets for fewer sources, so parts are only as many as give a system four items a
// multiprocessor: chunk is a share of the system's pairs, between kNearChunkMin and kNearChunk
// (groups of packed leaves, set for throughput: kNearChunk).  Screened FP64 / mixed, us, chunks
// of 512k against this: 20k in leaves of 500 359 / 121 -> 117 / 68; 50k, 300: 426 / 160 -> 248 / 144; 10k,
// 200: 89 / 51 -> 46 / 41; 200k, 500: 1332 / 470 either way; 64k for all: 1369 / 559 at 200k, 17.3 for 17.0
// ms at 2M, 48 packed systems 3.2 for 2.8 ms.  (Cutting a group's targets instead gave nothing: most
// lists are short.)  The count follows from the system's own lists alone, so that its result does
// not depend on what else is evaluated, nor on the memory budget: without room for the scratch a
// group's first item takes the parts one after the other (near.cu), the same sums, later.
static void near_items(Lists* L, Ctx* c, const std::vector<unsigned long long>& pairs,
                       const std::vector<int>& tc, const std::vector<int>& sys, bool packed) {
  const int ng = (int)pairs.size();
  std::vector<int> K(ng);
  std::vector<unsigned long long> of_sys(ng ? 1 + *std::max_element(sys.begin(), sys.end()) : 0, 0);
  for (int g = 0; g < ng; g++) of_sys[sys[g]] += pairs[g];
  auto chunk = [&](int s) {
    const unsigned long long share = of_sys[s] / (unsigned long long)(4 * c->num_sms);
    return packed ? (unsigned long long)kNearChunk
                  : std::min<unsigned long long>(kNearChunk, std::max<unsigned long long>(kNearChunkMin, share));
  };
  std::vector<long long> off(ng, 0);
  long long tot = 0;
  for (int g = 0; g < ng; g++) {
    K[g] = (int)std::max(1ull, std::min<unsigned long long>(kNearParts, pairs[g] / chunk(sys[g])));
    off[g] = tot;
    if (K[g] > 1) tot += (long long)K[g] * tc[g];
  }
  L->part_total = tot;
  std::vector<std::pair<unsigned long long, int2>> it;
  for (int g = 0; g < ng; g++)
    for (int k = 0; k < K[g]; k++) it.push_back({pairs[g] / K[g], make_int2(g, k | K[g] << 16)});
  std::stable_sort(it.begin(), it.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
  L->h_items.resize(it.size());
  for (size_t i = 0; i < it.size(); i++) L->h_items[i] = it[i].second;
  cudaStream_t s = c->stream;
  L->items.ensure(c, it.size());
  L->part_off.ensure(c, ng);
  L->part_done.ensure(c, ng);
  BIT_CUDA(cudaMemcpyAsync(L->items.p, L->h_items.data(), it.size() * sizeof(int2), cudaMemcpyHostToDevice, s));
  BIT_CUDA(cudaMemcpyAsync(L->part_off.p, off.data(), ng * sizeof(long long), cudaMemcpyHostToDevice, s));
  BIT_CUDA(cudaMemsetAsync(L->part_done.p, 0, ng * sizeof(int), s));
  BIT_CUDA(cudaStreamSynchronize(s));  // the host arrays are done with
}

void build_lists(Tree* t, Lists* L, const ListKey& key, int ntargets, const double* tx,
                 const double* ty, const double* tz, const SysEval* d_sys, const ListKey* alt) {
  if (alt && (!alt->sysmac.empty() || !key.sysmac.empty() || t->nsys != 1)) alt = nullptr;
  L->valid = false;  // the arrays are rewritten below; valid again once the build completes
  L->alt_valid = false;
  Ctx* c = t->ctx;
  cudaStream_t s = c->stream;
  std::vector<int> ts, tc, gsys;
  if (key.points) {
    if (t->nsys != 1) fail(BIT_ERR_INVALID_ARGUMENT, "external points need a single-system tree");
    const int size = point_group(ntargets, c->num_sms);
    for (int e = 0; e < ntargets; e += size) {
      ts.push_back(e);
      tc.push_back(std::min(size, ntargets - e));
      gsys.push_back(0);
    }
  } else {
    particle_groups(t, key.group, ts, tc, gsys);
  }
  const int ng = (int)ts.size();
  L->ngroups = ng;
  L->ntargets = ntargets;
  L->g_tstart.ensure(c, ng);
  L->g_tcount.ensure(c, ng);
  BIT_CUDA(cudaMemcpyAsync(L->g_tstart.p, ts.data(), ng * sizeof(int), cudaMemcpyHostToDevice, s));
  BIT_CUDA(cudaMemcpyAsync(L->g_tcount.p, tc.data(), ng * sizeof(int), cudaMemcpyHostToDevice, s));
  L->g_sys.ensure(c, ng);
  BIT_CUDA(cudaMemcpyAsync(L->g_sys.p, gsys.data(), ng * sizeof(int), cudaMemcpyHostToDevice, s));
  L->h_g_sys = gsys;
  L->far_off.ensure(c, ng);
  L->near_off.ensure(c, ng);
  L->far_moff.ensure(c, ng);
  L->near_moff.ensure(c, ng);
  L->far_cnt.ensure(c, ng);
  L->near_cnt.ensure(c, ng);
  L->g_near.ensure(c, ng);
  DBuf<unsigned long long> cnt;  // totals[4], pairs[2], err (as the 7th word), most visits
  cnt.ensure(c, 8);
  ListArgs a{};
  a.g_tstart = L->g_tstart.p;
  a.g_tcount = L->g_tcount.p;
  a.tx = tx; a.ty = ty; a.tz = tz;
  a.nodec = t->nodec.p;
  a.kids = t->kids.p;
  a.sys = d_sys;
  a.g_sys = L->g_sys.p;
  a.far_off = L->far_off.p; a.near_off = L->near_off.p;
  a.far_moff = L->far_moff.p; a.near_moff = L->near_moff.p;
  a.far_cnt = L->far_cnt.p; a.near_cnt = L->near_cnt.p;
  a.g_near = L->g_near.p;
  a.totals = cnt.p;
  a.pairs = cnt.p + 4;
  a.err = reinterpret_cast<int*>(cnt.p + 6);
  if (alt) {
    a.has_alt = 1;
    a.alt_acc = alt->acc;
    a.alt_add = alt->add_del;
    a.alt_sub = alt->sub_del;
  }
  long long words = 0;
  for (int g = 0; g < ng; g++) words += (tc[g] + 31) / 32;
  // sizes of this tree's last build, else of the context's last build under the same MAC
  const ListSizing* hint = L->last.ngroups > 0 ? &L->last : nullptr;
  if (!hint && c->list_hint.ngroups > 0 && c->list_hint.acc == key.acc &&
      c->list_hint.points == key.points)
    hint = &c->list_hint;
  unsigned long long cap[4];
  if (hint) {
    const double f = 1.25 * (double)ng / hint->ngroups;
    for (int k = 0; k < 4; k++) cap[k] = (unsigned long long)(f * hint->totals[k]) + 1024;
  } else {
    cap[0] = 192ull * ng + 1024;
    cap[1] = 192ull * words + 1024;
    cap[2] = 48ull * ng + 1024;
    cap[3] = 48ull * words + 1024;
  }
  // one region per resident CTA; a group visits a node once at most
  int maxw = 1;
  for (int g = 0; g < ng; g++) maxw = std::max(maxw, (tc[g] + 31) / 32);
  L->max_targets = 32 * maxw;
  L->field_chunk = field_chunk(tc, c->num_sms);
  L->far_chunk = far_chunk(tc, c->num_sms);
  int per_sm = 0;
  BIT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lists, QT, 0));
  const long long nodes = std::max(t->numtree, 1);
  long long visits = std::min(nodes, hint && hint->visits > 0 ? hint->visits + hint->visits / 4 + 64 : kVisitsFirst);
  L->far_cut.ensure(c, (size_t)ng * kFarWarps);
  L->near_tot.ensure(c, ng);
  L->head.ensure(c, 1);
  a.far_cut = L->far_cut.p; a.near_tot = L->near_tot.p;
  a.visits = cnt.p + 7;
  a.head = L->head.p;
  a.ngroups = ng;
  unsigned long long h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  std::vector<int> hf(ng), hn(ng);
  std::vector<unsigned long long> hp(ng);
  int err = 0;
  L->fallback = false;
  for (;;) {
    L->far_node.ensure(c, cap[0]);
    L->far_mask.ensure(c, cap[1]);
    L->near_node.ensure(c, cap[2]);
    L->near_mask.ensure(c, cap[3]);
    L->far_tgt.ensure(c, L->far_node.n);
    L->near_tgt.ensure(c, L->near_node.n);
    L->near_pre.ensure(c, L->near_node.n / 32 + 1);
    for (int k = 0; k < 4; k++) a.cap[k] = cap[k];
    a.far_node = L->far_node.p; a.far_mask = L->far_mask.p;
    a.near_node = L->near_node.p; a.near_mask = L->near_mask.p;
    a.far_tgt = L->far_tgt.p; a.near_tgt = L->near_tgt.p;
    a.near_pre = L->near_pre.p;
    const long long per = (long long)(maxw + kVisitWords) * sizeof(unsigned);  // bytes a visit
    const size_t room = std::min(kRegionBytes, std::max(L->gstage.n * sizeof(unsigned), ctx_room(c)));
    a.stage = visits * (maxw + kVisitWords);
    long long slots = std::min<long long>(ng, (long long)c->num_sms * std::max(per_sm, 1));
    slots = std::min<long long>(slots, room / (visits * per));
    slots = std::max(slots, 1LL);
    L->gstage.ensure(c, (size_t)slots * (size_t)a.stage);
    a.gstage = L->gstage.p;
    BIT_CUDA(cudaMemsetAsync(cnt.p, 0, 8 * sizeof(unsigned long long), s));
    BIT_CUDA(cudaMemsetAsync(L->head.p, 0, sizeof(int), s));
    count_launch(), k_lists<<<(unsigned)slots, QT, 0, s>>>(a);
    BIT_CHECK_LAUNCH();
    copy_d2h_batch(c, {{h, cnt.p, 8 * sizeof(unsigned long long)},
                       {hf.data(), L->far_cnt.p, ng * sizeof(int)},
                       {hn.data(), L->near_cnt.p, ng * sizeof(int)},
                       {hp.data(), L->g_near.p, ng * sizeof(unsigned long long)}});
    err = (int)(h[6] & 0xffffffffu);
    if (!(err & 3)) break;
    L->fallback = true;
    if (err & 1) visits = std::min(nodes, 4 * visits);  // (the totals are not complete)
    else for (int k = 0; k < 4; k++) cap[k] = h[k];
  }
  if (key.points) L->gstage.release();  // (dev_alloc finds the trees' own lists only)
  ListSizing& z = L->last;
  z.ngroups = ng;
  z.acc = key.acc;
  z.points = key.points;
  for (int k = 0; k < 4; k++) z.totals[k] = h[k];
  z.visits = (long long)h[7];
  c->list_hint = z;
  L->nfar = (long long)h[0];
  L->nnear = (long long)h[2];
  L->far_pairs = (long long)h[4];
  L->near_pairs = (long long)h[5];
  // heaviest groups first, so the evaluation kernels' tail is short
  std::vector<int> ord(ng);
  std::iota(ord.begin(), ord.end(), 0);
  std::vector<long long> wk(ng);
  for (int g = 0; g < ng; g++) wk[g] = (40LL * hf[g] + hn[g]) * (long long)tc[g];
  std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return wk[x] > wk[y]; });
  L->h_work = wk;
  L->order.ensure(c, ng);
  BIT_CUDA(cudaMemcpyAsync(L->order.p, ord.data(), ng * sizeof(int), cudaMemcpyHostToDevice, s));
  near_items(L, c, hp, tc, gsys, key.group > 0 && !key.points);  // (synchronises)
  L->key = key;
  L->valid = true;
  L->version++;
  L->alt_valid = alt && !(err & 4);
  if (L->alt_valid) {
    L->alt_key = key;
    L->alt_key.acc = alt->acc;
    L->alt_key.add_del = alt->add_del;
    L->alt_key.sub_del = alt->sub_del;
  }
}

}  // namespace bit
