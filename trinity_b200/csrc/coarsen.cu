/*
 * coarsen.cu — edge collapse (Coarse::run body, coarsening.cpp:480-503).
 *
 *   k_coarse_pre     activity flags: corners -1, live vertices 1, others 0;
 *                    clear repair tags (coarsening.cpp:257-281)
 *   k_coarse_filter  per active vertex: the shortest collapse target among
 *                    neighbours closer than 1/sqrt(2) whose simulated collapse
 *                    keeps every surviving element CCW with edges <= sqrt(2)
 *                    (Coarse::identifyTarget, coarsening.cpp:47-133); ties are
 *                    broken in adjacency order, like the reference's multimap
 *   k_coarse_filter_group  the same search by 4, 8 or 16 lanes per vertex, for
 *                    levels that list few vertices (free mode)
 *   k_collapse       per independent vertex: erase the 1-2 shell elements,
 *                    move the rest of the stencil to the target, relabel,
 *                    tag repairs, re-activate the 1-ring (Coarse::collapseEdge,
 *                    coarsening.cpp:136-254 with Mesh::copyStencil mesh.cpp:497)
 * Independent sources touch disjoint elements, so the collapses of one level
 * run in parallel; appends to a shared target's stencil are atomic and the
 * repair pass sorts them.
 */
#include "trn_internal.h"
#include "trn_level.cuh"
#include "trn_mixed.cuh"

#include <algorithm>

namespace trn {

/* with `act`, the active vertices also go onto the list act (free mode's
 * first level; the list is unordered by design) */
__global__ void k_coarse_pre(DMesh m, int nb_nodes, int* __restrict__ act, int* act_n) {
  nb_nodes = trn_nodes(m, nb_nodes);
  for (int base = blockIdx.x * blockDim.x; base < nb_nodes; base += trn_grid_stride()) {
    const int v = base + threadIdx.x;
    int8_t a = 0;
    if (v < nb_nodes) {
      if (m.tags[v] & TRN_TAG_CORNER) a = -1;
      else a = m.alive[v] ? 1 : 0;
      m.activ[v] = a;
      m.fixes[v] = 0;
    }
    if (act) trn_block_append(act, act_n, v, a > 0);
  }
}

/* is the collapse of source onto destin valid: every element that remains
 * CCW with no edge longer than sqrt(2)? The destination's point and tensor are
 * the caller's, so an element costs two gathers of each. */
template <bool F32>
__device__ __forceinline__ bool collapse_valid(const DMesh& m, int source, int destin, const TrnRow& st, int deg,
                                               bool both_bound, double2 pd, TenT<F32> td) {
  int shared = 0;
  for (int k = 0; k < deg; ++k) {
    const int4 n = m.tri[st[k]];
    const int pos = n.x == source ? 0 : (n.y == source ? 1 : 2);
    const int a = pos == 0 ? n.y : (pos == 1 ? n.z : n.x);
    const int b = pos == 0 ? n.z : (pos == 1 ? n.x : n.y);
    if (a == destin || b == destin) {
      if (++shared > 1 && both_bound) return false;
      continue;
    }
    const double2 pa = m.pts[a], pb = m.pts[b];
    if (!trn_ccw_from(pd, pa, pb, pos)) return false;
    const TenT<F32> ta = ten_load<F32>(m, a), tb = ten_load<F32>(m, b);
    if (length_gt<F32>(pd, pa, td, ta, TRN_L_MAX) || length_gt<F32>(pb, pd, tb, td, TRN_L_MAX) ||
        length_gt<F32>(pa, pb, ta, tb, TRN_L_MAX))
      return false;
  }
  return true;
}

/* A lane's array for whichever serial path it takes: the device reserves the
 * deepest stack for every thread it can hold (0.3 GB a KB on 148
 * multiprocessors), so the paths share one. Candidates are places in the
 * source's row, which a byte holds (bucket <= 256). */
union SerialBuf {
  int ids[2 * TRN_MAX_DEG];   /* build_one_vicin; the repair and the collapse use half */
  struct {
    float lo[TRN_MAX_DEG], hi[TRN_MAX_DEG];
    uint8_t at[TRN_MAX_DEG];
  } cand;
};

/* The candidates are tried by increasing upper bound of their length
 * (length_below), and the exact length is computed only between two valid
 * ones whose bounds overlap: the pick is the valid one of smallest (length,
 * adjacency index), as the reference's multimap gives it. */
template <bool F32>
__device__ __forceinline__ int identify_target(const DMesh& m, int source, SerialBuf& buf) {
  const bool bound_source = (m.tags[source] & TRN_TAG_BOUND) != 0;
  float* lo = buf.cand.lo;
  float* hi = buf.cand.hi;
  uint8_t* at = buf.cand.at;
  int nc = 0;
  const TrnRow vc = trn_row(m.vic, m, source);
  const int nv = m.vdeg[source];
  const double2 ps = m.pts[source];
  const TenT<F32> ts = ten_load<F32>(m, source);
  for (int b = 0; b < nv; ++b) {
    const int neigh = vc[b];
    if (bound_source && !(m.tags[neigh] & TRN_TAG_BOUND)) continue;
    float l, h;
    if (length_below<F32>(ps, m.pts[neigh], ts, ten_load<F32>(m, neigh), TRN_L_MIN, &l, &h)) {
      int p = nc;
      while (p > 0 && hi[p - 1] > h) {
        hi[p] = hi[p - 1];
        lo[p] = lo[p - 1];
        at[p] = at[p - 1];
        --p;
      }
      hi[p] = h;
      lo[p] = l;
      at[p] = (uint8_t) b;
      nc++;
    }
  }
  const TrnRow st = trn_row(m.stenc, m, source);
  const int deg = trn_deg(m, source);
  int best = -1;
  float best_hi = 0.f;
  for (int k = 0; k < nc; ++k) {
    if (best >= 0 && lo[k] > best_hi) continue;   /* certainly longer */
    const int c = vc[at[k]];
    const bool both = bound_source && (m.tags[c] & TRN_TAG_BOUND) != 0;
    const double2 pc = m.pts[c];
    const TenT<F32> tc = ten_load<F32>(m, c);
    if (!collapse_valid<F32>(m, source, c, st, deg, both, pc, tc)) continue;
    if (best < 0) {
      best = c;
      best_hi = hi[k];
      continue;
    }
    LenT<F32> s1, r1;
    const LenT<F32> s0 = length_squares<F32>(ps, pc, ts, tc, &s1);
    const LenT<F32> r0 = length_squares<F32>(ps, m.pts[best], ts, ten_load<F32>(m, best), &r1);
    const double lc = (double) length_of_squares(s0, s1), lb = (double) length_of_squares(r0, r1);
    if (lc < lb || (lc == lb && c < best)) {   /* rows are in id order */
      best = c;
      best_hi = hi[k] > best_hi ? hi[k] : best_hi;
    }
  }
  return best;
}

template <bool F32>
__global__ void k_coarse_filter(DMesh m, int nb_nodes, int* __restrict__ target,
                                uint8_t* __restrict__ flag) {
  nb_nodes = trn_nodes(m, nb_nodes);
  if (trn_failed(m)) return;
  SerialBuf buf;
  for (int v = trn_tid(); v < nb_nodes; v += trn_grid_stride()) {
    uint8_t f = 0;
    if (m.activ[v] > 0) {
      m.activ[v] = 0;
      int t = identify_target<F32>(m, v, buf);
      target[v] = t;
      f = t > -1 ? 1 : 0;
    }
    flag[v] = f;
  }
}

/* any block size of the tuner's, which caps the registers at 64: 32 warps an
 * SM to hide the scan's gathers. 2M-triangle workload, coarsening of three
 * rounds: 8.98 ms at two 256-thread blocks, 8.41 at three, 8.31 at four; with
 * the scan that computed every candidate's length, gathered three corners an
 * element and tested lengths with roots and logarithms, 10.08 ms. */
constexpr int kSearchThreads = 1024;

/* free mode: one pass per level rebuilds the adjacency of each active vertex,
 * finds its target and appends the candidates (in no particular order: the
 * independent set is chosen by hashed priorities, not by list position),
 * marking them undecided for the independent-set rounds */
template <bool F32>
__global__ void __launch_bounds__(kSearchThreads) k_coarse_filter_append(DMesh m, const int* __restrict__ act, const int* act_n,
                                       int* __restrict__ target, int* __restrict__ cand, int* count,
                                       uint8_t* __restrict__ state, int min_n) {
  if (blockIdx.x == 0 && threadIdx.x == 0) trn_level_clear(m, nullptr);
  if (trn_failed(m)) return;
  const int n = *act_n;
  if (n < min_n) return;
  SerialBuf buf;
  /* warp-aggregated appends: a block-wide one would make every thread wait
   * for its block's longest search at each step */
  for (int q = trn_tid(); q < n; q += trn_grid_stride()) {
    const int v = act[q];
    if (m.activ[v] <= 0) continue;
    m.activ[v] = 0;
    build_one_vicin(m, v, buf.ids);
    const int t = identify_target<F32>(m, v, buf);
    target[v] = t;
    if (t > -1) {
      state[v] = 1;
      trn_append(cand, count, v);
    }
  }
}

/* build_one_vicin by G lanes, two elements a lane: the elements' next
 * vertices, and the one previous vertex that is no next one (a boundary
 * vertex), are the neighbours; a neighbour's place is the number of smaller
 * ones, counted by shuffles. Longer or irregular stencils by the group's first
 * lane. v < 0: no vertex; all lanes of the warp call it. */
template <int G>
__device__ __forceinline__ void build_vicin_group(const DMesh& m, int v, SerialBuf& buf) {
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), g0 = lane & ~(G - 1);
  const unsigned gm = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << g0;
  const int deg = v >= 0 && m.alive[v] ? trn_deg(m, v) : 0;
  bool odd = deg > 2 * G;
  int a[2], b[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = gl + h * G;
    a[h] = b[h] = 0x7fffffff;
    if (k < deg && !odd) {
      const int e = trn_row(m.stenc, m, v)[k];
      const int4 n = e >= 0 ? m.tri[e] : make_int4(-1, -1, -1, 0);
      a[h] = v == n.x ? n.y : (v == n.y ? n.z : n.x);
      b[h] = v == n.x ? n.z : (v == n.y ? n.x : n.y);
      odd |= !(v == n.x || v == n.y || v == n.z);
    }
  }
  /* uniform over the warp: how many entries any of its vertices has */
  const int most = __reduce_max_sync(0xffffffffu, odd ? 0 : deg);
  int rank[2] = {0, 0};
  bool found[2] = {false, false};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h * G >= most) break;
    for (int k = 0; k < G; ++k) {
      if (h * G + k >= most) break;
      const int x = __shfl_sync(0xffffffffu, a[h], k, G);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        rank[o] += x < a[o];
        found[o] |= x == b[o];
        odd |= a[o] != 0x7fffffff && x == a[o] && (h * G + k) != (o * G + gl);
      }
    }
  }
  int extra = 0, x = 0x7fffffff;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const unsigned miss = __ballot_sync(0xffffffffu, b[h] != 0x7fffffff && !found[h]) & gm;
    const int from = __shfl_sync(0xffffffffu, b[h], miss ? __ffs(miss) - 1 : 0);
    if (miss) x = from;
    extra += __popc(miss);
  }
  const bool serial = (__ballot_sync(0xffffffffu, odd || extra > 1 || deg + extra > m.bucket) & gm) != 0;
  if (!serial && v >= 0) {
    const TrnRow row = trn_row(m.vic, m, v);
    int below = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (a[h] != 0x7fffffff) {
        row[rank[h] + (extra && x < a[h] ? 1 : 0)] = a[h];
        below += a[h] < x;
      }
    if (extra) {
#pragma unroll
      for (int o = G / 2; o >= 1; o >>= 1) below += __shfl_xor_sync(gm, below, o);
      if (gl == 0) row[below] = x;
    }
    if (gl == 0) m.vdeg[v] = deg + extra;
  } else if (serial && gl == 0) {
    build_one_vicin(m, v, buf.ids);
  }
  __syncwarp();
}

/* the same search by a group of G lanes per vertex, for the levels that
 * list few vertices, where one lane's chain of dependent gathers (adjacency,
 * stencil, triangles, points, tensors) sets the time. The lanes compute the
 * neighbours' metric lengths, then check every (candidate, element) pair at
 * once; the per-candidate verdicts are combined as bit masks, and the pick is
 * the smallest (length, adjacency index) among the valid candidates, which is
 * the first valid one in the serial search's stable length order, so the
 * targets are the same. Vertices with more than 32 neighbours fall back to
 * the serial search on the group's first lane. v (the same on all lanes of a
 * group, < 0: no vertex) gets its adjacency row too; all lanes of the warp
 * call it, and the group's first lane receives the target. */
template <bool F32, int G>
__device__ __forceinline__ int search_group(const DMesh& m, int v, SerialBuf& buf) {
  const int lane = threadIdx.x & 31;
  const int gl = lane & (G - 1);
  build_vicin_group<G>(m, v, buf);
  const int nv = v >= 0 ? m.vdeg[v] : 0;
  const bool serial = nv > 32;
  const bool grp = v >= 0 && !serial;
  const TrnRow vc = trn_row(m.vic, m, (v >= 0 ? v : 0));
  const TrnRow st = trn_row(m.stenc, m, (v >= 0 ? v : 0));
  const bool bsrc = v >= 0 && (m.tags[v] & TRN_TAG_BOUND) != 0;
  double2 ps = make_double2(0, 0);
  TenT<F32> ts{};
  if (grp) {
    ps = m.pts[v];
    ts = ten_load<F32>(m, v);
  }
  /* neighbours b = gl + G * k: candidates closer than 1/sqrt(2) */
  double lenk[32 / G];
  unsigned candm = 0, boundm = 0;
  for (int k = 0; k < 32 / G; ++k) {
    const int b = gl + G * k;
    lenk[k] = 0.0;
    if (grp && b < nv) {
      const int w = vc[b];
      const bool bd = (m.tags[w] & TRN_TAG_BOUND) != 0;
      if (bd) boundm |= 1u << b;
      if (!(bsrc && !bd)) {
        double len;
        if (length_lt<F32>(ps, m.pts[w], ts, ten_load<F32>(m, w), TRN_L_MIN, &len)) {
          candm |= 1u << b;
          lenk[k] = len;
        }
      }
    }
  }
  for (int o = G / 2; o >= 1; o >>= 1) {
    candm |= __shfl_xor_sync(0xffffffffu, candm, o);
    boundm |= __shfl_xor_sync(0xffffffffu, boundm, o);
  }
  /* every (candidate, element) pair of the simulated collapses */
  const int deg = grp ? trn_deg(m, v) : 0;
  const int np = (grp && candm) ? nv * deg : 0;
  const int iters = __reduce_max_sync(0xffffffffu, (np + G - 1) / G);
  unsigned failm = 0, once = 0, twice = 0;
  for (int k = 0; k < iters; ++k) {
    const int p = gl + G * k;
    if (p >= np) continue;
    const int b = p / deg, a = p - b * deg;
    if (!((candm >> b) & 1u)) continue;
    const unsigned bit = 1u << b;
    const int destin = vc[b];
    const int4 e = m.tri[st[a]];
    if ((v == e.x && destin == e.y) || (v == e.y && destin == e.x) || (v == e.y && destin == e.z) ||
        (v == e.z && destin == e.y) || (v == e.z && destin == e.x) || (v == e.x && destin == e.z)) {
      twice |= once & bit;
      once |= bit;
      continue;
    }
    const int f0 = (e.x == v ? destin : e.x);
    const int f1 = (e.y == v ? destin : e.y);
    const int f2 = (e.z == v ? destin : e.z);
    const double2 p0 = m.pts[f0], p1 = m.pts[f1], p2 = m.pts[f2];
    if (trn_ccw(p0, p1, p2)) {
      const TenT<F32> t0 = ten_load<F32>(m, f0), t1 = ten_load<F32>(m, f1), t2 = ten_load<F32>(m, f2);
      if (length_gt<F32>(p0, p1, t0, t1, TRN_L_MAX) || length_gt<F32>(p1, p2, t1, t2, TRN_L_MAX) ||
          length_gt<F32>(p2, p0, t2, t0, TRN_L_MAX))
        failm |= bit;
    } else {
      failm |= bit;
    }
  }
  for (int o = G / 2; o >= 1; o >>= 1) {
    const unsigned fo = __shfl_xor_sync(0xffffffffu, failm, o);
    const unsigned oo = __shfl_xor_sync(0xffffffffu, once, o);
    const unsigned to = __shfl_xor_sync(0xffffffffu, twice, o);
    twice |= to | (once & oo);
    once |= oo;
    failm |= fo;
  }
  const unsigned valid = candm & ~failm & ~(bsrc ? (twice & boundm) : 0u);
  /* the smallest (length, adjacency index) among the valid candidates */
  double best = 0.0;
  int bestb = -1;
  for (int k = 0; k < 32 / G; ++k) {
    const int b = gl + G * k;
    if (b < 32 && ((valid >> b) & 1u) && (bestb < 0 || lenk[k] < best)) {
      best = lenk[k];
      bestb = b;
    }
  }
  for (int o = G / 2; o >= 1; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int obb = __shfl_xor_sync(0xffffffffu, bestb, o);
    if (obb >= 0 && (bestb < 0 || ob < best || (ob == best && obb < bestb))) {
      best = ob;
      bestb = obb;
    }
  }
  if (gl != 0 || v < 0) return -1;
  return serial ? identify_target<F32>(m, v, buf) : (bestb >= 0 ? vc[bestb] : -1);
}

/* the listed vertices by the groups of the warps warp, warp + nwarps, ... */
template <bool F32, int G>
__device__ __forceinline__ void search_list(const DMesh& m, const int* act, int n, int warp, int nwarps, int* target,
                                            int* cand, int* count, uint8_t* state, SerialBuf& buf) {
  constexpr int per_warp = 32 / G;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  for (int base = warp * per_warp; base < n; base += nwarps * per_warp) {
    const int q = base + lane / G;
    int v = q < n ? act[q] : -1;
    if (v >= 0 && m.activ[v] <= 0) v = -1;
    __syncwarp();
    if (gl == 0 && v >= 0) m.activ[v] = 0;
    const int t = search_group<F32, G>(m, v, buf);
    if (gl == 0 && v >= 0) {
      target[v] = t;
      if (t > -1) {
        state[v] = 1;
        trn_append(cand, count, v);
      }
    }
  }
}

template <bool F32, int G>
__global__ void k_coarse_filter_group(DMesh m, const int* __restrict__ act, const int* act_n,
                                      int* __restrict__ target, int* __restrict__ cand, int* count,
                                      uint8_t* __restrict__ state, int max_n) {
  if (blockIdx.x == 0 && threadIdx.x == 0) trn_level_clear(m, nullptr);
  if (trn_failed(m)) return;
  const int n = *act_n;
  if (n > max_n) return;
  SerialBuf buf;
  search_list<F32, G>(m, act, n, trn_tid() >> 5, trn_grid_stride() >> 5, target, cand, count, state, buf);
}

/* one collapse (Coarse::collapseEdge) by one lane: long stencils */
__device__ __noinline__ void collapse_serial(const DMesh& m, int source, int destin, int* rest) {
  const TrnRow st = trn_row(m.stenc, m, source);
  const int deg = trn_deg(m, source);
  const int limit = (m.tags[source] & TRN_TAG_BOUND) ? 1 : 2;
  int k = 0, trash0 = -1, trash1 = -1;
  int opp[2] = {-1, -1};
  for (int a = 0; k < limit && a < deg; ++a) {
    int4 n = m.tri[st[a]];
    int o = -2;
    if ((source == n.x && destin == n.y) || (destin == n.x && source == n.y)) o = n.z;
    else if ((source == n.y && destin == n.z) || (destin == n.y && source == n.z)) o = n.x;
    else if ((source == n.z && destin == n.x) || (destin == n.z && source == n.x)) o = n.y;
    if (o != -2) {
      opp[k] = o;
      if (k == 0) trash0 = a; else trash1 = a;
      ++k;
    }
  }
  int nr = 0;
  for (int a = 0; a < deg; ++a) {
    int e = st[a];
    if (a == trash0 || a == trash1) {
      m.tri[e] = make_int4(-1, -1, -1, 0);
      continue;
    }
    rest[nr++] = e;
  }
  for (int j = 0; j < k; ++j)
    if (opp[j] >= 0) trn_tag_fix(m, opp[j]);
  trn_stenc_append_n(m, destin, rest, nr);
  for (int a = 0; a < nr; ++a) {
    int4 n = m.tri[rest[a]];
    if (n.x == source) n.x = destin;
    else if (n.y == source) n.y = destin;
    else if (n.z == source) n.z = destin;
    m.tri[rest[a]] = n;
  }
  trn_tag_fix(m, destin);
  const TrnRow vc = trn_row(m.vic, m, source);
  const int nv = m.vdeg[source];
  /* re-activate the 1-ring: independent flag atomics, newly set ids listed
   * in batches of 16 with one atomic each */
  int ids[16], na = 0;
  for (int b = 0; b < nv; ++b) {
    const int t = vc[b];
    if (trn_byte_cas01(m.activ + t)) ids[na++] = t;
    if (na == 16) {
      if (m.act_next) trn_list_push_n(m.act_next, m.act_next_n, ids, na);
      na = 0;
    }
  }
  if (m.act_next) trn_list_push_n(m.act_next, m.act_next_n, ids, na);
  m.vdeg[source] = 0;
  m.alive[source] = 0;
  for (int a = 0; a < deg; ++a) st[a] = -1;
  m.deg[source] = 0;
}

/* where a collapse's newly tagged vertices go: straight onto the lists (one
 * atomic per warp and push), or, in a grid-wide launch, into the block's
 * shared buffers, which one atomic each empties (thousands of warps pushing a
 * few ids each serialise on the two counters in L2) */
struct DirectSink {
  __device__ __forceinline__ void fix(const DMesh& m, int v) const { trn_tag_fix(m, v); }
  __device__ __forceinline__ void act(const DMesh& m, int v) const { trn_activate(m, v); }
};

constexpr int kSinkAct = 512, kSinkFix = 192;
struct BlockLists {
  int act[kSinkAct], fix[kSinkFix];
  int nact, nfix, act0, fix0;
};
struct BlockSink {
  BlockLists* b;
  __device__ __forceinline__ void fix(const DMesh& m, int v) const {
    if (!trn_byte_cas01(m.fixes + v) || !m.fix_list) return;
    const int k = atomicAdd(&b->nfix, 1);
    if (k < kSinkFix) b->fix[k] = v;
    else trn_list_push(m.fix_list, m.fix_n, v);
  }
  __device__ __forceinline__ void act(const DMesh& m, int v) const {
    if (!trn_byte_cas01(m.activ + v) || !m.act_next) return;
    const int k = atomicAdd(&b->nact, 1);
    if (k < kSinkAct) b->act[k] = v;
    else trn_list_push(m.act_next, m.act_next_n, v);
  }
};

/* one collapse by 8 lanes, up to four elements a lane: the shell elements are
 * the first one (boundary source) or two that hold both ends; the others move
 * to the destination. Every step's gathers and atomics are in flight together,
 * where one lane went through its elements and its neighbours one after the
 * other. Levels of a few hundred collapses: 20-29 us -> 6 us inside the level
 * loop, 14 us as a launch; the first level of the 2M-triangle workload 141 ->
 * 60 us (a level's pushes through the block's buffers; straight onto the
 * lists it took twice the one-lane kernel's time). */
constexpr int kCollapseLanes = 8, kCollapseEach = 4;

template <class Sink>
__device__ __forceinline__ void collapse_group(const DMesh& m, int source, int destin, const Sink& sink, int* buf) {
  const int lane = threadIdx.x & 31, gl = lane & (kCollapseLanes - 1), g0 = lane & ~(kCollapseLanes - 1);
  const unsigned gm = 0xffu << g0;
  /* through a shuffle: every lane has read the count before the first lane's
   * serial collapse can clear it, and all of them take the same branch */
  const int deg = __shfl_sync(gm, trn_deg(m, source), 0, kCollapseLanes);
  if (deg > kCollapseLanes * kCollapseEach) {
    if (gl == 0) collapse_serial(m, source, destin, buf);
    __syncwarp(gm);
    return;
  }
  const TrnRow st = trn_row(m.stenc, m, source), vc = trn_row(m.vic, m, source);
  const int nv = m.vdeg[source];
  const int limit = (m.tags[source] & TRN_TAG_BOUND) ? 1 : 2;
  int e[kCollapseEach];
  int4 n[kCollapseEach];
#pragma unroll
  for (int c = 0; c < kCollapseEach; ++c) {
    const int at = c * kCollapseLanes + gl;
    e[c] = at < deg ? st[at] : -1;
  }
#pragma unroll
  for (int c = 0; c < kCollapseEach; ++c) n[c] = e[c] >= 0 ? m.tri[e[c]] : make_int4(-1, -1, -1, 0);
  int shells = 0, nr = 0, place[kCollapseEach] = {-1, -1, -1, -1}, opp[kCollapseEach] = {-1, -1, -1, -1};
  unsigned trash = 0;
#pragma unroll
  for (int c = 0; c < kCollapseEach; ++c) {
    if (c * kCollapseLanes >= deg) break;   /* the same on every lane of the group */
    int o = -2;
    if (e[c] >= 0) {
      if ((source == n[c].x && destin == n[c].y) || (destin == n[c].x && source == n[c].y)) o = n[c].z;
      else if ((source == n[c].y && destin == n[c].z) || (destin == n[c].y && source == n[c].z)) o = n[c].x;
      else if ((source == n[c].z && destin == n[c].x) || (destin == n[c].z && source == n[c].x)) o = n[c].y;
    }
    const unsigned both = (__ballot_sync(gm, o != -2) & gm) >> g0;
    const bool shell = o != -2 && shells + __popc(both & ((1u << gl) - 1u)) < limit;
    shells += __popc(both);
    if (shell) {
      trash |= 1u << c;
      opp[c] = o;
    }
    const bool live = c * kCollapseLanes + gl < deg && !shell;
    const unsigned keep = (__ballot_sync(gm, live) & gm) >> g0;
    if (live) place[c] = nr + __popc(keep & ((1u << gl) - 1u));
    nr += __popc(keep);
  }
  int k = 0;
  if (gl == 0) k = atomicAdd(m.deg + destin, nr);
  k = __shfl_sync(gm, k, 0, kCollapseLanes);
  const bool full = k + nr > m.bucket;
  if (full && gl == 0) trn_set_error(m.err, TRN_DERR_BUCKET);
  const TrnRow dst = trn_row(m.stenc, m, destin);
#pragma unroll
  for (int c = 0; c < kCollapseEach; ++c) {
    const int at = c * kCollapseLanes + gl;
    if (place[c] >= 0) {
      if (!full) dst[k + place[c]] = e[c];
      if (n[c].x == source) n[c].x = destin;
      else if (n[c].y == source) n[c].y = destin;
      else if (n[c].z == source) n[c].z = destin;
      if (e[c] >= 0) m.tri[e[c]] = n[c];
    } else if ((trash >> c) & 1u) {
      m.tri[e[c]] = make_int4(-1, -1, -1, 0);
      if (opp[c] >= 0) sink.fix(m, opp[c]);
    }
    if (at < deg) st[at] = -1;
  }
  if (gl == 0) sink.fix(m, destin);
  for (int b = gl; b < nv; b += kCollapseLanes) sink.act(m, vc[b]);
  __syncwarp(gm);   /* every lane has read the counts */
  if (gl == 0) {
    m.vdeg[source] = 0;
    m.alive[source] = 0;
    m.deg[source] = 0;
  }
}

__global__ void __launch_bounds__(TRN_THREADS) k_collapse(DMesh m, const int* __restrict__ indep, const int* count,
                                                         const int* __restrict__ target,
                                                         const uint8_t* __restrict__ cand_flag) {
  __shared__ BlockLists lists;
  if (trn_failed_block(m)) return;
  const int n_indep = *count;
  const BlockSink sink{&lists};
  int buf[TRN_MAX_DEG];
  constexpr int groups = TRN_THREADS / kCollapseLanes;
  for (int base = blockIdx.x * groups; base < n_indep; base += gridDim.x * groups) {
    if (threadIdx.x == 0) lists.nact = lists.nfix = 0;
    __syncthreads();
    const int q = base + (int) threadIdx.x / kCollapseLanes;
    if (q < n_indep) {
      const int source = indep[q];
      if (source < 0 || source >= m.capa_node || (cand_flag && !cand_flag[source])) {
        if ((threadIdx.x & (kCollapseLanes - 1)) == 0) trn_set_error(m.err, TRN_DERR_REPLAY);
      } else {
        collapse_group(m, source, target[source], sink, buf);
      }
    }
    __syncthreads();
    const int na = min(lists.nact, kSinkAct), nf = min(lists.nfix, kSinkFix);
    if (threadIdx.x == 0 && na) lists.act0 = atomicAdd(m.act_next_n, na);
    if (threadIdx.x == 32 && nf) lists.fix0 = atomicAdd(m.fix_n, nf);
    __syncthreads();
    for (int i = threadIdx.x; i < na; i += TRN_THREADS) m.act_next[lists.act0 + i] = lists.act[i];
    for (int i = threadIdx.x; i < nf; i += TRN_THREADS) m.fix_list[lists.fix0 + i] = lists.fix[i];
    __syncthreads();
  }
}

/* ---- the levels of a short list in one launch (trn_level.cuh) ---- */

constexpr int kMaxMisRounds = 8;

template <bool F32>
__global__ void __launch_bounds__(kTailThreads) k_coarsen_tail(DMesh m, int* act0, int* act1, int* status, int* target,
                                                               int* cand, uint8_t* s0, uint8_t* s1, int* indep,
                                                               int* open, Seed sd, int rounds, int cap) {
  SerialBuf buf;
  const int tid = trn_tid(), stride = trn_grid_stride();
  for (int level = 0;; ++level) {
    const int* act = (level & 1) ? act1 : act0;
    m.act_next = (level & 1) ? act0 : act1;
    const bool failed = tail_failed(m);
    /* the filter; the counters of the later steps start empty */
    if (tid == 0) {
      trn_level_clear(m, nullptr);
      status[S_NINDEP] = 0;
      for (int r = 0; r < kMaxMisRounds; ++r) open[r] = 0;
    }
    /* more lanes a vertex while the list leaves lanes idle */
    const int na = failed ? 0 : status[S_ACT];
    if (na * 16 <= 2 * stride)
      search_list<F32, 16>(m, act, na, tid >> 5, stride >> 5, target, cand, status + S_NTASK, s0, buf);
    else
      search_list<F32, 8>(m, act, na, tid >> 5, stride >> 5, target, cand, status + S_NTASK, s0, buf);
    cluster_sync();
    /* the independent set: rounds until no candidate is undecided (the
     * rounds after that would only copy the states) */
    const int nc = status[S_NTASK];
    const uint64_t base = trn_seed(sd);
    MisCand mine;
    if (tid < nc) mine.load(m, cand[tid]);
    int r = 0;
    while (r < rounds) {
      const uint8_t* in = (r & 1) ? s1 : s0;
      uint8_t* out = (r & 1) ? s0 : s1;
      const uint64_t seed = base + 0x9e3779b97f4a7c15ULL * r;
      bool wait = false;
      if (mine.v >= 0) {
        mine.round(m, in, out, seed);
        wait = mine.st == 1;
      }
      for (int q = tid + stride; q < nc; q += stride) {   /* more candidates than threads */
        MisCand c;
        c.load(m, cand[q]);
        c.st = in[c.v];
        c.round(m, in, out, seed);
        wait |= c.st == 1;
      }
      if (wait) open[r] = 1;
      cluster_sync();
      if (!tail_word(open + r++)) break;
    }
    uint8_t* state = (r & 1) ? s1 : s0;
    uint8_t* other = (r & 1) ? s0 : s1;
    for (int q = tid; q < nc; q += stride) {
      const int v = cand[q];
      const uint8_t st = q == tid ? mine.st : state[v];
      if (st == 2) trn_append(indep, status + S_NINDEP, v);
      else if (st == 1) trn_activate(m, v);
      state[v] = 0;
      other[v] = 0;
    }
    cluster_sync();
    const int ni = tail_failed(m) ? 0 : status[S_NINDEP];
    for (int q = tid / kCollapseLanes; q < ni; q += stride / kCollapseLanes) {
      const int v = indep[q];
      collapse_group(m, v, target[v], DirectSink(), buf.ids);
    }
    cluster_sync();
    if (tid == 0) tail_level_end(m, status, kLevelCoarsen, cap);
    if (!tail_failed(m)) tail_fix(m, tid, stride, buf.ids);
    cluster_sync();
    if (!tail_word(status + S_CONT)) return;
  }
}

bool coarsen_tail(const DMesh& m, int* act0, int* act1, int* status, int* target, int* cand, HeurWs& ws, int* indep,
                  Seed sd, int rounds, int cap, bool fp32, cudaStream_t s) {
  if (rounds > kMaxMisRounds) return false;
  ProfScope ps("coarsen_tail", s, 0.0);
  int* open = ws.cnt + 112;
  return fp32 ? cluster_launch<k_coarsen_tail<true>>(s, m, act0, act1, status, target, cand, ws.state, ws.state2,
                               indep, open, sd, rounds, cap)
              : cluster_launch<k_coarsen_tail<false>>(s, m, act0, act1, status, target, cand, ws.state, ws.state2,
                               indep, open, sd, rounds, cap);
}

void coarsen_pre(const DMesh& m, int nb_nodes, cudaStream_t s, int* act, int* act_n) {
  if (act) cudaMemsetAsync(act_n, 0, sizeof(int), s);
  k_coarse_pre<<<grid_for(nb_nodes), TRN_THREADS, 0, s>>>(m, nb_nodes, act, act_n);
  note_launch();
  check_launch("coarsen_pre");
}

void coarsen_filter(const DMesh& m, int nb_nodes, int* target, uint8_t* flag, bool fp32, cudaStream_t s) {
  ProfScope ps("coarsen_filter", s, (double) nb_nodes * (1 + 1 + 4 + 1));
  if (fp32) k_coarse_filter<true><<<grid_for(nb_nodes), TRN_THREADS, 0, s>>>(m, nb_nodes, target, flag);
  else k_coarse_filter<false><<<grid_for(nb_nodes), TRN_THREADS, 0, s>>>(m, nb_nodes, target, flag);
  note_launch();
  check_launch("coarsen_filter");
}



void coarsen_filter_append(const DMesh& m, const int* act, const int* act_n, int* target, int* cand,
                           int* count, uint8_t* state, bool fp32, cudaStream_t s, long long bound) {
  ProfScope ps("coarsen_filter", s, 0.0);
  /* a level listing at most group_max vertices runs the grouped search
   * (measured on B200 with 8 lanes: faster below ~16k listed vertices, 2x
   * slower on full-mesh levels), a larger one the one-lane search. A known
   * bound (the level's list length) picks the form; with an unknown one (a
   * captured round) both are launched, and the one that is not the device
   * count's case returns at once. group_lanes = 1: the one-lane search at
   * every size (a launch shape for the tests: the same targets). */
  const Tune& t = tune();
  const bool one = t.group_lanes == 1;
  const int gm = one ? -1 : t.group_max;
  const bool small = !one && bound >= 0 && bound <= gm;
  const bool large = one || bound > gm;
  const int g = grid_bounded(bound, m.capa_node, t.filter_threads);
  const int gg = grid_bounded(bound < 0 ? -1 : bound * t.group_lanes, (long long) gm * t.group_lanes);
#define TRN_GROUP(F, G)                                                                              \
  k_coarse_filter_group<F, G><<<gg, TRN_THREADS, 0, s>>>(m, act, act_n, target, cand, count, state, gm)
  if (!large) {
    if (fp32) {
      if (t.group_lanes == 4) TRN_GROUP(true, 4);
      else if (t.group_lanes == 16) TRN_GROUP(true, 16);
      else TRN_GROUP(true, 8);
    } else {
      if (t.group_lanes == 4) TRN_GROUP(false, 4);
      else if (t.group_lanes == 16) TRN_GROUP(false, 16);
      else TRN_GROUP(false, 8);
    }
    note_launch();
  }
#undef TRN_GROUP
  if (!small) {
    /* alone (a known long list, or one lane throughout), it takes any count */
    const int min_n = large ? 0 : gm + 1;
    auto* kern = fp32 ? k_coarse_filter_append<true> : k_coarse_filter_append<false>;
    kern<<<grid_resident(reinterpret_cast<const void*>(kern), t.filter_threads, g), t.filter_threads, 0, s>>>(
        m, act, act_n, target, cand, count, state, min_n);
    note_launch();
  }
  check_launch("coarsen_filter_append");
}

void collapse(const DMesh& m, const int* indep, const int* count, const int* target,
              const uint8_t* cand_flag, cudaStream_t s, long long bound) {
  ProfScope ps("collapse", s, 0.0);
  const int g = grid_bounded(bound < 0 ? bound : kCollapseLanes * bound, (long long) kCollapseLanes * m.capa_node);
  k_collapse<<<TRN_RESIDENT(k_collapse, g, TRN_THREADS), TRN_THREADS, 0, s>>>(m, indep, count, target, cand_flag);
  note_launch();
  check_launch("collapse");
}

}  // namespace trn
