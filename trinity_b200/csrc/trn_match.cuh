/*
 * trn_match.cuh — the swap matchings' rules, one dual row at a time: the
 * handshake's phases and the greedy loop's rounds, shared by the grid-wide
 * kernels (heuristics.cu) and the level loop of short lists (swap.cu).
 */
#ifndef TRN_MATCH_CUH
#define TRN_MATCH_CUH

#include "trn_internal.h"
#include "trn_level.cuh"

namespace trn {

/* ---------------- matching ---------------- */
constexpr int kMatchRounds = 4;

/* The rank of dual edge (row i, slot q) in the upper bits of its weight, and
 * the mask of the lower bits a hash fills. Row order (rank == nullptr): the
 * slot of the edge in the row of its lower-id candidate end, first slots
 * first, as the reference's greedy takes each candidate's first free
 * neighbour. Gain: rank[4 i + q], the quantized quality change of the flip.
 * Both ends of an edge between two candidates compute the same rank. */
__device__ __forceinline__ uint32_t edge_rank(const int* __restrict__ dual, const int* __restrict__ dual_n,
                                              const uint32_t* __restrict__ rank, const int* __restrict__ map,
                                              int ntasks, int i, int q, uint32_t* low) {
  if (rank) {
    *low = 0x3ffu;
    return rank[i * 4 + q];
  }
  const int c = dual[i * 4], n = dual[i * 4 + q];
  int pos = q;
  if (n < c) {
    const int x = map[n];
    if (x >= 0 && x < ntasks && dual[x * 4] == n)
      for (int e = 1; e < dual_n[x]; ++e)
        if (dual[x * 4 + e] == c) pos = e;
  }
  *low = 0x3fffffffu;
  return (uint32_t) (4 - pos) << 30;
}

/* the weight of dual edge (row i, slot q): its rank, then a symmetric hash of
 * the pair, so equal ranks break ties at random and the edge weighs the same
 * from both ends */
__device__ __forceinline__ uint32_t edge_weight(const int* __restrict__ dual, const int* __restrict__ dual_n,
                                                const uint32_t* __restrict__ rank, const int* __restrict__ map,
                                                int ntasks, int i, int q, uint64_t seed, int round) {
  const int a = dual[i * 4], b = dual[i * 4 + q];
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  const uint64_t h = trn_hash64(seed ^ ((uint64_t) (uint32_t) lo << 32 | (uint32_t) hi) ^
                                ((uint64_t) round * 0xd1b54a32d192ed03ULL));
  uint32_t low;
  const uint32_t r = edge_rank(dual, dual_n, rank, map, ntasks, i, q, &low);
  return (r & ~low) | ((uint32_t) (h >> 32) & low) | 1u;
}

struct MatchArgs {
  const int* dual;
  const int* dual_n;
  const uint32_t* rank;   /* gain ranks, or nullptr for row order */
  const int* map;
  int* mate;
  unsigned long long* prop;
  int* choice;
};

__device__ __forceinline__ void match_reset_item(const MatchArgs& a, int i) {
  for (int q = 0; q < a.dual_n[i]; ++q) {
    const int e = a.dual[i * 4 + q];
    a.mate[e] = -1;
    a.prop[e] = 0ULL;
  }
}

__device__ __forceinline__ void match_propose_item(const MatchArgs& a, int ntasks, int i, uint64_t seed,
                                                   int round) {
  const int c = a.dual[i * 4];
  int best = -1;
  uint32_t bw = 0;
  if (a.mate[c] == -1) {
    for (int q = 1; q < a.dual_n[i]; ++q) {
      const int n = a.dual[i * 4 + q];
      if (a.mate[n] != -1) continue;
      const uint32_t w = edge_weight(a.dual, a.dual_n, a.rank, a.map, ntasks, i, q, seed, round);
      if (w > bw) { bw = w; best = n; }
    }
    if (best >= 0) atomicMax(a.prop + best, ((unsigned long long) bw << 32) | (uint32_t) c);
  }
  a.choice[i] = best;
}

/* a mutual choice between two candidates, or a non-candidate's heaviest
 * proposer, is a match */
__device__ __forceinline__ void match_accept_item(const MatchArgs& a, int ntasks, int i, uint64_t seed,
                                                  int round, int* pairs, int* npairs) {
  const int n = a.choice[i];
  if (n < 0) return;
  const int c = a.dual[i * 4];
  const int x = a.map[n];
  const bool n_cand = x >= 0 && x < ntasks && a.dual[x * 4] == n;
  bool ok;
  if (n_cand) {
    ok = (a.choice[x] == c) && (c < n);
  } else {
    int q = 1;
    while (q < a.dual_n[i] - 1 && a.dual[i * 4 + q] != n) ++q;
    const uint32_t w = edge_weight(a.dual, a.dual_n, a.rank, a.map, ntasks, i, q, seed, round);
    ok = a.prop[n] == (((unsigned long long) w << 32) | (uint32_t) c);
  }
  if (ok) {
    a.mate[c] = n;
    a.mate[n] = c;
    const int p = trn_warp_reserve(npairs);
    pairs[2 * p] = c;
    pairs[2 * p + 1] = n;
  }
}

__device__ __forceinline__ void match_clear_item(const MatchArgs& a, int i) {
  for (int q = 1; q < a.dual_n[i]; ++q) a.prop[a.dual[i * 4 + q]] = 0ULL;
}

/* ---------------- greedy matching in interleaved element order ----------------
 *
 * The reference's matching (Match::computeGreedyMatching / matchAndUpdate,
 * matching.cpp:81-135) is a loop over the dual rows in list order, i.e. in
 * increasing candidate id: a row whose candidate is still free marks it
 * taken, then takes its free neighbours in slot order, going past each
 * neighbour that is not itself a candidate (the "continue" of
 * matching.cpp:124) and stopping at the first one that is; the candidate's
 * partner is the last neighbour taken. This is that loop without the
 * degree-1 stack, over the rows in the order (id mod 4, id): four
 * interleaved sweeps of the candidate ids.
 *
 * Its result is computed exactly, in parallel, as the greedy matching of an
 * order is: in each round a row decides once it comes first, under that
 * order, among the undecided rows that list any of its elements; such rows
 * share no element with one another, so they decide independently, and what
 * each finds is what the sequential loop would have found. Rows propose
 * their key with a 64-bit atomicMin on every element of their row into the
 * round's buffer (keys of later rounds compare lower, so no buffer needs
 * clearing between rounds); a row is ready when every element holds its own
 * key. A round decides the ready rows and lets the others propose for the
 * next round into the other buffer, so one launch per round. The rounds
 * run over a compacted list of the undecided rows; once that list is short
 * one block finishes the remaining rounds with block barriers. After
 * kGreedyRounds rounds any row still undecided stays unmatched (a valid, if
 * not maximal, matching). On the 2M-triangle workload the deepest level
 * needs 48 rounds, the mean is 12.
 *
 * The four-way interleave keeps the chains of dependent rows short (a plain
 * increasing-id sweep has chains as long as a row of the grid), and the
 * final meshes' metric edge-length histograms stay within half a point per
 * bin of the reference's, where a maximal handshake matching, which flips
 * more pairs, is a point and a half off. */
constexpr int kGreedyRounds = 64;
constexpr int kGreedyTail = 2048;   /* undecided rows left to the one-block rounds */
/* rows waiting above which a round runs as its own grid launch: what the
 * threads of a cluster keep in registers (greedy_cluster). Matching of the
 * 2M-triangle workload's three rounds 3.80 ms with a cooperative grid for the
 * rounds after that, 3.22 ms with the cluster. */
constexpr int kGreedyGrid = 1 << 15;

struct GreedyArgs {
  const int* dual;
  const int* dual_n;
  const int* map;
  int* vis;                 /* per element: -1 free, else taken */
  unsigned long long* mk0;  /* per element: lowest key proposed, even rounds */
  unsigned long long* mk1;  /* odd rounds */
  int* list0;               /* undecided rows, even rounds */
  int* list1;
  int* cnt;                 /* [3] list lengths, by round mod 3 */
  int* ran;                 /* [kGreedyRounds] round r ran on the grid */
};

__device__ __forceinline__ unsigned long long greedy_key(int r, int c) {
  return ((unsigned long long) (kGreedyRounds - r) << 40) | ((unsigned long long) (c & 3) << 32) |
         (uint32_t) c;
}

/* "is a candidate" as matching.cpp:124 asks it: the element has a row in the
 * map, which keeps the rows of earlier levels of the same call (it is reset
 * once per call, swapping.cpp:161-162) */
__device__ __forceinline__ bool greedy_is_row(const GreedyArgs& a, int ntasks, int e) {
  (void) ntasks;
  return a.map[e] >= 0;
}


__device__ __forceinline__ void greedy_propose(const GreedyArgs& a, int r, int i) {
  unsigned long long* mk = (r & 1) ? a.mk1 : a.mk0;
  const unsigned long long key = greedy_key(r, a.dual[i * 4]);
  for (int q = 0; q < a.dual_n[i]; ++q) atomicMin(mk + a.dual[i * 4 + q], key);
}

/* is row i first on all its elements in round r? The loads of the row's
 * slots past its length read slot 0 again (always there), so that every
 * load can be issued before any compare */
__device__ __forceinline__ bool greedy_ready(const GreedyArgs& a, int r, int i) {
  const unsigned long long* mk = (r & 1) ? a.mk1 : a.mk0;
  const int4 row = reinterpret_cast<const int4*>(a.dual)[i];
  const int dn = a.dual_n[i];
  const unsigned long long key = greedy_key(r, row.x);
  const unsigned long long k0 = mk[row.x], k1 = mk[dn > 1 ? row.y : row.x];
  const unsigned long long k2 = mk[dn > 2 ? row.z : row.x], k3 = mk[dn > 3 ? row.w : row.x];
  return k0 == key && k1 == key && k2 == key && k3 == key;
}

/* row i in round r, its readiness known: decide it when it is first on all
 * its elements (and return false), else propose it for round r + 1 (and
 * return true) */
__device__ __forceinline__ bool greedy_act(const GreedyArgs& a, int ntasks, int r, int i, bool ready,
                                           int* pairs, int* npairs) {
  const int c = a.dual[i * 4];
  const int dn = a.dual_n[i];
  if (!ready) {
    greedy_propose(a, r + 1, i);
    return true;
  }
  if (a.vis[c] != -1) return false;
  a.vis[c] = 1;
  int partner = -1;
  for (int q = 1; q < dn; ++q) {
    const int n = a.dual[i * 4 + q];
    if (a.vis[n] != -1) continue;
    a.vis[n] = 1;
    partner = n;
    if (greedy_is_row(a, ntasks, n)) break;
  }
  if (partner >= 0) {
    const int p = trn_warp_reserve(npairs);
    pairs[2 * p] = c;
    pairs[2 * p + 1] = partner;
  }
  return false;
}

__device__ __forceinline__ bool greedy_item(const GreedyArgs& a, int ntasks, int r, int i, int* pairs,
                                            int* npairs) {
  return greedy_act(a, ntasks, r, i, greedy_ready(a, r, i), pairs, npairs);
}


/* a dual row of the greedy matching, kept in registers over the rounds (the
 * rule is greedy_item's, trn_match.cuh): a round costs its four keys and, once
 * the row is first on all of them, its four elements' states */
struct TailRow {
  int4 row = make_int4(-1, -1, -1, -1);
  int dn = 0;
  unsigned rows = 0;   /* bit q: element q has a row itself */
  bool open = false;

  __device__ __forceinline__ int at(int q) const { return q == 0 ? row.x : (q == 1 ? row.y : (q == 2 ? row.z : row.w)); }
  __device__ __forceinline__ void load(const GreedyArgs& a, int i) {
    row = reinterpret_cast<const int4*>(a.dual)[i];
    dn = a.dual_n[i];
#pragma unroll
    for (int q = 1; q < 4; ++q)
      if (q < dn && a.map[at(q)] >= 0) rows |= 1u << q;
    open = true;
  }
  __device__ __forceinline__ void propose(const GreedyArgs& a, int r) const {
    unsigned long long* mk = (r & 1) ? a.mk1 : a.mk0;
    const unsigned long long key = greedy_key(r, row.x);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q < dn) atomicMin(mk + at(q), key);
  }
  __device__ __forceinline__ void round(const GreedyArgs& a, int r, int* pairs, int* npairs) {
    const unsigned long long* mk = (r & 1) ? a.mk1 : a.mk0;
    const unsigned long long key = greedy_key(r, row.x);
    bool ready = true;
    unsigned free = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q < dn) {
        ready &= mk[at(q)] == key;
        if (a.vis[at(q)] == -1) free |= 1u << q;
      }
    if (!ready) {
      propose(a, r + 1);
      return;
    }
    open = false;
    if (!(free & 1u)) return;
    a.vis[row.x] = 1;
    int partner = -1;
    bool done = false;
#pragma unroll
    for (int q = 1; q < 4; ++q)
      if (!done && ((free >> q) & 1u)) {
        a.vis[at(q)] = 1;
        partner = at(q);
        done = (rows >> q) & 1u;
      }
    if (partner >= 0) {
      const int p = trn_warp_reserve(npairs);
      pairs[2 * p] = row.x;
      pairs[2 * p + 1] = partner;
    }
  }
};

/* The rounds of the greedy matching by one cluster, to the end: with r0 < 0
 * the whole matching of rows 0 .. ntasks - 1, else from round r0, whose
 * undecided rows are in its list and have proposed. While more rows wait than
 * the threads can keep (kClusterRows each) the rounds go over the lists as the
 * grid's do; then every thread keeps its rows in registers, and a round is
 * their keys, a few stores and a barrier. All threads of the cluster call it;
 * it ends after a barrier. */
constexpr int kClusterRows = 4;

__device__ __forceinline__ void greedy_cluster(const GreedyArgs& a, int ntasks, int r0, int* pairs, int* npairs) {
  const int tid = trn_tid(), stride = trn_grid_stride();
  const bool whole = r0 < 0;
  int* more = a.cnt + 4;   /* [3] rows left open, by round mod 3 */
  int r = whole ? 0 : r0;
  int n = whole ? ntasks : tail_word(a.cnt + r % 3);
  const bool lists = n > kClusterRows * stride;
  if (tid == 0) {
    more[0] = more[1] = more[2] = 0;
    if (whole) a.cnt[1] = a.cnt[2] = 0;
  }
  if (whole && lists) {
    if (tid == 0) a.cnt[0] = ntasks;
    for (int i = tid; i < ntasks; i += stride) {
      greedy_propose(a, 0, i);
      a.list0[i] = i;
    }
  }
  cluster_sync();
  if (lists)
    for (; r < kGreedyRounds; ++r) {
      n = tail_word(a.cnt + r % 3);
      if (n <= kClusterRows * stride) break;
      const int* in = (r & 1) ? a.list1 : a.list0;
      int* out = (r & 1) ? a.list0 : a.list1;
      if (tid == 0) a.cnt[(r + 2) % 3] = 0;
      for (int q = tid; q < n; q += stride) {
        const int i = in[q];
        if (greedy_item(a, ntasks, r, i, pairs, npairs)) trn_append(out, a.cnt + (r + 1) % 3, i);
      }
      cluster_sync();
    }
  if (r >= kGreedyRounds || n == 0) return;
  const int* in = (r & 1) ? a.list1 : a.list0;
  TailRow mine[kClusterRows];
#pragma unroll
  for (int k = 0; k < kClusterRows; ++k) {
    const int q = tid + k * stride;
    if (q < n) mine[k].load(a, whole && !lists ? q : in[q]);
  }
  if (whole && !lists) {
#pragma unroll
    for (int k = 0; k < kClusterRows; ++k)
      if (mine[k].open) mine[k].propose(a, 0);
    cluster_sync();
  }
  for (const int first = r; r < kGreedyRounds; ++r) {
    if (r > first && tail_word(more + r % 3) == 0) return;
    if (tid == 0) more[(r + 2) % 3] = 0;   /* the round after next's word */
    bool left = false;
#pragma unroll
    for (int k = 0; k < kClusterRows; ++k)
      if (mine[k].open) {
        mine[k].round(a, r, pairs, npairs);
        left |= mine[k].open;
      }
    if (left) more[(r + 1) % 3] = 1;
    cluster_sync();
  }
}

}  // namespace trn

#endif
