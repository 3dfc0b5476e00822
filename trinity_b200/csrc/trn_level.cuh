/*
 * trn_level.cuh — what the levels of coarsening and swapping share: the
 * stencil repair, and the cluster that runs the levels of short lists.
 */
#ifndef TRN_LEVEL_CUH
#define TRN_LEVEL_CUH

#include "trn_cluster.h"
#include "trn_internal.h"

namespace trn {

/* repair of one tagged stencil (Mesh::fixTagged, mesh.cpp:716-760): keep the
 * entries whose element still holds v, sorted, without duplicates. Stencils
 * of up to 16 entries stay in registers (the element loads all in flight at
 * once, a sorting network, no local memory); longer ones take the scratch
 * array. Both give the same entries in the same order. */
constexpr int kFixRegs = 16;

__device__ __forceinline__ void fix_stencil(const DMesh& m, int v, int* buf) {
  const TrnRow s = trn_row(m.stenc, m, v);
  const int d = trn_deg(m, v);
  int k = 0;
  if (d <= kFixRegs) {
    int r[kFixRegs];
#pragma unroll
    for (int c = 0; c < kFixRegs / 4; ++c) {   /* a chunk of the row is two vector loads */
      const int4 x = 4 * c < d ? *reinterpret_cast<const int4*>(s.p + (size_t) (c / 2) * s.plane + 4 * (c & 1))
                               : make_int4(-1, -1, -1, -1);
      r[4 * c] = 4 * c < d ? x.x : -1;
      r[4 * c + 1] = 4 * c + 1 < d ? x.y : -1;
      r[4 * c + 2] = 4 * c + 2 < d ? x.z : -1;
      r[4 * c + 3] = 4 * c + 3 < d ? x.w : -1;
    }
#pragma unroll
    for (int a = 0; a < kFixRegs; ++a) {
      int keep = 0x7fffffff;
      if (r[a] >= 0) {
        const int4 nn = m.tri[r[a]];
        if (v == nn.x || v == nn.y || v == nn.z) keep = r[a];
      }
      r[a] = keep;
    }
#pragma unroll
    for (int p = 0; p < kFixRegs; ++p)
#pragma unroll
      for (int a = p & 1; a + 1 < kFixRegs; a += 2) {
        const int lo = min(r[a], r[a + 1]), hi = max(r[a], r[a + 1]);
        r[a] = lo;
        r[a + 1] = hi;
      }
#pragma unroll
    for (int a = 0; a < kFixRegs; ++a)
      if (r[a] != 0x7fffffff && (a == 0 || r[a] != r[a - 1])) s[k++] = r[a];
  } else {
    for (int a = 0; a < d; ++a) {
      const int t = s[a];
      if (t < 0) continue;
      const int4 nn = m.tri[t];
      if (v == nn.x || v == nn.y || v == nn.z) buf[k++] = t;
    }
    trn_isort(buf, k);
    k = trn_iunique(buf, k);
    for (int a = 0; a < k; ++a) s[a] = buf[a];
  }
  for (int a = k; a < d; ++a) s[a] = -1;
  m.deg[v] = k;
}

/* the same repair by 16 lanes, two entries a lane (longer stencils by the
 * first lane): an entry's place among the kept ones is the number of smaller
 * ids, counted by shuffles. `gm`: the group's lanes, all of which call it. */
constexpr int kFixLanes = 16;

__device__ __forceinline__ void fix_stencil_group(const DMesh& m, int v, unsigned gm, int* buf) {
  const int gl = threadIdx.x & (kFixLanes - 1);
  /* through a shuffle: every lane has read the count before the first lane's
   * serial repair can change it, and all of them take the same branch */
  const int d = __shfl_sync(gm, trn_deg(m, v), 0, kFixLanes);
  if (d > 2 * kFixLanes) {
    if (gl == 0) fix_stencil(m, v, buf);
    __syncwarp(gm);
    return;
  }
  const TrnRow s = trn_row(m.stenc, m, v);
  int r[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = gl + h * kFixLanes;
    r[h] = k < d ? s[k] : -1;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    int keep = 0x7fffffff;
    if (r[h] >= 0) {
      const int4 nn = m.tri[r[h]];
      if (v == nn.x || v == nn.y || v == nn.z) keep = r[h];
    }
    r[h] = keep;
  }
  int below[2] = {0, 0};
  bool dup[2] = {false, false};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h * kFixLanes >= d) break;   /* the same on every lane of the group */
    for (int k = 0; k < kFixLanes; ++k) {
      const int x = __shfl_sync(gm, r[h], k, kFixLanes);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        below[o] += x < r[o];
        dup[o] |= x == r[o] && h * kFixLanes + k < o * kFixLanes + gl;
      }
    }
  }
  const bool keep0 = r[0] != 0x7fffffff, keep1 = r[1] != 0x7fffffff;
  /* a duplicate (never met) would shift the places after it: one lane then */
  const bool twice = __any_sync(gm, (keep0 && dup[0]) || (keep1 && dup[1]));
  if (twice) {
    if (gl == 0) fix_stencil(m, v, buf);
    __syncwarp(gm);
    return;
  }
  const int g0 = (threadIdx.x & 31) & ~(kFixLanes - 1);
  const int k = __popc((__ballot_sync(gm, keep0) & gm) >> g0) + __popc((__ballot_sync(gm, keep1) & gm) >> g0);
  if (keep0) s[below[0]] = r[0];
  if (keep1) s[below[1]] = r[1];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int at = gl + h * kFixLanes;
    if (at >= k && at < d) s[at] = -1;
  }
  if (gl == 0) m.deg[v] = k;
}

/* the repair of the listed vertices inside the level loop below */
__device__ __forceinline__ void tail_fix(const DMesh& m, int tid, int stride, int* buf) {
  const int n = *m.fix_n;
  const unsigned gm = 0xffffu << ((threadIdx.x & 31) & ~(kFixLanes - 1));
  for (int q = tid / kFixLanes; q < n; q += stride / kFixLanes) {
    const int v = m.fix_list[q];
    const bool on = m.fixes[v] != 0;
    __syncwarp(gm);   /* every lane has read the tag */
    if (!on) continue;
    if ((threadIdx.x & (kFixLanes - 1)) == 0) m.fixes[v] = 0;
    fix_stencil_group(m, v, gm, buf);
  }
}

/* one candidate of the independent set, kept in registers over the rounds:
 * its neighbours, of which a round reads the states (in flight together; the
 * rule is mis_item's of heuristics.cu) */
struct MisCand {
  int v = -1, nv = 0;
  int w[kRowChunk];
  uint8_t st = 0;

  __device__ __forceinline__ void load(const DMesh& m, int id) {
    v = id;
    st = 1;   /* the filter marks every candidate undecided */
    nv = m.vdeg[v];
    const int* row = trn_row(m.vic, m, v).p;
#pragma unroll
    for (int j = 0; j < kRowChunk; ++j) w[j] = j < nv ? row[j] : -1;
  }
  __device__ __forceinline__ void round(const DMesh& m, const uint8_t* in, uint8_t* out, uint64_t seed) {
    if (st == 1) {
      const uint64_t pv = trn_prio(seed, v);
      bool is_max = true, leave = false;
      uint8_t sw[kRowChunk];
#pragma unroll
      for (int j = 0; j < kRowChunk; ++j) sw[j] = w[j] >= 0 ? in[w[j]] : 0;
#pragma unroll
      for (int j = 0; j < kRowChunk; ++j) {
        leave |= sw[j] == 2;
        if (sw[j] == 1 && trn_prio(seed, w[j]) > pv) is_max = false;
      }
      const TrnRow vc = trn_row(m.vic, m, v);
      for (int b = kRowChunk; b < nv; ++b) {
        const int x = vc[b];
        const uint8_t s = in[x];
        leave |= s == 2;
        if (s == 1 && trn_prio(seed, x) > pv) is_max = false;
      }
      st = leave ? 0 : (is_max ? 2 : 1);
    }
    out[v] = st;
  }
};

/* ---- the level loop of short lists ----
 * A level is five steps with a dependence between each (filter, the
 * heuristic's rounds, collapse or flip, repair, decision), and its list
 * shrinks from the whole mesh to a handful over some fifteen levels. Once a
 * list is short, a step is a chain of a few dependent gathers, and the
 * launches and the host's read back between the steps cost several times
 * that. So the levels left run inside one launch: one thread-block cluster,
 * its steps separated by the hardware's cluster barrier (no spinning, and
 * every block of a cluster is resident by definition), the decision read by
 * all blocks after it. The blocks take the same branches: whatever decides a
 * branch around a barrier was written before the barrier before it, and an
 * error only makes the steps' items do nothing until the level's end stops
 * the loop. The steps are those of the grid-wide kernels on the same state,
 * so a call ends on the same mesh wherever it switches. A coarsening level of
 * some hundred vertices takes about 30 us here (search 7, four or five rounds
 * of the independent set 10, collapse 6, repair 5), 110 us as four launches
 * and a read back; a swapping level 35 us instead of 165. The 100 x 100
 * workload's three rounds, before any cluster and now: coarsening 5.02 -> 2.58
 * ms, swapping 2.22 -> 1.27. */
constexpr int kTailThreads = 512;

__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile(
      "barrier.cluster.arrive.release;\n"
      "barrier.cluster.wait.acquire;\n" ::
          : "memory");
}

/* trn_failed as one value for the whole warp: another thread may raise the
 * error word at any time, and lanes that disagreed about it would part ways
 * before the shuffles and votes of their group (all 32 lanes call it) */
__device__ __forceinline__ bool tail_failed(const DMesh& m) {
  int f = 0;
  if ((threadIdx.x & 31) == 0) f = trn_failed(m) ? 1 : 0;
  return __shfl_sync(0xffffffffu, f, 0) != 0;
}

/* a word that decides a branch around a barrier */
__device__ __forceinline__ int tail_word(const int* p) { return *(const volatile int*) p; }

/* launches `kernel` as one cluster on the current device; false when it could
 * not (the caller then takes the grid-wide kernels) */
template <auto kernel, class... Args>
bool cluster_launch(cudaStream_t s, Args... args) {
  static ClusterSizes sizes;   /* of this kernel */
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kTailThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  /* an error of these calls is answered here and not left for the next check */
  auto ok = [](cudaError_t e) {
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
  };
  auto probe = [&](int c) {
    int n = 0;
    cfg.gridDim = dim3(c);
    at[0].val.clusterDim.x = c;
    return (c <= 8 || ok(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))) &&
           ok(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg)) && n > 0;
  };
  auto launch = [&](int c) {
    cfg.gridDim = dim3(c);
    at[0].val.clusterDim.x = c;
    return ok(cudaLaunchKernelEx(&cfg, kernel, args...));
  };
  if (!sizes.launch(dev, probe, launch)) return false;
  note_launch();
  return true;
}

/* the end of a level inside the loop, by one thread: level_end_decide, and no
 * further level after an error */
__device__ __forceinline__ void tail_level_end(const DMesh& m, int* status, int kind, int cap) {
  level_end_decide(status, kind, cap, 0, 0);
  if (trn_failed(m)) status[S_CONT] = 0;
}

}  // namespace trn

#endif
