/*
 * trn_patch.cuh — sorted unions of short id rows, for the sums over the 2-ring
 * element patch of a vertex (metric.cu) and over the vertices whose patch
 * holds an element (adjoint.cu).
 *
 * The reference sums over a patch in ascending id without duplicates
 * (std::set order, mesh.cpp:396-432), so the union of the rows must be
 * sorted before it is summed. The rows are sorted already and short (a
 * planar triangulation averages 6 entries), so one thread merges up to N / 8
 * of them, 8 entries each, in registers with Batcher's odd-even merge: no
 * local memory and every compare of a layer independent. What does not fit
 * (a longer row, more rows, a row out of order) is left to the caller's
 * general path, which sorts any patch; both give the same ids in the same
 * order.
 */
#ifndef TRN_PATCH_CUH
#define TRN_PATCH_CUH

#include "trn_common.cuh"

constexpr int kRowRegs = kRowChunk;         /* entries of a row kept in registers */
constexpr int kNoId = 0x7fffffff;           /* pads the unused slots, sorts last */
constexpr int kPatchRows = 8;               /* the vertex's own row and 7 neighbours' */
constexpr int kPatchKeys = kPatchRows * kRowRegs;

/* odd-even merge of the sorted halves of a[0..N) */
template <int N>
__device__ __forceinline__ void patch_merge(int* a) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) patch_cmp(a[i], a[i + N / 2]);
#pragma unroll
  for (int k = N / 4; k >= 1; k >>= 1)
#pragma unroll
    for (int i = k; i + k < N; i += 2 * k)
#pragma unroll
      for (int j = 0; j < k; ++j) patch_cmp(a[i + j], a[i + j + k]);
}

/* N / 8 sorted rows of 8 into one sorted array */
template <int N>
__device__ __forceinline__ void patch_merge_rows(int* a) {
  if constexpr (N >= 16) {
#pragma unroll
    for (int i = 0; i < N; i += 16) patch_merge<16>(a + i);
  }
  if constexpr (N >= 32) {
#pragma unroll
    for (int i = 0; i < N; i += 32) patch_merge<32>(a + i);
  }
  if constexpr (N >= 64) patch_merge<64>(a);
}

/* the first n entries of a row (its first chunk, one aligned sector), the
 * rest kNoId; false when they are not in ascending order */
__device__ __forceinline__ bool patch_row(const TrnRow& row, int n, int* out) {
  int4 a = make_int4(kNoId, kNoId, kNoId, kNoId), b = a;
  if (n > 0) a = *reinterpret_cast<const int4*>(row.p);
  if (n > 4) b = *reinterpret_cast<const int4*>(row.p + 4);
  out[0] = n > 0 ? a.x : kNoId;
  out[1] = n > 1 ? a.y : kNoId;
  out[2] = n > 2 ? a.z : kNoId;
  out[3] = n > 3 ? a.w : kNoId;
  out[4] = n > 4 ? b.x : kNoId;
  out[5] = n > 5 ? b.y : kNoId;
  out[6] = n > 6 ? b.z : kNoId;
  out[7] = n > 7 ? b.w : kNoId;
  bool sorted = true;
#pragma unroll
  for (int i = 0; i < 7; ++i) sorted &= out[i] <= out[i + 1];
  return sorted;
}

/* the 2-ring element patch of v as kPatchKeys ascending ids, duplicates
 * adjacent, kNoId last; false when the rows do not fit the registers */
__device__ __forceinline__ bool patch_keys(const DMesh& m, int v, int* key) {
  const int d = trn_deg(m, v), nv = m.vdeg[v];
  if (d > kRowRegs || nv > kPatchRows - 1) return false;
  bool ok = patch_row(trn_row(m.stenc, m, v), d, key);
  int w[kRowRegs];
  patch_row(trn_row(m.vic, m, v), nv, w);   /* any order will do */
  int dw[kPatchRows - 1];
#pragma unroll
  for (int b = 0; b < kPatchRows - 1; ++b) {
    dw[b] = b < nv ? trn_deg(m, w[b]) : 0;
    ok &= dw[b] <= kRowRegs;
  }
  if (!ok) return false;
#pragma unroll
  for (int b = 0; b < kPatchRows - 1; ++b)
    ok &= patch_row(trn_row(m.stenc, m, b < nv ? w[b] : v), dw[b], key + (b + 1) * kRowRegs);
  if (!ok) return false;
  patch_merge_rows<kPatchKeys>(key);
  return true;
}

/* The general path, one warp a vertex: the patch gathered into `buf` (shared,
 * TRN_MAX_PATCH ids), sorted, duplicates left for the caller to skip. Returns
 * the ids gathered; a longer patch sets the error word.
 * All 32 lanes take part. */
__device__ __forceinline__ int patch_sort_warp(const DMesh& m, int v, int* buf) {
  const int lane = threadIdx.x & 31;
  const int d = trn_deg(m, v), nv = m.vdeg[v];
  int k = 0;
  for (int b = -1; b < nv; ++b) {
    const int w = b < 0 ? v : trn_row(m.vic, m, v)[b];
    const int dw = b < 0 ? d : trn_deg(m, w);
    const TrnRow s = trn_row(m.stenc, m, w);
    const int room = TRN_MAX_PATCH - k;
    if (dw > room && lane == 0) trn_set_error(m.err, TRN_DERR_BUCKET);
    const int n = dw < room ? dw : room;
    for (int a = lane; a < n; a += 32) buf[k + a] = s[a];
    k += n;
  }
  int size = 32;
  while (size < k) size <<= 1;
  for (int i = k + lane; i < size; i += 32) buf[i] = kNoId;
  __syncwarp();
  /* bitonic sort */
  for (int s = 2; s <= size; s <<= 1)
    for (int o = s >> 1; o > 0; o >>= 1) {
      for (int i = lane; i < size / 2; i += 32) {
        const int lo = 2 * i - (i & (o - 1)), hi = lo + o;
        const bool up = (lo & s) == 0;
        const int x = buf[lo], y = buf[hi];
        if ((x > y) == up) {
          buf[lo] = y;
          buf[hi] = x;
        }
      }
      __syncwarp();
    }
  return k;
}

/* the same by one lane, in its own array: the ids without duplicates. Every
 * id is searched among those kept so far, so the array holds a third of what
 * the rows hold (an element is in the rows of its three vertices). */
__device__ __forceinline__ int patch_sort_lane(const DMesh& m, int v, int* ids) {
  const int nv = m.vdeg[v];
  int k = 0, gathered = 0;
  for (int b = -1; b < nv; ++b) {
    const int w = b < 0 ? v : trn_row(m.vic, m, v)[b];
    const int dw = trn_deg(m, w);
    const TrnRow s = trn_row(m.stenc, m, w);
    const int room = TRN_MAX_PATCH - gathered;
    if (dw > room) trn_set_error(m.err, TRN_DERR_BUCKET);
    const int n = dw < room ? dw : room;
    gathered += n;
    for (int a = 0; a < n; ++a) {
      const int x = s[a];
      int lo = 0, hi = k;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ids[mid] < x) lo = mid + 1;
        else hi = mid;
      }
      if (lo < k && ids[lo] == x) continue;
      for (int j = k; j > lo; --j) ids[j] = ids[j - 1];
      ids[lo] = x;
      ++k;
    }
  }
  return k;
}

#endif
