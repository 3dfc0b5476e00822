/*
 * trn_metric.cuh — the FP64 metric recovery's steps for one element or vertex,
 * shared by the grid-wide kernels (metric.cu) and the one-launch recovery of
 * small meshes (noalloc.cu).
 */
#ifndef TRN_METRIC_CUH
#define TRN_METRIC_CUH

#include "trn_numeric.cuh"
#include "trn_patch.cuh"

namespace trn {

/* An element's share of a patch sum depends on the element alone, and an
 * element lies in the patches of about 12 vertices: it is computed once into a
 * 32-byte record (one sector a gather) instead of once per patch. What bounds
 * the patch sums: the record gathers (24 a vertex, mostly L1/L2 hits) and the
 * integer merge of the rows. One vertex a thread that gathered, sorted in
 * local memory and computed every element of its patch took 582 us for the
 * gradient and 650 us for the Hessian of the 2M-triangle mesh; records, the
 * merge in registers and the ids in a shared column (metric.cu) take 165 and
 * 180 us, the records' kernels included. */
/* Where the first 16 bytes of element i's record are, in units of 16 bytes;
 * the second are at the slot ^ 1. With `mix` (kRecMix; the buffer then has
 * room for a multiple of 4 records) the 8 slots of a 128-byte line are
 * exchanged by the line's number: the threads of a warp gather the records of
 * neighbouring vertices' elements, about two elements and so 64 bytes apart,
 * and would meet in two of the eight slots of a line, a quarter of the banks.
 * A record keeps its sector. */
constexpr unsigned kRecMix = 7;
__device__ __forceinline__ size_t rec_slot(int i, unsigned mix) { return ((size_t) i * 2) ^ (((unsigned) i >> 2) & mix); }

__device__ __forceinline__ void rec_store(double4* rec, int i, unsigned mix, const double4& r) {
  double2* p = reinterpret_cast<double2*>(rec);
  const size_t at = rec_slot(i, mix);
  p[at] = make_double2(r.x, r.y);
  p[at ^ 1] = make_double2(r.z, r.w);
}

__device__ __forceinline__ double4 rec_load(const double4* rec, int i, unsigned mix) {
  const double2* p = reinterpret_cast<const double2*>(rec);
  const size_t at = rec_slot(i, mix);
  const double2 a = p[at], b = p[at ^ 1];
  return make_double4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ double4 elem_gradient(const DMesh& m, int t, const double* solut) {
  if (m.tri[t].x < 0) return make_double4(0.0, 0.0, 0.0, 0.0);
  const ElemGrad g = elem_grad(m, t);
  const double s0 = solut[g.v.x], s1 = solut[g.v.y], s2 = solut[g.v.z];
  double ex = 0, ey = 0;
  ex += s0 * g.d[0];
  ey += s0 * g.d[1];
  ex += s1 * g.d[2];
  ey += s1 * g.d[3];
  ex += s2 * g.d[4];
  ey += s2 * g.d[5];
  return make_double4(g.area, g.area * ex, g.area * ey, 0.0);
}

__device__ __forceinline__ double4 elem_hessian(const DMesh& m, int t, const double2* grad) {
  if (m.tri[t].x < 0) return make_double4(0.0, 0.0, 0.0, 0.0);
  const ElemGrad g = elem_grad(m, t);
  const double2 g0 = grad[g.v.x], g1 = grad[g.v.y], g2 = grad[g.v.z];
  double dl[4] = {0, 0, 0, 0};
  dl[0] += (g0.x * g.d[0]);
  dl[1] += (g0.x * g.d[1]);
  dl[2] += (g0.y * g.d[0]);
  dl[3] += (g0.y * g.d[1]);
  dl[0] += (g1.x * g.d[2]);
  dl[1] += (g1.x * g.d[3]);
  dl[2] += (g1.y * g.d[2]);
  dl[3] += (g1.y * g.d[3]);
  dl[0] += (g2.x * g.d[4]);
  dl[1] += (g2.x * g.d[5]);
  dl[2] += (g2.y * g.d[4]);
  dl[3] += (g2.y * g.d[5]);
  return make_double4(g.area * dl[0], g.area * dl[1], g.area * dl[2], g.area * dl[3]);
}

/* the sums over one patch: load() the record of an element, add() them in
 * ascending element order, finish() the vertex. The reference stores the
 * per-element values and sums afterwards in the same element order;
 * interleaving its loops keeps every sum's order. */
struct GradSum {
  const double4* rec;
  unsigned mix;   /* of the records (rec_slot) */
  double2* grad;
  double* atot;   /* patch areas, for the Hessian's mean too */
  double total_area = 0, gx = 0, gy = 0;
  using Rec = double4;
  __device__ __forceinline__ void begin(const DMesh&, int) {}
  __device__ __forceinline__ Rec load(const DMesh&, int t) const { return rec_load(rec, t, mix); }
  __device__ __forceinline__ void add(const Rec& r) {
    total_area += r.x;
    gx += r.y;
    gy += r.z;
  }
  __device__ __forceinline__ void finish(const DMesh&, int v) {
    gx /= total_area;
    gy /= total_area;
    grad[v] = make_double2(gx, gy);
    atot[v] = total_area;
  }
};

struct HessSum {
  const double4* rec;
  unsigned mix;
  const double* atot;   /* the gradient pass's sums: the same areas in the same order */
  double scale_exp;
  double4* hsym;
  double4* mloc;
  double h[4] = {0, 0, 0, 0};
  using Rec = double4;
  __device__ __forceinline__ void begin(const DMesh&, int) {}
  __device__ __forceinline__ Rec load(const DMesh&, int t) const { return rec_load(rec, t, mix); }
  __device__ __forceinline__ void add(const Rec& r) {
    h[0] += r.x;
    h[1] += r.y;
    h[2] += r.z;
    h[3] += r.w;
  }
  __device__ __forceinline__ void finish(const DMesh& m, int v) {
    const double total_area = atot[v];
    for (int j = 0; j < 4; ++j) h[j] /= total_area;
    /* symmetrise (hessian.cpp:149-152) */
    double t0 = h[0];
    double t1 = 0.5 * (h[1] + h[2]);
    double t2 = h[3];
    if (hsym) hsym[v] = make_double4(t0, t1, t2, 0.0);
    /* normalizeLocally (metric.cpp:107-149) */
    double mm[4] = {t0, t1, t1, t2};
    double val[2] = {0, 0}, vec[4] = {0, 0, 0, 0};
    trn_eigen(mm, val, vec);
    val[0] = trn_dmax(fabs(val[0]), TRN_EPS);
    val[1] = trn_dmax(fabs(val[1]), TRN_EPS);
    double det = val[0] * val[1];
    double scale_loc = trn_pow(det, scale_exp);
    val[0] *= scale_loc;
    val[1] *= scale_loc;
    const double4 r = trn_recompose(val, vec);
    m.ten[v] = r;
    if (mloc) mloc[v] = r;
  }
};

/* one thread a vertex, its patch merged in registers; false when its rows do
 * not fit */
template <class Sum, int Batch>
__device__ __forceinline__ bool patch_sum_regs(const DMesh& m, int v, const Sum& zero) {
  int key[kPatchKeys];
  if (!patch_keys(m, v, key)) return false;
  Sum s = zero;
  s.begin(m, v);
#pragma unroll
  for (int c = 0; c < kPatchKeys; c += Batch) {
    typename Sum::Rec r[Batch];
#pragma unroll
    for (int j = 0; j < Batch; ++j)
      if (key[c + j] != kNoId && (c + j == 0 || key[c + j] != key[c + j - 1])) r[j] = s.load(m, key[c + j]);
#pragma unroll
    for (int j = 0; j < Batch; ++j)
      if (key[c + j] != kNoId && (c + j == 0 || key[c + j] != key[c + j - 1])) s.add(r[j]);
  }
  s.finish(m, v);
  return true;
}

/* the same with the patch's ids, duplicates dropped, in the thread's own
 * column of shared memory (Ids entries, Stride apart); false also when they
 * are more */
template <class Sum, int Batch, int Ids, int Stride>
__device__ __forceinline__ bool patch_sum_column(const DMesh& m, int v, const Sum& zero, int* col) {
  int n = 0;
  {
    int key[kPatchKeys];
    if (!patch_keys(m, v, key)) return false;
#pragma unroll
    for (int c = 0; c < kPatchKeys; ++c)
      if (key[c] != kNoId && (c == 0 || key[c] != key[c - 1])) {
        if (n < Ids) col[n * Stride] = key[c];
        ++n;
      }
  }
  if (n > Ids) return false;
  Sum s = zero;
  s.begin(m, v);
  for (int c = 0; c < n; c += Batch) {
    typename Sum::Rec r[Batch];
#pragma unroll
    for (int j = 0; j < Batch; ++j) r[j] = s.load(m, col[min(c + j, n - 1) * Stride]);
#pragma unroll
    for (int j = 0; j < Batch; ++j)
      if (c + j < n) s.add(r[j]);
  }
  s.finish(m, v);
  return true;
}

/* a warp a vertex: every lane walks the sorted patch (the loads are warp-wide
 * broadcasts) and the first writes */
template <class Sum>
__device__ __forceinline__ void patch_sum_warp(const DMesh& m, int v, const Sum& zero, int* buf) {
  const int k = patch_sort_warp(m, v, buf);
  Sum s = zero;
  s.begin(m, v);
  for (int i = 0; i < k; ++i)
    if (i == 0 || buf[i] != buf[i - 1]) s.add(s.load(m, buf[i]));
  if ((threadIdx.x & 31) == 0) s.finish(m, v);
  __syncwarp();
}

__device__ __forceinline__ double complexity_term(const DMesh& m, int i) {
  const int4 v = m.tri[i];
  if (v.x < 0) return 0.0;
  double2 p0 = m.pts[v.x], p1 = m.pts[v.y], p2 = m.pts[v.z];
  double s0 = p1.x - p0.x;
  double s1 = p2.x - p0.x;
  double s2 = p1.y - p0.y;
  double s3 = p2.y - p0.y;
  double area = 0.5 * (s0 * s3 - s1 * s2);
  double rho = 0.;
  int ids[3] = {v.x, v.y, v.z};
  for (int j = 0; j < 3; ++j) {
    double4 t = m.ten[ids[j]];
    double det = t.x * t.z - trn_pow(t.y, 2);
    rho += sqrt(det);
  }
  rho /= 3;
  return rho * area;
}

/* the global scale and the eigenvalue clamp (metric.cpp:188-238) */
__device__ __forceinline__ double4 normalize_tensor(double4 t, double fact, double eig_min, double eig_max) {
  double mm[4] = {t.x, t.y, t.y, t.z};
  double val[2], vec[4];
  trn_eigen(mm, val, vec);
  val[0] *= fact;
  val[1] *= fact;
  for (int j = 0; j < 2; ++j) {
    val[j] = trn_dmin(val[j], eig_min);
    val[j] = trn_dmax(val[j], eig_max);
  }
  return trn_recompose(val, vec);
}

}  // namespace trn

#endif
