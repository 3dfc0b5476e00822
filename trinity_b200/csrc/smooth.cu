/*
 * smooth.cu — anisotropic smart-Laplacian smoothing (Smooth::run,
 * smoothing.cpp:274-302).
 *
 *   k_smooth_pre   live vertices: interior ones active, boundary ones not
 *                  (smoothing.cpp:129-142)
 *   k_smooth_move  one launch per color class: every listed interior vertex
 *                  moves to the mean over its neighbours b of
 *                  p_a + (p_b - p_a)/L_M(a,b), takes the log-Euclidean mean of
 *                  the neighbours' tensors, and keeps the move only if every
 *                  incident element stays CCW with quality above the old
 *                  stencil minimum, backing off the step 1, 1/2, .., 1/16
 *                  (Smooth::moveSmartLaplacian, smoothing.cpp:40-126).
 *   k_smooth_move_grp  the same with 2, 4 or 8 lanes per vertex (launch shape
 *                  smooth_lanes; the same results)
 * Vertices of one color share no element, so a class moves in parallel; the
 * classes run in order, as in the reference.
 */
#include "trn_internal.h"
#include "trn_mixed.cuh"

#include <algorithm>

namespace trn {

__global__ void k_smooth_pre(DMesh m, int nb_nodes) {
  nb_nodes = trn_nodes(m, nb_nodes);
  for (int v = trn_tid(); v < nb_nodes; v += trn_grid_stride())
    if (m.alive[v]) m.activ[v] = (m.tags[v] & TRN_TAG_BOUND) ? 0 : 1;
}

/* Element metrics of the back-off: the log-Euclidean mean of an element's
 * three tensors (and the square root of its determinant) does not depend on
 * where the moved vertex sits, only on its new tensor, so it is computed once
 * per stencil element before the tries and kept in shared memory (kj slots a
 * thread, stride blockDim.x so that a warp's slots are contiguous); the
 * tries only redo the geometry. Elements past the kj-th (rare: long
 * stencils) take the metric inline. Same operations, same bits as
 * evaluating the whole quality in every try. */
template <bool F32>
using JmT = LogT<F32>;

template <bool F32>
__device__ int move_laplacian(const DMesh& m, int i, JmT<F32>* jc, int kj) {
  const TrnRow vc = trn_row(m.vic, m, i);
  const TrnRow st = trn_row(m.stenc, m, i);
  const int deg = trn_deg(m, i);
  const int nb_neigh = m.vdeg[i];
  double q_min = 1.7976931348623157e308;
  for (int a = 0; a < deg; ++a) q_min = trn_dmin(q_min, m.qual[st[a]]);
  const double2 pini = m.pts[i];
  const double4 tini = m.ten[i];
  const TenT<F32> tinf = ten_load<F32>(m, i);
  const LogT<F32> lini = log_load<F32>(m, i);
  double ox = 0, oy = 0;
  LogSum<F32> lsum;
  if constexpr (F32) {
    /* the mean displacement in single precision, added to the FP64 point */
    float dx = 0.f, dy = 0.f;
    for (int k = 0; k < nb_neigh; ++k) {
      const int nb = vc[k];
      const double2 pb = m.pts[nb];
      const float il = __frcp_rn(trnf_dist2(pini, pb, tenf_of(tinf), tenf_of(ten_load<F32>(m, nb))));
      dx += (float) (pb.x - pini.x) * il;
      dy += (float) (pb.y - pini.y) * il;
      lsum.add(log_load<F32>(m, nb));
    }
    const float inv = __frcp_rn((float) nb_neigh);
    ox = pini.x + (double) (dx * inv);
    oy = pini.y + (double) (dy * inv);
  } else {
    for (int k = 0; k < nb_neigh; ++k) {
      const int nb = vc[k];
      const double2 pb = m.pts[nb];
      const double4 tb = m.ten[nb];
      const double len = length_x<F32>(pini, pb, tini, tb);
      ox += pini.x + ((pb.x - pini.x) / len);
      oy += pini.y + ((pb.y - pini.y) / len);
      lsum.add(log_load<F32>(m, nb));
    }
    ox /= nb_neigh;
    oy /= nb_neigh;
  }
  double tn[3];
  lsum.finish(nb_neigh, tn);
  const double4 tnew = make_double4(tn[0], tn[1], tn[2], 0.0);
  const LogT<F32> lnew = log_of<F32>(tn[0], tn[1], tn[2]);
  ten_store<F32>(m, i, tnew);
  log_store<F32>(m, i, lnew);
  const int nj = deg < kj ? deg : kj;
  for (int a = 0; a < nj; ++a) {
    const int4 n = m.tri[st[a]];
    const LogT<F32> l0 = (n.x == i) ? lnew : log_load<F32>(m, n.x);
    const LogT<F32> l1 = (n.y == i) ? lnew : log_load<F32>(m, n.y);
    const LogT<F32> l2 = (n.z == i) ? lnew : log_load<F32>(m, n.z);
    jc[(size_t) a * blockDim.x] = qmetric_x(l0, l1, l2);
  }
  double qual[TRN_MAX_DEG];
  bool valid;
  int retry = 0;
  double weight = 1;
  do {
    valid = true;
    double2 pa;
    pa.x = (1 - weight) * pini.x + weight * ox;
    pa.y = (1 - weight) * pini.y + weight * oy;
    m.pts[i] = pa;
    for (int a = 0; valid && a < deg; ++a) {
      const int4 n = m.tri[st[a]];
      const double2 p0 = (n.x == i) ? pa : m.pts[n.x];
      const double2 p1 = (n.y == i) ? pa : m.pts[n.y];
      const double2 p2 = (n.z == i) ? pa : m.pts[n.z];
      valid = false;
      if (trn_ccw(p0, p1, p2)) {
        JmT<F32> jm;
        if (a < nj) {
          jm = jc[(size_t) a * blockDim.x];
        } else {
          const LogT<F32> l0 = (n.x == i) ? lnew : log_load<F32>(m, n.x);
          const LogT<F32> l1 = (n.y == i) ? lnew : log_load<F32>(m, n.y);
          const LogT<F32> l2 = (n.z == i) ? lnew : log_load<F32>(m, n.z);
          jm = qmetric_x(l0, l1, l2);
        }
        qual[a] = qgeom_x(p0, p1, p2, jm);
        valid = (qual[a] > q_min);
      }
    }
    weight *= 0.5;
  } while (!valid && ++retry < 5);
  if (valid) {
    for (int a = 0; a < deg; ++a) m.qual[st[a]] = qual[a];
  } else {
    m.pts[i] = pini;
    ten_store<F32>(m, i, tini);
    log_store<F32>(m, i, lini);
  }
  return valid ? 1 : 0;
}

/* the algorithmic bytes of one listed vertex (profiled runs only): its list
 * entry and flags; when it moves, its own point, tensor and logarithm read
 * and written, its stencil and adjacency rows, its elements' records and
 * qualities (read and written), and the point, tensor and logarithm of each
 * neighbour that no other vertex of the launch has counted yet (a bitmap
 * over the vertices keeps them distinct) */
template <bool F32>
__device__ unsigned long long smooth_bytes(const DMesh& m, int v, bool moved, unsigned* seen) {
  constexpr unsigned long long kTenB = F32 ? 16 + 32 : 32;   /* FP32 reads its copy, writes both */
  constexpr unsigned long long kLogB = F32 ? 16 : 32;
  unsigned long long b = 4 + 1 + 4;
  if (!moved) return b;
  const int deg = trn_deg(m, v), nv = m.vdeg[v];
  b += 4 + 2 * (16 + kTenB + kLogB);
  b += (unsigned long long) deg * (4 + 16 + 8 + 8) + (unsigned long long) nv * 4;
  const TrnRow vc = trn_row(m.vic, m, v);
  for (int k = 0; k < nv; ++k) {
    const int w = vc[k];
    const unsigned bit = 1u << (w & 31);
    if (!(atomicOr(seen + (w >> 5), bit) & bit)) b += 16 + (F32 ? 16 : 32) + kLogB;
  }
  return b;
}

/* MinB: 256-thread blocks an SM the registers are capped for (2: up to 128,
 * 3: 80, 4: 64); more warps hide more of the gathers' latency, at the cost of
 * spills */
template <bool F32, int MinB>
__global__ void __launch_bounds__(256, MinB) k_smooth_move(DMesh m, const int* __restrict__ list,
                                                                   int n, const int* off, int c, int* counters,
                                                                   int kj, ByteCount bc) {
  extern __shared__ __align__(16) unsigned char smooth_smem[];
  JmT<F32>* jc = reinterpret_cast<JmT<F32>*>(smooth_smem) + threadIdx.x;
  if (trn_failed(m)) return;
  if (off) {   /* color class c of a device-side partition */
    list += off[c];
    n = off[c + 1] - off[c];
  }
  int tasks = 0, commit = 0;
  unsigned long long bytes = 0;
  for (int q = trn_tid(); q < n; q += trn_grid_stride()) {
    const int v = list[q];
    if (v < 0 || v >= m.capa_node) {
      trn_set_error(m.err, TRN_DERR_REPLAY);
      continue;
    }
    const bool moved = m.activ[v] && m.vdeg[v] != 0;
    if (bc.bytes) bytes += smooth_bytes<F32>(m, v, moved, bc.seen);
    if (!moved) continue;
    tasks++;
    commit += move_laplacian<F32>(m, v, jc, kj);
  }
  trn_warp_add(counters, tasks);
  trn_warp_add(counters + 1, commit);
  if (bytes) atomicAdd(bc.bytes, bytes);
}

/* The same move with G lanes per vertex: lane j gathers the neighbours
 * j, j+G, ... and evaluates the elements j, j+G, ... of the stencil. The
 * displacement and the tensor-logarithm sums are accumulated in neighbour
 * order by every lane from the lanes' terms (shuffles), the stencil minimum
 * is a min-reduction and validity an all-vote, so the results are the bits
 * of move_laplacian. More loads in flight per vertex and no per-thread
 * quality array: the one-lane form is bound by gather latency, divergence
 * and registers. */
template <class T>
__device__ __forceinline__ T grp_shfl(unsigned mask, T v, int src, int width);
template <>
__device__ __forceinline__ double grp_shfl(unsigned mask, double v, int src, int width) {
  return __shfl_sync(mask, v, src, width);
}
template <>
__device__ __forceinline__ float grp_shfl(unsigned mask, float v, int src, int width) {
  return __shfl_sync(mask, v, src, width);
}
template <>
__device__ __forceinline__ double4 grp_shfl(unsigned mask, double4 v, int src, int width) {
  return make_double4(__shfl_sync(mask, v.x, src, width), __shfl_sync(mask, v.y, src, width),
                      __shfl_sync(mask, v.z, src, width), __shfl_sync(mask, v.w, src, width));
}
template <>
__device__ __forceinline__ float4 grp_shfl(unsigned mask, float4 v, int src, int width) {
  return make_float4(__shfl_sync(mask, v.x, src, width), __shfl_sync(mask, v.y, src, width),
                     __shfl_sync(mask, v.z, src, width), __shfl_sync(mask, v.w, src, width));
}

/* quality of stencil element t of vertex i with i at pa (log lnew); false
 * when it is not CCW */
template <bool F32>
__device__ __forceinline__ bool elem_quality_at(const DMesh& m, int i, int4 n, double2 pa, LogT<F32> lnew,
                                                double* q) {
  const double2 p0 = (n.x == i) ? pa : m.pts[n.x];
  const double2 p1 = (n.y == i) ? pa : m.pts[n.y];
  const double2 p2 = (n.z == i) ? pa : m.pts[n.z];
  if (!trn_ccw(p0, p1, p2)) return false;
  const LogT<F32> l0 = (n.x == i) ? lnew : log_load<F32>(m, n.x);
  const LogT<F32> l1 = (n.y == i) ? lnew : log_load<F32>(m, n.y);
  const LogT<F32> l2 = (n.z == i) ? lnew : log_load<F32>(m, n.z);
  *q = quality_x(p0, p1, p2, l0, l1, l2);
  return true;
}

/* a[j] of a small register array, j known only at run time: predicated
 * selects, so the array stays in registers */
template <int K, class T>
__device__ __forceinline__ T reg_pick(const T (&a)[K], int j) {
  T r = a[0];
#pragma unroll
  for (int k = 1; k < K; ++k)
    if (j == k) r = a[k];
  return r;
}

template <int K, class T>
__device__ __forceinline__ void reg_put(T (&a)[K], int j, T v) {
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (j == k) a[k] = v;
}

/* The moved vertex's new tensor (the exponentiated mean of its neighbours'
 * logarithms) and its logarithm, computed by every lane of a group: the two
 * eigenvalues' exp (log) go to the two lanes of a pair, one each, and are
 * swapped by a shuffle, so the group issues one transcendental chain where
 * it issued two. Same functions on the same inputs, composed as
 * trn_interp_finish / trn_log_tensor do: the same bits. FP64 form. */
template <int G>
__device__ __forceinline__ void finish_pair(double* lm, int nb, double* res, int lane, unsigned gmask) {
  double val[2], vec[4], cache[4];
  for (int i = 0; i < 4; ++i) lm[i] /= nb;
  trn_eigen(lm, val, vec);
  const bool h = lane & 1;
  const double mine = trn_exp(h ? val[1] : val[0]);
  const double other = __shfl_xor_sync(gmask, mine, 1, G);
  val[0] = h ? other : mine;
  val[1] = h ? mine : other;
  trn_eigen_compose(val, vec, cache);
  res[0] = cache[0];
  res[1] = cache[1];
  res[2] = cache[3];
}

template <int G>
__device__ __forceinline__ double4 log_pair(double t0, double t1, double t2, int lane, unsigned gmask) {
  double copy[4] = {t0, t1, t1, t2}, val[2], vec[4], cache[4];
  trn_eigen(copy, val, vec);
  const bool h = lane & 1;
  const double mine = trn_log(h ? val[1] : val[0]);
  const double other = __shfl_xor_sync(gmask, mine, 1, G);
  val[0] = h ? other : mine;
  val[1] = h ? mine : other;
  trn_eigen_compose(val, vec, cache);
  return make_double4(cache[0], cache[1], cache[2], cache[3]);
}

/* ---- the sweep's decisions ----
 * A try only needs to know whether every element stays CCW with quality above
 * the old minimum; the qualities themselves are wanted for the one try that
 * is kept. So the sweep decides with a cheap estimate whose error is bounded,
 * evaluates exactly only what the bound leaves open (a floating-point filter,
 * Shewchuk 1997), and the commit evaluates the kept try exactly: the same
 * decisions and the same bits as exact qualities throughout.
 *
 * The element has corners (i, B, C), i moving along pini + w (o - pini). With
 * u = B - pini, v = C - pini, d = o - pini, b = C - B, twice its area is
 * u x v - w d x b and its squared metric edge lengths are
 * |u|^2 - 2 w <u,d> + w^2 |d|^2, the same with v, and |b|^2: three quadratics
 * in w whose coefficients are taken in FP64 once for the five tries. Each
 * value is rounded to FP32, where square roots and reciprocals are one
 * instruction. Error of the estimate, relative, in units of 1e-7: an edge 1.5
 * (conversion 2^-24 halved by the root, root 2^-23), the perimeter p 2.7,
 * min(p/3, 3/p) 5.1, f(2-f) 6.3, its cube 20, 1/p^2 8.4, the products 3:
 * under 32, so 80 (kTryMargin) decides. The FP64 part must stay far below:
 * with t = j0 + j2, every term of a squared length is at most 2 t (|u|^2 +
 * |d|^2) and is rounded to 1e-15 of that, and the tried positions themselves
 * are rounded to e = 1e-15 times the coordinates, which moves a squared length
 * by a relative sqrt(t) e / length; lengths that are not 1e8 times above
 * either, and areas that are not, are left to the exact evaluation (flat or
 * nearly degenerate elements, anisotropy beyond 1e4). Smoothing of two rounds
 * of the 2M-triangle workload, FP64: 8.03 ms with five exact evaluations,
 * 6.57 ms with the estimate (2 lanes, two blocks an SM). */
constexpr float kTryMargin = 8.e-6f;

__device__ __forceinline__ float try_rcp(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

/* bits 0-4: try w passes this element; bits 5-9: try w is undecided */
__device__ __forceinline__ unsigned try_filter(double2 pini, double2 o, double2 B, double2 C, double4 jm,
                                               double q_min) {
  const double dx = o.x - pini.x, dy = o.y - pini.y;
  const double ux = B.x - pini.x, uy = B.y - pini.y, vx = C.x - pini.x, vy = C.y - pini.y;
  const double bx = C.x - B.x, by = C.y - B.y;
  const double mdx = __fma_rn(jm.x, dx, jm.y * dy), mdy = __fma_rn(jm.y, dx, jm.z * dy);
  const double uu = __fma_rn(ux, __fma_rn(jm.x, ux, jm.y * uy), uy * __fma_rn(jm.y, ux, jm.z * uy));
  const double vv = __fma_rn(vx, __fma_rn(jm.x, vx, jm.y * vy), vy * __fma_rn(jm.y, vx, jm.z * vy));
  const double bb = __fma_rn(bx, __fma_rn(jm.x, bx, jm.y * by), by * __fma_rn(jm.y, bx, jm.z * by));
  const double dd = __fma_rn(dx, mdx, dy * mdy);
  const double ud = -2.0 * __fma_rn(ux, mdx, uy * mdy), vd = -2.0 * __fma_rn(vx, mdx, vy * mdy);
  const double h = 0.5 * jm.w;
  const double a0 = h * __fma_rn(ux, vy, -(uy * vx)), a1 = -h * __fma_rn(dx, by, -(dy * bx));
  /* what must be exceeded: lt for the squared lengths, at for area x sqrt(det) */
  const double e = 1.e-15 * (fabs(pini.x) + fabs(pini.y) + fabs(o.x) + fabs(o.y));
  const double L = fabs(ux) + fabs(uy) + fabs(vx) + fabs(vy) + fabs(dx) + fabs(dy);
  const double LL = L * L;
  const float lt = (float) ((jm.x + jm.z) * __fma_rn(4.e-8, LL, 1.e16 * (e * e)));
  const float at = (float) (h * __fma_rn(4.e-8, LL, 1.e8 * (e * L)));
  const float ae = (float) (h * __fma_rn(1.e-14, LL, 1.e1 * (e * L)));
  const float ccw = (float) (2.0 * h * TRN_EPS);
  const float fbb = (float) bb, lb = trnf_sqrt_approx(fbb);
  const float qlo = (float) q_min * (1.f - kTryMargin), qhi = (float) q_min * (1.f + kTryMargin);
  const bool base = fbb > lt && qlo > 1.e-20f;
  unsigned m = 0;
  double w = 1;
#pragma unroll
  for (int k = 0; k < 5; ++k, w *= 0.5) {
    const float fu = (float) __fma_rn(w, __fma_rn(w, dd, ud), uu);
    const float fv = (float) __fma_rn(w, __fma_rn(w, dd, vd), vv);
    const float fa = (float) __fma_rn(w, a1, a0);
    const float p = trnf_sqrt_approx(fu) + trnf_sqrt_approx(fv) + lb;
    const float ip = try_rcp(p);
    const float f = fminf(p * 0.333333343f, 3.f * ip);
    const float g = f * (2.f - f);
    const float q = fa * (20.78460969082653f * (g * g * g)) * (ip * ip);
    const bool sure = base && fu > lt && fv > lt && fa > at && fa > (ccw + ae) * (1.f + 1.e-6f);
    const bool flat = fa + ae < ccw * (1.f - 1.e-6f);   /* certainly not CCW */
    if (sure && q > qhi) m |= 1u << k;
    else if (!(flat || (sure && q < qlo))) m |= 32u << k;
  }
  return m;
}

/* the passing tries of one element (bit w), all five decided */
template <bool F32>
__device__ __forceinline__ unsigned try_mask(const DMesh& m, int i, int4 n, double2 pini, double2 o, JmT<F32> jm,
                                             double q_min) {
  const double2 b0 = (n.x == i) ? pini : m.pts[n.x];
  const double2 b1 = (n.y == i) ? pini : m.pts[n.y];
  const double2 b2 = (n.z == i) ? pini : m.pts[n.z];
  unsigned ok = 0, open = 0x1f;
  if constexpr (!F32) {
    if (n.x == i || n.y == i || n.z == i) {
      const double2 B = n.x == i ? b1 : (n.y == i ? b2 : b0), C = n.x == i ? b2 : (n.y == i ? b0 : b1);
      const unsigned f = try_filter(pini, o, B, C, jm, q_min);
      ok = f & 0x1f;
      open = f >> 5;
    }
    if (!open) return ok;
  }
  double weight = 1;
#pragma unroll
  for (int w = 0; w < 5; ++w, weight *= 0.5) {
    if (!F32 && !(open & (1u << w))) continue;
    double2 pw;
    pw.x = (1 - weight) * pini.x + weight * o.x;
    pw.y = (1 - weight) * pini.y + weight * o.y;
    const double2 p0 = (n.x == i) ? pw : b0;
    const double2 p1 = (n.y == i) ? pw : b1;
    const double2 p2 = (n.z == i) ? pw : b2;
    if (trn_ccw(p0, p1, p2) && qgeom_x(p0, p1, p2, jm) > q_min) ok |= 1u << w;
  }
  return ok;
}

/* the element metric of stencil element n of vertex i, whose new logarithm is lnew */
template <bool F32>
__device__ __forceinline__ JmT<F32> elem_metric(const DMesh& m, int i, int4 n, LogT<F32> lnew) {
  return qmetric_x((n.x == i) ? lnew : log_load<F32>(m, n.x), (n.y == i) ? lnew : log_load<F32>(m, n.y),
                   (n.z == i) ? lnew : log_load<F32>(m, n.z));
}

/* V selects how the back-off runs:
 *   0  the tries in turn, element metrics in registers;
 *   1  one sweep over the lane's elements decides all five tries (try_mask),
 *      the group ANDs the lanes' five-bit pass masks and keeps the first try
 *      that passes, whose qualities the commit evaluates. A warp of 8 groups
 *      or more almost always runs all five tries in turn anyway (half the
 *      moves fail every try), so this costs no extra issue and turns a serial
 *      chain into parallel ones. The element metrics of the lane's first KQ
 *      elements wait in shared memory (stride blockDim.x), which frees
 *      registers; those of later ones (long stencils) are taken again.
 * Same tries, same arithmetic, same first passing try: the same bits. */
template <bool F32, int G, int V>
__device__ int move_laplacian_grp(const DMesh& m, int i, int lane, unsigned gmask, unsigned char* smem) {
  static_assert(G >= 2, "lane groups of two or more");
  constexpr bool SW = V == 1;
  constexpr int KQ = G >= 4 ? 2 : 3;
  JmT<F32>* js = reinterpret_cast<JmT<F32>*>(smem) + threadIdx.x;
  const TrnRow vc = trn_row(m.vic, m, i);
  const TrnRow st = trn_row(m.stenc, m, i);
  const int deg = trn_deg(m, i);
  const int nb_neigh = m.vdeg[i];
  double q_min = 1.7976931348623157e308;
  for (int a = lane; a < deg; a += G) q_min = trn_dmin(q_min, m.qual[st[a]]);
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) q_min = trn_dmin(q_min, __shfl_xor_sync(gmask, q_min, o, G));
  const double2 pini = m.pts[i];
  const double4 tini = m.ten[i];
  const TenT<F32> tinf = ten_load<F32>(m, i);
  using R = typename std::conditional<F32, float, double>::type;
  R sx = 0, sy = 0;
  LogSum<F32> lsum;
  for (int b = 0; b < nb_neigh; b += G) {
    const int k = b + lane;
    R tx = 0, ty = 0;
    LogT<F32> l{};
    if (k < nb_neigh) {
      const int nb = vc[k];
      const double2 pb = m.pts[nb];
      if constexpr (F32) {
        const float il = __frcp_rn(trnf_dist2(pini, pb, tenf_of(tinf), tenf_of(ten_load<F32>(m, nb))));
        tx = (float) (pb.x - pini.x) * il;
        ty = (float) (pb.y - pini.y) * il;
      } else {
        const double len = length_x<F32>(pini, pb, tini, m.ten[nb]);
        tx = pini.x + ((pb.x - pini.x) / len);
        ty = pini.y + ((pb.y - pini.y) / len);
      }
      l = log_load<F32>(m, nb);
    }
    const int cnt = min(G, nb_neigh - b);
    for (int j = 0; j < cnt; ++j) {
      sx += grp_shfl(gmask, tx, j, G);
      sy += grp_shfl(gmask, ty, j, G);
      lsum.add(grp_shfl(gmask, l, j, G));
    }
  }
  double ox, oy;
  if constexpr (F32) {
    const float inv = __frcp_rn((float) nb_neigh);
    ox = pini.x + (double) (sx * inv);
    oy = pini.y + (double) (sy * inv);
  } else {
    ox = sx / nb_neigh;
    oy = sy / nb_neigh;
  }
  double tn[3];
  LogT<F32> lnew;
  if constexpr (!F32) {
    finish_pair<G>(lsum.lm, nb_neigh, tn, lane, gmask);
    lnew = log_pair<G>(tn[0], tn[1], tn[2], lane, gmask);
  } else {
    lsum.finish(nb_neigh, tn);
    lnew = log_of<F32>(tn[0], tn[1], tn[2]);
  }
  const double4 tnew = make_double4(tn[0], tn[1], tn[2], 0.0);
  /* the element metrics of this lane's first KQ elements: they do not depend
   * on where the vertex sits, so the tries below only redo the geometry (a
   * stencil of 6 elements fits: 2 a lane with 4 lanes, 3 with 2) */
  if constexpr (SW) {
    const double2 o = make_double2(ox, oy);
    unsigned okm = 0x1fu;   /* bit w: every element of this lane passes try w */
    int j = 0;
    for (int a = lane; a < deg; a += G, ++j) {
      const int4 n = m.tri[st[a]];
      const JmT<F32> q = elem_metric<F32>(m, i, n, lnew);
      if (j < KQ) js[(size_t) j * blockDim.x] = q;
      okm &= try_mask<F32>(m, i, n, pini, o, q, q_min);
    }
#pragma unroll
    for (int d = G / 2; d > 0; d >>= 1) okm &= __shfl_xor_sync(gmask, okm, d, G);
    if (!okm) return 0;
    double weight = 1;
    for (int w = __ffs(okm) - 1; w > 0; --w) weight *= 0.5;
    double2 pa;
    pa.x = (1 - weight) * pini.x + weight * ox;
    pa.y = (1 - weight) * pini.y + weight * oy;
    j = 0;
    for (int a = lane; a < deg; a += G, ++j) {
      const int4 n = m.tri[st[a]];
      const JmT<F32> q = j < KQ ? js[(size_t) j * blockDim.x] : elem_metric<F32>(m, i, n, lnew);
      const double2 p0 = (n.x == i) ? pa : m.pts[n.x];
      const double2 p1 = (n.y == i) ? pa : m.pts[n.y];
      const double2 p2 = (n.z == i) ? pa : m.pts[n.z];
      m.qual[st[a]] = qgeom_x(p0, p1, p2, q);
    }
    if (lane == 0) {
      m.pts[i] = pa;
      ten_store<F32>(m, i, tnew);
      log_store<F32>(m, i, lnew);
    }
    return 1;
  } else {
    double qv[KQ];
    JmT<F32> jv[KQ];
#pragma unroll
    for (int j = 0; j < KQ; ++j) {
      const int a = lane + j * G;
      if (a < deg) jv[j] = elem_metric<F32>(m, i, m.tri[st[a]], lnew);
    }
    bool valid;
    int retry = 0;
    double weight = 1;
    double2 pa;
    do {
      pa.x = (1 - weight) * pini.x + weight * ox;
      pa.y = (1 - weight) * pini.y + weight * oy;
      bool ok = true;
      int j = 0;
      for (int a = lane; ok && a < deg; a += G, ++j) {
        double q = 0;
        if (j < KQ) {
          const int4 n = m.tri[st[a]];
          const double2 p0 = (n.x == i) ? pa : m.pts[n.x];
          const double2 p1 = (n.y == i) ? pa : m.pts[n.y];
          const double2 p2 = (n.z == i) ? pa : m.pts[n.z];
          ok = trn_ccw(p0, p1, p2);
          if (ok) {
            q = qgeom_x(p0, p1, p2, reg_pick(jv, j));
            ok = q > q_min;
          }
          reg_put(qv, j, q);
        } else {
          ok = elem_quality_at<F32>(m, i, m.tri[st[a]], pa, lnew, &q) && (q > q_min);
        }
      }
      valid = __all_sync(gmask, ok);
      weight *= 0.5;
    } while (!valid && ++retry < 5);
    if (valid) {
      int j = 0;
      for (int a = lane; a < deg; a += G, ++j) {
        double q = 0;
        if (j < KQ) q = reg_pick(qv, j);
        else elem_quality_at<F32>(m, i, m.tri[st[a]], pa, lnew, &q);
        m.qual[st[a]] = q;
      }
      if (lane == 0) {
        m.pts[i] = pa;
        ten_store<F32>(m, i, tnew);
        log_store<F32>(m, i, lnew);
      }
    }
    return valid ? 1 : 0;
  }
}

template <bool F32, int G, int MinB, int V>
__global__ void __launch_bounds__(256, MinB) k_smooth_move_grp(DMesh m, const int* __restrict__ list,
                                                                       int n, const int* off, int c,
                                                                       int* counters, ByteCount bc) {
  extern __shared__ __align__(16) unsigned char smooth_smem[];
  if (trn_failed(m)) return;
  if (off) {
    list += off[c];
    n = off[c + 1] - off[c];
  }
  const int lane = threadIdx.x % G;
  const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) - lane));
  const long long g0 = ((long long) blockIdx.x * blockDim.x + threadIdx.x) / G;
  const long long gs = ((long long) gridDim.x * blockDim.x) / G;
  int tasks = 0, commit = 0;
  unsigned long long bytes = 0;
  for (long long q = g0; q < n; q += gs) {
    const int v = list[q];
    if (v < 0 || v >= m.capa_node) {
      if (lane == 0) trn_set_error(m.err, TRN_DERR_REPLAY);
      continue;
    }
    const bool moved = m.activ[v] && m.vdeg[v] != 0;
    if (bc.bytes && lane == 0) bytes += smooth_bytes<F32>(m, v, moved, bc.seen);
    if (!moved) continue;
    tasks++;
    commit += move_laplacian_grp<F32, G, V>(m, v, lane, gmask, smooth_smem);
  }
  /* the group's tallies sit on its first lane (0 on the others) */
  trn_warp_add(counters, tasks * (lane == 0));
  trn_warp_add(counters + 1, commit * (lane == 0));
  if (lane == 0 && bytes) atomicAdd(bc.bytes, bytes);
}

void smooth_pre(const DMesh& m, int nb_nodes, cudaStream_t s) {
  k_smooth_pre<<<grid_for(nb_nodes), TRN_THREADS, 0, s>>>(m, nb_nodes);
  note_launch();
  check_launch("smooth_pre");
}

/* The default shape (2 lanes, the sweep at 128 registers) stands for a choice
 * by the class's length and the form. A vertex is a chain of gathers and
 * arithmetic: a class too short to fill the chip takes as long as one chain,
 * which more lanes shorten; a long one is bound by issue, which the lanes'
 * shared part (the new tensor) then repeats. Two passes over the classes, ms,
 * by live vertices (a class is a quarter of them at most):
 *   FP64   8 lanes   4 lanes   2 lanes      FP32   8, sweep  8, in turn  2, sweep
 *   10 k   0.42      0.52      0.69         10 k   0.37      0.40        0.57
 *   103 k  0.72      0.76      0.90         103 k  0.58      0.59        0.74
 *   187 k  0.98      0.96      1.08         187 k  0.73      0.72        0.89
 *   294 k  1.35      1.26      1.29         294 k  0.96      0.90        1.03
 *   578 k  2.39      2.12      2.06         578 k  1.67      1.48        1.63 */
static void smooth_shape(int n, bool fp32, int* lanes, int* regs) {
  if (fp32) {
    *lanes = 8;
    *regs = n <= 32768 ? 5 : 2;
  } else if (n <= 65536) {
    *lanes = n <= 32768 ? 8 : 4;
    *regs = n <= 8192 ? 7 : (n <= 32768 ? 5 : 7);
  }
}

static void smooth_launch(const DMesh& m, const int* list, int n, const int* off, int c, int hint,
                          int* counters, bool fp32, cudaStream_t s) {
  /* per moved vertex: list id, flag, counts, own point/tensor read+write,
   * stencil and adjacency rows, its elements and their cached qualities
   * (read+write); neighbours' points/tensors once each (at most 6 per vertex,
   * at most every vertex) */
  const double own = 4 + 1 + 8 + 2 * (kPt + kTen) + kAvgDeg * (2 * kIdx + kTri + 2 * kQ);
  const double nbr = (double) std::min<long long>((long long) m.capa_node, 6LL * n) * (kPt + kTen);
  ByteCount bc;
  ProfScope ps("smooth_move", s, n * own + nbr, &bc);
  const int t = tune().smooth_threads;
  int lanes = tune().smooth_lanes, regs = tune().smooth_regs;
  if (lanes == 2 && regs == 7) smooth_shape(hint, fp32, &lanes, &regs);
  const int g = grid_for((long long) hint * lanes, t);
  if (lanes == 8 || lanes == 4 || lanes == 2) {
    /* smooth_regs 0, 1, 2 (and 3): the tries in turn, registers capped for
     * two, three, four 256-thread blocks an SM; 4, 5 (and 8), 6 (and 7): the
     * sweep, capped for four, three, two, with the element metrics in shared
     * memory (KQ = 2 slots a thread for 4 or 8 lanes, 3 for 2) */
    const int kq = lanes >= 4 ? 2 : 3;
    const size_t js_smem = (size_t) kq * t * (fp32 ? sizeof(float4) : sizeof(double4));
#define TRN_GRP(F, G, B, V)                                                                   \
  do {                                                                                        \
    auto* kern = k_smooth_move_grp<F, G, B, V>;                                               \
    const size_t sm = V == 1 ? js_smem : 0;                                                   \
    kern<<<grid_resident(reinterpret_cast<const void*>(kern), t, g, sm), t, sm, s>>>(m, list, n, off, c, \
                                                                                     counters, bc); \
  } while (0)
#define TRN_GRP_B(F, G)                                                                       \
  do {                                                                                        \
    if (regs == 0) TRN_GRP(F, G, 2, 0);                                                       \
    else if (regs == 1) TRN_GRP(F, G, 3, 0);                                                  \
    else if (regs <= 3) TRN_GRP(F, G, 4, 0);                                                  \
    else if (regs == 4) TRN_GRP(F, G, 4, 1);                                                  \
    else if (regs == 5 || regs == 8) TRN_GRP(F, G, 3, 1);                                     \
    else TRN_GRP(F, G, 2, 1);                                                                 \
  } while (0)
    if (lanes == 8) {
      if (fp32) TRN_GRP_B(true, 8);
      else TRN_GRP_B(false, 8);
    } else if (lanes == 4) {
      if (fp32) TRN_GRP_B(true, 4);
      else TRN_GRP_B(false, 4);
    } else {
      if (fp32) TRN_GRP_B(true, 2);
      else TRN_GRP_B(false, 2);
    }
#undef TRN_GRP_B
#undef TRN_GRP
  } else {
    /* element-metric slots a thread: what 40 KB of shared memory a block
     * holds, at most 8 (FP64) or 12 (FP32) */
    const int slot = fp32 ? (int) sizeof(float4) : (int) sizeof(double4);
    const int kj = std::min(fp32 ? 12 : 8, (40 << 10) / (t * slot));
    const size_t smem = (size_t) kj * t * slot;
#define TRN_ONE(F, B)                                                                           \
  do {                                                                                          \
    auto* kern = k_smooth_move<F, B>;                                                           \
    kern<<<grid_resident(reinterpret_cast<const void*>(kern), t, g, smem), t, smem, s>>>(m, list, n, off, \
                                                                                        c, counters, kj, bc); \
  } while (0)
#define TRN_ONE_B(F) \
  do { if (regs == 0) TRN_ONE(F, 2); else if (regs == 1) TRN_ONE(F, 3); else TRN_ONE(F, 4); } while (0)
    if (fp32) TRN_ONE_B(true);
    else TRN_ONE_B(false);
#undef TRN_ONE_B
#undef TRN_ONE
  }
  note_launch();
  check_launch("smooth_move");
}

void smooth_color(const DMesh& m, const int* list, int n, int* counters, bool fp32, cudaStream_t s) {
  if (n <= 0) return;
  smooth_launch(m, list, n, nullptr, 0, n, counters, fp32, s);
}

void smooth_class(const DMesh& m, const int* parts, const int* part_off, int c, int hint, int* counters,
                  bool fp32, cudaStream_t s) {
  smooth_launch(m, parts, hint, part_off, c, hint, counters, fp32, s);
}

}  // namespace trn
