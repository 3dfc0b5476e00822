/*
 * smooth.cu — anisotropic smart-Laplacian smoothing (Smooth::run,
 * smoothing.cpp:274-302).
 *
 *   k_smooth_pre   live vertices: interior ones active, boundary ones not
 *                  (smoothing.cpp:129-142)
 *   k_smooth_move_grp  one launch per color class: every listed interior
 *                  vertex (by 2, 4 or 8 lanes) moves to the mean over its neighbours b of
 *                  p_a + (p_b - p_a)/L_M(a,b), takes the log-Euclidean mean of
 *                  the neighbours' tensors, and keeps the move only if every
 *                  incident element stays CCW with quality above the old
 *                  stencil minimum, backing off the step 1, 1/2, .., 1/16
 *                  (Smooth::moveSmartLaplacian, smoothing.cpp:40-126).
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
 * per stencil element before the tries; the tries only redo the geometry.
 * Same operations, same bits as evaluating the whole quality in every try. */
template <bool F32>
using JmT = LogT<F32>;

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

/* A move by G lanes per vertex: lane j gathers the neighbours j, j+G, ... and
 * evaluates the elements j, j+G, ... of the stencil. The displacement and the
 * tensor-logarithm sums are accumulated in neighbour order by every lane from
 * the lanes' terms (shuffles), the stencil minimum is a min-reduction and
 * validity a vote, so the results are those of one lane in the reference's
 * order. */
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

template <bool F32>
struct VertexPark {
  double2 pini, o;
  double tn[3], q_min;
  LogT<F32> lnew;
};

/* One sweep over the lane's elements decides all five tries (try_mask), the
 * group ANDs the lanes' five-bit pass masks and keeps the first try that
 * passes, whose qualities the commit evaluates. A warp of 4 groups or more
 * almost always needs every try of some group anyway (half the moves fail all
 * five), so this costs no extra issue over trying in turn, and turns a serial
 * chain into parallel ones. The element metrics of the lane's first KQ elements
 * wait in shared memory (stride blockDim.x); those of later ones (long
 * stencils) are taken again. What the elements need of the vertex waits there
 * too (VertexPark): held in registers over the element loop it took 128 of
 * them, or spilled; without it 80 hold the kernel, three 256-thread blocks an
 * SM instead of two, and 64 all but 128 bytes. Two passes over the classes of
 * the 2M-triangle workload, FP64 / mixed: 6.49 / 4.98 ms before, 5.61 / 4.32. */
template <bool F32, int G>
__device__ int move_laplacian_grp(const DMesh& m, int i, int lane, unsigned gmask, unsigned char* smem) {
  static_assert(G >= 2, "lane groups of two or more");
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
  VertexPark<F32>* park = reinterpret_cast<VertexPark<F32>*>(smem + (size_t) KQ * blockDim.x * sizeof(JmT<F32>)) +
                          threadIdx.x / G;
  if (lane == 0) {
    park->pini = pini;
    park->o = make_double2(ox, oy);
    park->q_min = q_min;
    park->tn[0] = tn[0];
    park->tn[1] = tn[1];
    park->tn[2] = tn[2];
    park->lnew = lnew;
  }
  __syncwarp(gmask);
  unsigned okm = 0x1fu;   /* bit w: every element of this lane passes try w */
  int j = 0;
  for (int a = lane; a < deg; a += G, ++j) {
    const int4 n = m.tri[st[a]];
    const JmT<F32> q = elem_metric<F32>(m, i, n, park->lnew);
    if (j < KQ) js[(size_t) j * blockDim.x] = q;
    okm &= try_mask<F32>(m, i, n, park->pini, park->o, q, park->q_min);
  }
#pragma unroll
  for (int d = G / 2; d > 0; d >>= 1) okm &= __shfl_xor_sync(gmask, okm, d, G);
  if (okm) {
    double weight = 1;
    for (int w = __ffs(okm) - 1; w > 0; --w) weight *= 0.5;
    double2 pa;
    pa.x = (1 - weight) * park->pini.x + weight * park->o.x;
    pa.y = (1 - weight) * park->pini.y + weight * park->o.y;
    j = 0;
    for (int a = lane; a < deg; a += G, ++j) {
      const int4 n = m.tri[st[a]];
      const JmT<F32> q = j < KQ ? js[(size_t) j * blockDim.x] : elem_metric<F32>(m, i, n, park->lnew);
      const double2 p0 = (n.x == i) ? pa : m.pts[n.x];
      const double2 p1 = (n.y == i) ? pa : m.pts[n.y];
      const double2 p2 = (n.z == i) ? pa : m.pts[n.z];
      m.qual[st[a]] = qgeom_x(p0, p1, p2, q);
    }
    if (lane == 0) {
      m.pts[i] = pa;
      ten_store<F32>(m, i, make_double4(park->tn[0], park->tn[1], park->tn[2], 0.0));
      log_store<F32>(m, i, park->lnew);
    }
  }
  __syncwarp(gmask);   /* the next vertex reuses the place */
  return okm ? 1 : 0;
}

/* MinB: 256-thread blocks an SM the registers are capped for (2: 112 are
 * used, 3: 80, 4: 64) */
template <bool F32, int G, int MinB>
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
    commit += move_laplacian_grp<F32, G>(m, v, lane, gmask, smooth_smem);
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

/* the blocks an SM that the values of smooth_regs cap the registers for */
static constexpr int kRegsBlocks[9] = {2, 3, 4, 4, 4, 3, 2, 2, 3};

/* The default shape (2 lanes, smooth_regs 7) stands for a choice by the class's
 * length and the form. A vertex is a chain of gathers and arithmetic: a class
 * too short to fill the chip takes as long as one chain, which more lanes
 * shorten; a long one is bound by issue, which the lanes' shared part (the new
 * tensor) then repeats. Two passes over the classes, ms, by live vertices (a
 * class is a quarter of them at most), lanes x 256-thread blocks an SM:
 *   FP64    8 x 3   4 x 4   2 x 3      mixed   8 x 4   4 x 4   2 x 4
 *   23 k    0.47    0.59    0.75       23 k    0.41    0.50    0.65
 *   187 k   0.89    0.92    1.02       187 k   0.69    0.74    0.86
 *   294 k   1.20    1.13    1.28       294 k   0.86    0.88    0.96
 *   578 k   2.12    1.86    1.89       578 k   1.41    1.36    1.42
 *   1181 k  3.95    3.34    3.10       1181 k  2.58    2.38    2.45 */
static void smooth_shape(int n, bool fp32, int* lanes, int* blocks) {
  if (fp32) {
    *lanes = n <= 98304 ? 8 : 4;
    *blocks = 4;
  } else if (n <= 49152) {
    *lanes = 8;
    *blocks = 3;
  } else if (n <= 163840) {
    *lanes = 4;
    *blocks = 4;
  } else {
    *lanes = 2;
    *blocks = 3;
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
  const int regs = tune().smooth_regs;
  int lanes = std::max(2, tune().smooth_lanes), blocks = kRegsBlocks[regs];
  if (tune().smooth_lanes == 2 && regs == 7) smooth_shape(hint, fp32, &lanes, &blocks);
  const int g = grid_for((long long) hint * lanes, t);
  /* KQ element metrics a thread, a VertexPark a vertex */
  const size_t smem = (size_t) (lanes >= 4 ? 2 : 3) * t * (fp32 ? sizeof(float4) : sizeof(double4)) +
                      (size_t) (t / lanes) * (fp32 ? sizeof(VertexPark<true>) : sizeof(VertexPark<false>));
#define TRN_GRP(F, G, B)                                                                         \
  do {                                                                                           \
    auto* kern = k_smooth_move_grp<F, G, B>;                                                     \
    kern<<<grid_resident(reinterpret_cast<const void*>(kern), t, g, smem), t, smem, s>>>(        \
        m, list, n, off, c, counters, bc);                                                       \
  } while (0)
#define TRN_GRP_B(F, G)                                                                          \
  do {                                                                                           \
    if (blocks == 2) TRN_GRP(F, G, 2);                                                           \
    else if (blocks == 3) TRN_GRP(F, G, 3);                                                      \
    else TRN_GRP(F, G, 4);                                                                       \
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
