/*
 * metric.cu — Hessian-based metric recovery (Metrics::run, metric.cpp:59-70).
 *
 *   k_elem_gradient   per element: its signed area and area x P1 gradient
 *   k_patch_sum<GradSum>  per vertex: area-weighted mean of those over the
 *                     2-ring element patch (hessian.cpp:24-83)
 *   k_elem_hessian    per element: area x the gradient field's derivatives
 *   k_patch_sum<HessSum>  per vertex: their mean, symmetrised
 *                     (hessian.cpp:86-153), then |H| eigen-clamp and local L^p
 *                     scale det^(-1/(2p+2)) (metric.cpp:100-150), fused
 *   k_sum_terms       per element: area * mean_k sqrt(det M_k)
 *                     (metric.cpp:159-181), summed by a deterministic
 *                     two-level tree (k_sum_final), or
 *   k_complexity_term, k_sum_sequential  by one thread in element order
 *                     (bit-identical to the reference's 1-thread sum)
 *   k_normalize       global scale target/complexity and eigenvalue clamp to
 *                     [1/h_max^2, 1/h_min^2] (metric.cpp:188-238)
 *   k_elem_edges, *Sum32, k_normalize_f32   the same recovery in FP32 for the
 *                     mixed-precision form
 *
 * Patch order matters: the reference sums over the patch in ascending element
 * id (std::set order, mesh.cpp:396-432), so the union of the stencils of the
 * vertex and of its neighbours is sorted and deduplicated first
 * (trn_patch.cuh): in registers where the rows are short, by a warp or a lane
 * for the vertices that the first pass lists as not fitting.
 */
#include "trn_internal.h"
#include "trn_metric.cuh"
#include "trn_mixed.cuh"

namespace trn {

__global__ void k_elem_gradient(DMesh m, int nb_elems, const double* __restrict__ solut,
                                double4* __restrict__ rec) {
  if (trn_failed(m)) return;
  for (int t = trn_tid(); t < nb_elems; t += trn_grid_stride()) rec_store(rec, t, kRecMix, elem_gradient(m, t, solut));
}

__global__ void k_elem_hessian(DMesh m, int nb_elems, const double2* __restrict__ grad,
                               double4* __restrict__ rec) {
  if (trn_failed(m)) return;
  for (int t = trn_tid(); t < nb_elems; t += trn_grid_stride()) rec_store(rec, t, kRecMix, elem_hessian(m, t, grad));
}

/* ---- the mixed-precision form of the recovery ----
 * The same patch means in FP32. Every coordinate difference is taken in
 * FP64 and then rounded; each nodal value enters as its difference to the
 * patch centre's value (the element's three P1 basis gradients sum to zero,
 * so this changes nothing in exact arithmetic and removes the cancellation
 * of summing values of nearly equal size, which single precision could not
 * afford); area x basis gradient is formed directly from the rotated edges
 * (area x 2/area x edge), so no division per element. The eigen-clamp, the
 * local L^p scale and the global scaling are FP32 too; the complexity sum
 * stays FP64. An element's record holds its area and rotated edges; the
 * differences to the centre are the patch's own. */
struct Edges32 {
  float4 a, b;   /* area, ey[3]; ex[3], unused */
};

__global__ void k_elem_edges(DMesh m, int nb_elems, float4* __restrict__ rec) {
  if (trn_failed(m)) return;
  for (int i = trn_tid(); i < nb_elems; i += trn_grid_stride()) {
    const int4 t = m.tri[i];
    if (t.x < 0) continue;
    const double2 p0 = m.pts[t.x], p1 = m.pts[t.y], p2 = m.pts[t.z];
    /* rotated edges: area x d[2j] = 2 ey[j], area x d[2j+1] = 2 ex[j] */
    const float c0 = (float) (p1.x - p0.x), c1 = (float) (p2.x - p0.x);
    const float c2 = (float) (p1.y - p0.y), c3 = (float) (p2.y - p0.y);
    const size_t at = rec_slot(i, kRecMix);
    rec[at] = make_float4(0.5f * (c0 * c3 - c1 * c2), (float) (p1.y - p2.y), (float) (p2.y - p0.y),
                                      (float) (p0.y - p1.y));
    rec[at ^ 1] = make_float4((float) (p2.x - p1.x), (float) (p0.x - p2.x), (float) (p1.x - p0.x), 0.f);
  }
}

struct GradSum32 {
  const float4* rec;
  const double* solut;
  double2* grad;
  double uv = 0;
  float tot = 0.f, gx = 0.f, gy = 0.f;
  struct Rec {
    Edges32 e;
    double u[3];
  };
  __device__ __forceinline__ void begin(const DMesh&, int v) { uv = solut[v]; }
  __device__ __forceinline__ Rec load(const DMesh& m, int i) const {
    const int4 t = m.tri[i];
    const size_t at = rec_slot(i, kRecMix);
    return Rec{{rec[at], rec[at ^ 1]}, {solut[t.x], solut[t.y], solut[t.z]}};
  }
  __device__ __forceinline__ void add(const Rec& r) {
    const float s[3] = {(float) (r.u[0] - uv), (float) (r.u[1] - uv), (float) (r.u[2] - uv)};
    tot += r.e.a.x;
    gx += 2.f * (s[0] * r.e.a.y + s[1] * r.e.a.z + s[2] * r.e.a.w);
    gy += 2.f * (s[0] * r.e.b.x + s[1] * r.e.b.y + s[2] * r.e.b.z);
  }
  __device__ __forceinline__ void finish(const DMesh&, int v) {
    const float it = __frcp_rn(tot);
    grad[v] = make_double2((double) (gx * it), (double) (gy * it));
  }
};

struct HessSum32 {
  const float4* rec;
  const double2* grad;
  float scale_exp;
  double2 gv = {0, 0};
  float tot = 0.f, h[4] = {0.f, 0.f, 0.f, 0.f};
  struct Rec {
    Edges32 e;
    double2 g[3];
  };
  __device__ __forceinline__ void begin(const DMesh&, int v) { gv = grad[v]; }
  __device__ __forceinline__ Rec load(const DMesh& m, int i) const {
    const int4 t = m.tri[i];
    const size_t at = rec_slot(i, kRecMix);
    return Rec{{rec[at], rec[at ^ 1]}, {grad[t.x], grad[t.y], grad[t.z]}};
  }
  __device__ __forceinline__ void add(const Rec& r) {
    tot += r.e.a.x;
    const float ey[3] = {r.e.a.y, r.e.a.z, r.e.a.w}, ex[3] = {r.e.b.x, r.e.b.y, r.e.b.z};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float dx = (float) (r.g[j].x - gv.x), dy = (float) (r.g[j].y - gv.y);
      h[0] += 2.f * (dx * ey[j]);
      h[1] += 2.f * (dx * ex[j]);
      h[2] += 2.f * (dy * ey[j]);
      h[3] += 2.f * (dy * ex[j]);
    }
  }
  __device__ __forceinline__ void finish(const DMesh& m, int v) {
    const float it = __frcp_rn(tot);
    const float t0 = h[0] * it, t1 = 0.5f * (h[1] + h[2]) * it, t2 = h[3] * it;
    float mm[4] = {t0, t1, t1, t2}, val[2], vec[4];
    trnf_eigen(mm, val, vec);
    val[0] = trnf_max(fabsf(val[0]), 1.e-9f);
    val[1] = trnf_max(fabsf(val[1]), 1.e-9f);
    const float scale_loc = powf(val[0] * val[1], scale_exp);
    val[0] *= scale_loc;
    val[1] *= scale_loc;
    const float c0 = val[0] * vec[0], c1 = val[0] * vec[2], c2 = val[1] * vec[1], c3 = val[1] * vec[3];
    m.ten[v] = make_double4((double) (vec[0] * c0 + vec[1] * c2), (double) (vec[0] * c1 + vec[1] * c3),
                            (double) (vec[2] * c1 + vec[3] * c3), 0.0);
  }
};

constexpr int kPatchThreads = 128;
constexpr int kPatchIds = 48;   /* an interior patch of these rows has 42 at most */
constexpr int kPatchBatch = 4;  /* records in flight a thread (2: 5% slower at 100 k vertices; 8: spills) */

/* The merged ids go to shared memory, so that the sums are a loop over the
 * patch instead of 64 predicated slots and the merge's registers are free
 * again: 5 blocks a multiprocessor where the sums over the registers had 3 (4
 * are as fast, 6 spill in single precision). Bound by the shared-memory data
 * path's wavefronts (80% of its peak before rec_slot mixed the records'
 * banks). Recovery of 1 002 001 vertices 517 us, 480 with the column, 445 with
 * the mixed records; of 101 124 vertices in single precision 140, 126, 116.
 * A vertex whose rows do not fit goes onto rest[*rest_n] (when given; the
 * second pass over the same rows finds the same ones) */
template <class Sum>
__global__ void __launch_bounds__(kPatchThreads, 5) k_patch_sum(DMesh m, int nb_nodes, Sum zero, int* rest,
                                                                int* rest_n) {
  __shared__ int s_ids[kPatchIds * kPatchThreads];
  if (trn_failed(m)) return;
  for (int v = trn_tid(); v < nb_nodes; v += trn_grid_stride())
    if (!patch_sum_column<Sum, kPatchBatch, kPatchIds, kPatchThreads>(m, v, zero, s_ids + threadIdx.x) && rest)
      trn_append(rest, rest_n, v);
}

/* The listed vertices, a warp each, or, where they are many and a good part of
 * the mesh, a lane each. A warp is quick about one patch but spends 32 lanes on
 * its serial sum: 2.4 to 6 ns a vertex, by the patch's length and the form,
 * against a lane's 1 ns behind some 100 us of latency. Lists that are long but
 * a small part of the mesh are spread over it, and a lane's gathers are then
 * alone on their cache lines. us a recovery, warps / lanes, FP64 and (mixed):
 * triangles cut in three (every vertex listed) 19,361 vertices 261 / 224 (343 /
 * 237), 36,521 386 / 253 (594 / 299), 270,601 2,208 / 683 (3,604 / 846); random
 * points (45 % listed) 60,000 302 / 409 (483 / 494), 250,000 866 / 743 (1,588 /
 * 1,071); an adapted mesh (15 %) of 354,918 453 / 611 (634 / 772). */
constexpr int kRestWarps = 32768;
/* records in flight a lane: at 4 the 80-byte records of the mixed form take 102
 * registers, and the warps' branch of the same kernel pays (1,611 -> 2,078 us
 * at 120,401 listed vertices) */
template <class Sum>
constexpr int kRestBatch = sizeof(typename Sum::Rec) > 32 ? 2 : 4;

template <class Sum>
__global__ void __launch_bounds__(kPatchThreads) k_patch_sum_rest(DMesh m, int nb_nodes, Sum zero,
                                                                  const int* rest, const int* rest_n) {
  __shared__ int s_buf[kPatchThreads / 32][TRN_MAX_PATCH];
  if (trn_failed(m)) return;
  const int n = *rest_n;
  if (n > kRestWarps && 4LL * n > nb_nodes) {
    int ids[TRN_MAX_PATCH];
    for (int q = trn_tid(); q < n; q += trn_grid_stride()) {
      const int v = rest[q], k = patch_sort_lane(m, v, ids);
      Sum s = zero;
      s.begin(m, v);
      for (int c = 0; c < k; c += kRestBatch<Sum>) {
        typename Sum::Rec r[kRestBatch<Sum>];
#pragma unroll
        for (int j = 0; j < kRestBatch<Sum>; ++j) r[j] = s.load(m, ids[min(c + j, k - 1)]);
#pragma unroll
        for (int j = 0; j < kRestBatch<Sum>; ++j)
          if (c + j < k) s.add(r[j]);
      }
      s.finish(m, v);
    }
    return;
  }
  for (int q = trn_tid() >> 5; q < n; q += trn_grid_stride() >> 5)
    patch_sum_warp(m, rest[q], zero, s_buf[threadIdx.x >> 5]);
}

__global__ void k_complexity_term(DMesh m, int nb_elems, double* __restrict__ terms) {
  if (trn_failed(m)) return;
  for (int i = trn_tid(); i < nb_elems; i += trn_grid_stride()) terms[i] = complexity_term(m, i);
}

/* one thread, element order: the 1-thread reference's summation */
__global__ void k_sum_sequential(const double* __restrict__ terms, int n, double* out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double phi = 0.;
  int i = 0;
  for (; i + 8 <= n; i += 8) {
    double a0 = terms[i], a1 = terms[i + 1], a2 = terms[i + 2], a3 = terms[i + 3];
    double a4 = terms[i + 4], a5 = terms[i + 5], a6 = terms[i + 6], a7 = terms[i + 7];
    phi += a0; phi += a1; phi += a2; phi += a3;
    phi += a4; phi += a5; phi += a6; phi += a7;
  }
  for (; i < n; ++i) phi += terms[i];
  *out = 0 + phi;
}

/* deterministic tree: fixed per-block partials, then one block in order */
__device__ __forceinline__ void block_partial(double s, double* partial) {
  __shared__ double sm[TRN_THREADS];
  sm[threadIdx.x] = s;
  __syncthreads();
  for (int o = TRN_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sm[threadIdx.x] += sm[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sm[0];
}

__global__ void k_sum_partial(const double* __restrict__ terms, int n, double* partial) {
  double s = 0;
  for (int i = trn_tid(); i < n; i += trn_grid_stride()) s += terms[i];
  block_partial(s, partial);
}

/* the elements' complexity terms straight into the tree's first level */
__global__ void k_sum_terms(DMesh m, int nb_elems, double* partial) {
  double s = 0;
  if (!trn_failed(m))
    for (int i = trn_tid(); i < nb_elems; i += trn_grid_stride()) s += complexity_term(m, i);
  block_partial(s, partial);
}

__global__ void k_sum_final(const double* __restrict__ partial, int nb, double* out) {
  __shared__ double sm[TRN_THREADS];
  double s = 0;
  for (int i = threadIdx.x; i < nb; i += TRN_THREADS) s += partial[i];
  sm[threadIdx.x] = s;
  __syncthreads();
  for (int o = TRN_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sm[threadIdx.x] += sm[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sm[0];
}

__global__ void k_normalize(DMesh m, int nb_nodes, const double* complexity, double target,
                            double eig_min, double eig_max) {
  if (trn_failed(m)) return;
  double fact = target / *complexity;
  for (int v = trn_tid(); v < nb_nodes; v += trn_grid_stride()) {
    const double4 t4 = normalize_tensor(m.ten[v], fact, eig_min, eig_max);
    m.ten[v] = t4;
    if (m.lten) m.lten[v] = trn_log_tensor(t4.x, t4.y, t4.z);
  }
}

__global__ void k_normalize_f32(DMesh m, int nb_nodes, const double* complexity, double target,
                                double eig_min, double eig_max) {
  if (trn_failed(m)) return;
  const float fact = (float) (target / *complexity);
  const float lo = (float) eig_max, hi = (float) eig_min;
  for (int v = trn_tid(); v < nb_nodes; v += trn_grid_stride()) {
    const double4 t = m.ten[v];
    float mm[4] = {(float) t.x, (float) t.y, (float) t.y, (float) t.z}, val[2], vec[4];
    trnf_eigen(mm, val, vec);
    for (int j = 0; j < 2; ++j) val[j] = trnf_max(trnf_min(val[j] * fact, hi), lo);
    const float c0 = val[0] * vec[0], c1 = val[0] * vec[2], c2 = val[1] * vec[1], c3 = val[1] * vec[3];
    const float r0 = vec[0] * c0 + vec[1] * c2, r1 = vec[0] * c1 + vec[1] * c3, r2 = vec[2] * c1 + vec[3] * c3;
    m.ten[v] = make_double4((double) r0, (double) r1, (double) r2, 0.0);
    if (m.tenf) m.tenf[v] = make_float4(r0, r1, r2, 0.f);
    if (m.lten) reinterpret_cast<float4*>(m.lten)[v] = trnf_log_tensor(r0, r1, r2);
  }
}

void sum_tree(const double* in, int n, double* partial, double* out, cudaStream_t s) {
  const int nb = grid_for(n);
  k_sum_partial<<<nb, TRN_THREADS, 0, s>>>(in, n, partial);
  note_launch();
  k_sum_final<<<1, TRN_THREADS, 0, s>>>(partial, nb, out);
  note_launch();
}

/* a patch mean: the elements' records are ready in ws.rec; the vertices
 * that the register merge cannot take are listed by the first pass (collect)
 * and served by the second kernel, which returns at once when there are none */
template <class Sum>
static void patch_sum(const DMesh& m, int nb_nodes, const Sum& zero, const MetricWs& ws, bool collect,
                      cudaStream_t s) {
  auto* fast = k_patch_sum<Sum>;
  auto* rest = k_patch_sum_rest<Sum>;
  fast<<<TRN_RESIDENT(fast, grid_for(nb_nodes, kPatchThreads), kPatchThreads), kPatchThreads, 0, s>>>(
      m, nb_nodes, zero, collect ? ws.rest : nullptr, ws.rest_n);
  note_launch();
  rest<<<TRN_RESIDENT(rest, grid_for(32LL * nb_nodes, kPatchThreads), kPatchThreads), kPatchThreads, 0, s>>>(
      m, nb_nodes, zero, ws.rest, ws.rest_n);
  note_launch();
}

void metric_patches(const DMesh& m, int nb_nodes, int nb_elems, const double* solut, double2* grad,
                    const MetricWs& ws, double scale_exp, cudaStream_t s, const MetricSaves* keep, bool fp32) {
  const double V = nb_nodes, E = nb_elems;
  const int ge = grid_for(nb_elems);
  cudaMemsetAsync(ws.rest_n, 0, sizeof(int), s);
  if (fp32) {
    float4* rec = reinterpret_cast<float4*>(ws.rec);
    {
    ProfScope ps("metric_gradient", s, V * (2 * kIdx + kAvgDeg * kIdx * 2 + 8 + kPt + 16) + E * kTri);
    k_elem_edges<<<ge, TRN_THREADS, 0, s>>>(m, nb_elems, rec);
    note_launch();
    GradSum32 z{rec, solut, grad};
    patch_sum(m, nb_nodes, z, ws, true, s);
    }
    ProfScope ps("metric_hessian", s, V * (2 * kIdx + kAvgDeg * kIdx * 2 + 16 + kPt + kTen) + E * kTri);
    HessSum32 z{rec, grad, (float) scale_exp};
    patch_sum(m, nb_nodes, z, ws, false, s);
    return;
  }
  double* atot = keep && keep->atot ? keep->atot : ws.atot;
  {
  ProfScope ps("metric_gradient", s, V * (2 * kIdx + kAvgDeg * kIdx * 2 + 8 + kPt + 16) + E * kTri);
  k_elem_gradient<<<ge, TRN_THREADS, 0, s>>>(m, nb_elems, solut, ws.rec);
  note_launch();
  GradSum z{ws.rec, kRecMix, grad, atot};
  patch_sum(m, nb_nodes, z, ws, true, s);
  }
  ProfScope ps("metric_hessian", s, V * (2 * kIdx + kAvgDeg * kIdx * 2 + 16 + kPt + kTen) + E * kTri);
  k_elem_hessian<<<ge, TRN_THREADS, 0, s>>>(m, nb_elems, grad, ws.rec);
  note_launch();
  HessSum z{ws.rec, kRecMix, atot, scale_exp, keep ? keep->hsym : nullptr, keep ? keep->mloc : nullptr};
  patch_sum(m, nb_nodes, z, ws, false, s);
}

void metric_complexity(const DMesh& m, int nb_elems, double* terms, double* partial, double* complexity,
                       bool exact_sum, cudaStream_t s) {
  if (exact_sum) {
    k_complexity_term<<<grid_for(nb_elems), TRN_THREADS, 0, s>>>(m, nb_elems, terms);
    note_launch();
    k_sum_sequential<<<1, 32, 0, s>>>(terms, nb_elems, complexity);
    note_launch();
    return;
  }
  const int nb = grid_for(nb_elems);
  k_sum_terms<<<nb, TRN_THREADS, 0, s>>>(m, nb_elems, partial);
  note_launch();
  k_sum_final<<<1, TRN_THREADS, 0, s>>>(partial, nb, complexity);
  note_launch();
}

void metric_run(const DMesh& m, int nb_nodes, int nb_elems, const double* solut, double2* grad,
                double* terms, double* complexity, bool exact_sum, const MetricParams& p, const MetricWs& ws,
                cudaStream_t s, const MetricSaves* keep, bool fp32) {
  const double V = nb_nodes, E = nb_elems;
  metric_patches(m, nb_nodes, nb_elems, solut, grad, ws, p.scale_exp, s, keep, fp32);
  {
  ProfScope ps("metric_complexity", s, E * (kTri + 8) + V * (kPt + kTen));
  /* partials live after the terms (terms has capa_elem + grid slots) */
  metric_complexity(m, nb_elems, terms, terms + m.capa_elem, complexity, exact_sum, s);
  }
  ProfScope ps("metric_normalize", s, V * 2 * kTen);
  if (fp32)
    k_normalize_f32<<<grid_for(nb_nodes), TRN_THREADS, 0, s>>>(m, nb_nodes, complexity, p.target, p.eig_min,
                                                              p.eig_max);
  else
    k_normalize<<<grid_for(nb_nodes), TRN_THREADS, 0, s>>>(m, nb_nodes, complexity, p.target, p.eig_min,
                                                          p.eig_max);
  note_launch();
  check_launch("metric_run");
}

}  // namespace trn
