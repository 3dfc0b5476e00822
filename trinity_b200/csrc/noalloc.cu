/*
 * noalloc.cu — metric recovery for one small mesh without any device
 * allocation: trn_metric_noalloc (declared in include/trinity_b200.h).
 *
 * Who needs it: a caller that owns every byte of device memory itself — a
 * solver running on a fixed, pre-reserved memory budget, or one whose device
 * memory all comes from its own pool allocator — may not let a library call
 * cudaMalloc/cudaFree in the middle of its time stepping (those calls also
 * synchronise the device). Such a caller hands over its own device buffers for
 * the input and the output; everything else this computation needs lives in
 * one file-scope __device__ array below.
 *
 * The scratch array is sized for at most TRN_NOALLOC_MAX_NODES vertices,
 * TRN_NOALLOC_MAX_ELEMS triangles and TRN_NOALLOC_BUCKET triangles around one
 * vertex; it takes about 7 MB on every GPU that loads this library, for as
 * long as the process lives. Every call on a device shares it: calls that
 * overlap on the GPU (other streams, other host threads) race and corrupt
 * each other's results, so serialise them. The array keeps the last call's
 * contents; each call starts by clearing what must be empty.
 *
 * Host code cannot use the array's name as a device address (in host code it
 * names a host-side stand-in), so the first call on each device looks the
 * address up with cudaGetSymbolAddress while that device is current and keeps
 * it.
 *
 * The computation is trn_metric_run's, step by step (gradient, Hessian with
 * local L^p scaling, complexity with the fixed-shape tree sum, global
 * scaling; trn_metric.cuh), so the tensors are identical to it when that
 * mesh also sums with the tree (its default; exact_sum and replay sum in
 * element order): in one launch of one cluster, or by its kernels where many
 * vertices have long rows or the device has no room for a cluster. They run on the caller's stream with the address
 * looked up for the current device, so the stream must belong to it.
 */
#include "trn_internal.h"
#include "trn_level.cuh"
#include "trn_libm.h"
#include "trn_metric.cuh"
#include "../../include/trinity_b200.h"

#include <cmath>
#include <cstdio>
#include <mutex>

namespace trn {

namespace {

constexpr size_t kMaxN = TRN_NOALLOC_MAX_NODES;
constexpr size_t kMaxE = TRN_NOALLOC_MAX_ELEMS;
constexpr size_t kB = TRN_NOALLOC_BUCKET;
constexpr size_t kPartials = 256;  /* one per 256 elements; the sum behind them (grid form) */

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t) 255; }

/* carve-up of the scratch array (byte offsets, each 256-byte aligned) */
constexpr size_t oTri = 0;
constexpr size_t oPts = oTri + align256(sizeof(int4) * kMaxE);
constexpr size_t oTen = oPts + align256(sizeof(double2) * kMaxN);
constexpr size_t oStenc = oTen + align256(sizeof(double4) * kMaxN);
constexpr size_t oVic = oStenc + align256(sizeof(int) * kMaxN * kB);
constexpr size_t oDeg = oVic + align256(sizeof(int) * kMaxN * kB);
constexpr size_t oVdeg = oDeg + align256(sizeof(int) * kMaxN);
constexpr size_t oAlive = oVdeg + align256(sizeof(int) * kMaxN);
constexpr size_t oGrad = oAlive + align256(kMaxN);
constexpr size_t oTerms = oGrad + align256(sizeof(double2) * kMaxN);
constexpr size_t oRec = oTerms + align256(sizeof(double) * (kPartials + 1));
constexpr size_t oAtot = oRec + align256(sizeof(double4) * kMaxE);
constexpr size_t oRest = oAtot + align256(sizeof(double) * kMaxN);
constexpr size_t oErr = oRest + align256(sizeof(int) * kMaxN);   /* the error word, the length of the list at oRest */
constexpr size_t kScratchBytes = oErr + 256;

}  // namespace

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
unsigned char* g_scratch_addr[kMaxDevices] = {nullptr};

/* device address of the scratch array on the current device; looked up once */
int scratch_address(unsigned char** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return TRN_ERR_CUDA;
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      std::fprintf(stderr, "trn_metric_noalloc: cudaGetSymbolAddress failed: %s\n",
                   cudaGetErrorString(e));
      return TRN_ERR_CUDA;
    }
    g_scratch_addr[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_scratch_addr[dev];
  return TRN_OK;
}

/* the steps before the recovery, for one vertex or element; the calls of one
 * step before any of the next */
__device__ __forceinline__ void na_vertex(const DMesh& d, int v, const double* points) {
  d.pts[v] = make_double2(points[2 * v], points[2 * v + 1]);
  d.deg[v] = d.vdeg[v] = 0;
  d.alive[v] = 1;
}

__device__ __forceinline__ void na_elem(const DMesh& d, int i, int nb_nodes, const int* tris) {
  const int a = tris[3 * i], b = tris[3 * i + 1], c = tris[3 * i + 2];
  const bool ok = a >= 0 && a < nb_nodes && b >= 0 && b < nb_nodes && c >= 0 && c < nb_nodes;
  if (!ok) atomicExch(d.err, TRN_DERR_INVALID);   /* before an overfull vertex, whichever is met first */
  d.tri[i] = ok ? make_int4(a, b, c, 0) : make_int4(-1, -1, -1, 0);
  if (!ok) return;
  trn_stenc_append(d, a, i);
  trn_stenc_append(d, b, i);
  trn_stenc_append(d, c, i);
}

/* the sorted row, and the adjacency from it and the elements alone */
__device__ __forceinline__ void na_row(const DMesh& d, int v) {
  int buf[2 * TRN_NOALLOC_BUCKET];
  const TrnRow row = trn_row(d.stenc, d, v);
  const int n = trn_deg(d, v);
  if (n <= kRowChunk) {
    int r[kRowChunk];
#pragma unroll
    for (int k = 0; k < kRowChunk; ++k) r[k] = k < n ? row.p[k] : kNoId;
    patch_sort8(r);
#pragma unroll
    for (int k = 0; k < kRowChunk; ++k)
      if (k < n) row.p[k] = r[k];
  } else {
    for (int k = 0; k < n; ++k) buf[k] = row[k];
    trn_isort(buf, n);
    for (int k = 0; k < n; ++k) row[k] = buf[k];
  }
  build_one_vicin(d, v, buf);
}

__device__ __forceinline__ void na_out(const DMesh& d, int v, double fact, double eig_min, double eig_max, double* out) {
  const double4 r = normalize_tensor(d.ten[v], fact, eig_min, eig_max);
  out[3 * v] = r.x;
  out[3 * v + 1] = r.y;
  out[3 * v + 2] = r.z;
}

/* The whole recovery in one launch of one thread-block cluster: at most 16,384
 * vertices are two a thread, so each step is a few dependent gathers, and as
 * fifteen launches and four clears they cost five times that. The steps are
 * separated by the cluster barrier; the error word is read once a warp and
 * step, so lanes agree about it. The complexity is summed in the tree of
 * k_sum_terms / k_sum_final: a partial per 256 elements (as metric_run's grid
 * has for so few), then one tree over the partials, which every block
 * computes for itself. 441 vertices 105 -> 67 us a call, 16,129
 * vertices 187 (before the element records) -> 110. */
constexpr int kNaPart = TRN_THREADS;

/* vertices of long rows that the cluster's 256 warps take, one after the
 * other: with more of them the kernel stops and the call goes on with
 * metric_run's kernels over the whole chip (na_recover_grid). Every triangle
 * of a grid cut into three at its centre (no row fits the registers), us a
 * call, cluster / grid after the cluster's start: 1,241 vertices 197 / 201,
 * 2,761 332 / 204, 10,921 1,100 / 289, 15,697 1,566 / 336; adapted meshes, a
 * quarter of whose rows are long: 4,083 vertices 128 / 183, 8,186 159 / 198,
 * 10,923 197 / 211. */
constexpr int kNaRest = 2048;

__device__ __forceinline__ double na_tree(double* sm, double s, int t) {
  sm[t] = s;
  __syncthreads();
  for (int o = kNaPart / 2; o > 0; o >>= 1) {
    if (t < o) sm[t] += sm[t + o];
    __syncthreads();
  }
  const double r = sm[0];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kTailThreads) k_na_recover(DMesh d, int nb_nodes, int nb_elems,
                                                            const double* __restrict__ points,
                                                            const int* __restrict__ tris,
                                                            const double* __restrict__ solut, double2* grad,
                                                            MetricWs ws, double* partial, double target,
                                                            double scale_exp, double eig_min, double eig_max,
                                                            double* __restrict__ out) {
  __shared__ int s_buf[kTailThreads / 32][TRN_MAX_PATCH];
  __shared__ double s_tree[kTailThreads / kNaPart][kNaPart];
  const int tid = trn_tid(), stride = trn_grid_stride(), half = threadIdx.x / kNaPart, t = threadIdx.x % kNaPart;
  if (tid == 0) {
    *d.err = 0;
    *ws.rest_n = 0;
  }
  for (int v = tid; v < nb_nodes; v += stride) na_vertex(d, v, points);
  cluster_sync();
  for (int i = tid; i < nb_elems; i += stride) na_elem(d, i, nb_nodes, tris);
  cluster_sync();
  if (!tail_failed(d)) {
    for (int v = tid; v < nb_nodes; v += stride) na_row(d, v);
    for (int i = tid; i < nb_elems; i += stride) ws.rec[i] = elem_gradient(d, i, solut);
  }
  cluster_sync();
  const GradSum gsum{ws.rec, 0, grad, ws.atot};
  const HessSum hsum{ws.rec, 0, ws.atot, scale_exp, nullptr, nullptr};
  const bool go = !tail_failed(d);
  if (go)
    for (int v = tid; v < nb_nodes; v += stride)
      if (!patch_sum_regs<GradSum, 4>(d, v, gsum)) trn_append(ws.rest, ws.rest_n, v);
  cluster_sync();
  const int nr = *ws.rest_n;
  if (nr > kNaRest) return;   /* every thread: too many for the cluster's warps */
  for (int q = tid >> 5; q < nr; q += stride >> 5)
    patch_sum_warp(d, ws.rest[q], gsum, s_buf[threadIdx.x >> 5]);
  cluster_sync();
  if (go)
    for (int i = tid; i < nb_elems; i += stride) ws.rec[i] = elem_hessian(d, i, grad);
  cluster_sync();
  if (go)
    for (int v = tid; v < nb_nodes; v += stride) patch_sum_regs<HessSum, 4>(d, v, hsum);
  for (int q = tid >> 5; q < nr; q += stride >> 5)
    patch_sum_warp(d, ws.rest[q], hsum, s_buf[threadIdx.x >> 5]);
  cluster_sync();
  /* one partial per 256 elements by each half of a block, the same number of
   * steps for all of them */
  const int parts = (nb_elems + kNaPart - 1) / kNaPart, halves = stride / kNaPart;
  for (int b0 = 0; b0 < parts; b0 += halves) {
    const int b = b0 + tid / kNaPart, i = b * kNaPart + t;
    const double s = na_tree(s_tree[half], go && b < parts && i < nb_elems ? 0 + complexity_term(d, i) : 0.0, t);
    if (t == 0 && b < parts) partial[b] = s;
  }
  cluster_sync();
  const double complexity = na_tree(s_tree[half], t < parts ? 0 + partial[t] : 0.0, t);
  if (tail_failed(d)) return;
  const double fact = target / complexity;
  for (int v = tid; v < nb_nodes; v += stride) na_out(d, v, fact, eig_min, eig_max, out);
}

static_assert(kMaxE <= (size_t) kNaPart * kNaPart, "one tree over the partials");

/* the same steps as launches of their own, around metric_run's kernels */
__global__ void k_na_vertices(DMesh d, int nb_nodes, const double* __restrict__ points) {
  if (trn_tid() == 0) *d.err = 0;
  for (int v = trn_tid(); v < nb_nodes; v += trn_grid_stride()) na_vertex(d, v, points);
}

__global__ void k_na_elems(DMesh d, int nb_nodes, int nb_elems, const int* __restrict__ tris) {
  for (int i = trn_tid(); i < nb_elems; i += trn_grid_stride()) na_elem(d, i, nb_nodes, tris);
}

__global__ void k_na_rows(DMesh d, int nb_nodes) {
  if (trn_failed(d)) return;
  for (int v = trn_tid(); v < nb_nodes; v += trn_grid_stride()) na_row(d, v);
}

__global__ void k_na_tensors(DMesh d, int nb_nodes, const double* complexity, double target, double eig_min,
                             double eig_max, double* __restrict__ out) {
  if (trn_failed(d)) return;
  const double fact = target / *complexity;
  for (int v = trn_tid(); v < nb_nodes; v += trn_grid_stride()) na_out(d, v, fact, eig_min, eig_max, out);
}

void na_recover_grid(const DMesh& d, int nb_nodes, int nb_elems, const double* points, const int* tris,
                     const double* solut, double2* grad, const MetricWs& ws, double* partial, double target,
                     double scale_exp, double eig_min, double eig_max, double* out, cudaStream_t s) {
  const int gv = grid_for(nb_nodes), ge = grid_for(nb_elems);
  double* complexity = partial + kPartials;
  k_na_vertices<<<gv, TRN_THREADS, 0, s>>>(d, nb_nodes, points);
  note_launch();
  k_na_elems<<<ge, TRN_THREADS, 0, s>>>(d, nb_nodes, nb_elems, tris);
  note_launch();
  k_na_rows<<<gv, TRN_THREADS, 0, s>>>(d, nb_nodes);
  note_launch();
  metric_patches(d, nb_nodes, nb_elems, solut, grad, ws, scale_exp, s);
  metric_complexity(d, nb_elems, nullptr, partial, complexity, false, s);
  k_na_tensors<<<gv, TRN_THREADS, 0, s>>>(d, nb_nodes, complexity, target, eig_min, eig_max, out);
  note_launch();
}

}  // namespace
}  // namespace trn

extern "C" int trn_metric_noalloc(int nb_nodes, int nb_elems, const double* d_points,
                                  const int* d_tris, const double* d_solut, double target_factor,
                                  int lp_norm, double h_min, double h_max, double* d_tensor,
                                  void* stream) {
  using namespace trn;
  if (nb_nodes <= 0 || nb_elems <= 0 || !d_points || !d_tris || !d_solut || !d_tensor ||
      lp_norm < 0 || h_min <= 0 || h_max <= 0)
    return TRN_ERR_INVALID;
  if ((size_t) nb_nodes > kMaxN || (size_t) nb_elems > kMaxE) {
    std::fprintf(stderr,
                 "trn_metric_noalloc: %d vertices / %d triangles exceed the fixed scratch "
                 "(at most %d vertices and %d triangles)\n",
                 nb_nodes, nb_elems, TRN_NOALLOC_MAX_NODES, TRN_NOALLOC_MAX_ELEMS);
    return TRN_ERR_CAPACITY;
  }
  unsigned char* base = nullptr;
  int rc = scratch_address(&base);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  DMesh d{};
  d.tri = reinterpret_cast<int4*>(base + oTri);
  d.pts = reinterpret_cast<double2*>(base + oPts);
  d.ten = reinterpret_cast<double4*>(base + oTen);
  d.stenc = reinterpret_cast<int*>(base + oStenc);
  d.vic = reinterpret_cast<int*>(base + oVic);
  d.deg = reinterpret_cast<int*>(base + oDeg);
  d.vdeg = reinterpret_cast<int*>(base + oVdeg);
  d.alive = base + oAlive;
  d.err = reinterpret_cast<int*>(base + oErr);
  d.bucket = (int) kB;
  d.capa_node = nb_nodes;
  d.capa_elem = nb_elems;
  double2* grad = reinterpret_cast<double2*>(base + oGrad);
  double* terms = reinterpret_cast<double*>(base + oTerms);

  const double target = (double) (int) std::floor(nb_nodes * target_factor);
  const double scale_exp = lp_norm ? -1. / (2 * lp_norm + 2) : 0.5;
  const double eig_min = 1 / trn_pow(h_min, 2);
  const double eig_max = 1 / trn_pow(h_max, 2);
  int* rest = reinterpret_cast<int*>(base + oRest);
  const MetricWs ws{reinterpret_cast<double4*>(base + oRec), reinterpret_cast<double*>(base + oAtot), rest, d.err + 1};
  int word[2] = {0, 0};   /* the error word, the vertices that the cluster's warps had to take */
  const int& err = word[0];
  auto read_back = [&](size_t n) {
    return cudaMemcpyAsync(word, d.err, n, cudaMemcpyDeviceToHost, s) == cudaSuccess &&
           cudaStreamSynchronize(s) == cudaSuccess;
  };
  const bool cluster = cluster_launch<k_na_recover>(s, d, nb_nodes, nb_elems, d_points, d_tris, d_solut, grad, ws,
                                                    terms, target, scale_exp, eig_min, eig_max, d_tensor);
  if (cluster && !read_back(sizeof(word))) return TRN_ERR_CUDA;
  /* no cluster fits this device (a part of one), or too much for the cluster */
  if (!cluster || (!err && word[1] > kNaRest)) {
    na_recover_grid(d, nb_nodes, nb_elems, d_points, d_tris, d_solut, grad, ws, terms, target, scale_exp, eig_min,
                    eig_max, d_tensor, s);
    if (cudaPeekAtLastError() != cudaSuccess || !read_back(sizeof(int))) return TRN_ERR_CUDA;
  }
  if (err == TRN_DERR_CAPACITY || err == TRN_DERR_BUCKET) {
    std::fprintf(stderr, "trn_metric_noalloc: a vertex has more than %d incident triangles\n",
                 TRN_NOALLOC_BUCKET);
    return TRN_ERR_CAPACITY;
  }
  if (err) return TRN_ERR_INVALID;
  return TRN_OK;
}
