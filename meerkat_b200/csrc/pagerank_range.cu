// PageRank of one vertex range of an out-edge graph (a member of a graph
// set), by push sweeps: no reverse graph needed.
//
// Same formula as the pull solver (reference: PageRankImpl.cuh:41-52,
// :89-144, PageRank.cuh:42-43) restricted to the range [lo, hi), N = hi - lo:
//   PR'[v] = (1-d)/N + d * sum_{u -> v} PR[u] / outdeg[u]
//                    + d * sum_{outdeg[u] = 0} PR[u] / N
// starting from PR = 1/N, stopping once delta * d / (1 - d) <= tol / 2 (the
// L1 error bound of the contraction) or after max_iter iterations.  The
// range must be closed under out-edges.  Out-degrees are the graph's live
// degrees, so a graph updated between calls needs no recount.
//
// A run first turns the range's live edges around: a counting sort by target
// (count, scan, fill over the slabs) leaves the (source, target) pairs grouped
// by target.  An iteration is then two launches:
//   gather  a warp takes kPrrChunk consecutive pairs and sums d PR[u] / outdeg[u]
//           over each target's run with segmented warp scans, so a target gets
//           one FP64 atomic per run piece instead of one per edge, and a hub's
//           run spreads over many warps;
//   step    PR' per vertex, its next contribution, |delta| and the dangling
//           mass of the next iteration.
// What bounds it: the pairs stream from L2 (8 bytes an edge) and the gathers
// of the contributions (8 bytes each, mostly L2).  Pushing straight from the
// slabs (k_prr_push) walks every 128-byte line and issues an atomic per edge
// in every iteration: about 130 us an iteration at 262,144 vertices and 4.1 M
// weighted edges, five launches and a host round trip each.  It stays for runs
// of few iterations and for when the pairs do not fit in memory.
// The device decides when to stop: iterations are issued kPrrBatch at a time,
// a launch behind the converged one returns at once, and the host reads the
// deltas once per batch.  FP64 accumulation keeps the result within the same
// L1 tolerance as the pull solver although the order of the sums varies from
// run to run.
#include <cuda_runtime.h>

#include <algorithm>

#include "mk_internal.h"
#include "mk_rows.h"
#include "mk_slab.cuh"

namespace mk {
namespace {

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
  return x;
}

// Block-reduced sum of per-thread values into *out.
__device__ __forceinline__ void block_add(double x, double *out) {
  __shared__ double part[32];
  x = warp_sum(x);
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  if (lane == 0) part[w] = x;
  __syncthreads();
  if (w == 0) {
    double y = lane < (blockDim.x >> 5) ? part[lane] : 0.0;
    y = warp_sum(y);
    if (lane == 0 && y != 0.0) atomicAdd(out, y);
  }
  __syncthreads();
}

__global__ void k_prr_fill(double *__restrict__ pr, uint32_t n, double x) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    pr[i] = x;
}

// acc[0] += dangling mass of pr
__global__ void k_prr_dangling(const double *__restrict__ pr, const uint32_t *__restrict__ deg,
                               uint32_t n, double *acc) {
  double x = 0.0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (deg[i] == 0) x += pr[i];
  block_add(x, acc);
}

__global__ void k_prr_base(double *__restrict__ nx, uint32_t n, const double *acc, double d) {
  const double base = (1.0 - d) / n + d * acc[0] / n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    nx[i] = base;
}

// One iteration straight from the slabs: an atomic per live edge.  A key
// outside the range is skipped and reported, as k_prr_turn does.
template <bool kW>
__global__ void k_prr_push(GraphView g, uint32_t lo, uint32_t n, uint32_t b0, uint32_t nb,
                           const double *__restrict__ pr, double *nx, double d) {
  const Lanes L = lanes();
  const uint32_t group = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const uint32_t ngroups = (gridDim.x * blockDim.x) >> 3;
  for (uint32_t i = group; i < nb; i += ngroups) {
    const uint32_t b = b0 + i;
    const uint32_t u = g.bowner[b];
    const uint32_t du = g.deg[u];
    if (du == 0) continue;
    const double c = d * pr[u - lo] / (double)du;
    walk_bucket(g, L, b, [&](const uint4 &q) {
      uint32_t k[4], w[4];
      lane_keys<kW>(q, L.gl, k, w);
#pragma unroll
      for (int j = 0; j < keys_per_lane<kW>(); ++j) {
        if (k[j] >= kTombKey) continue;
        const uint32_t v = k[j] - lo;
        if (v < n)  // (a key below lo wraps above n)
          atomicAdd(nx + v, c);
        else
          atomicOr(g.err, kErrInvalidId);
      }
    });
  }
}

// Iterations up to which a run pushes: turning the edges around costs what two
// to three pushes do.  Pushed / turned, microseconds: 4.1 M edges 142 / 354 at
// one iteration, 399 / 425 at three, 530 / 459 at four; 1 M edges (weighted)
// 79 / 191, 216 / 213, 282 / 230; 20,000 edges 41 / 84, 109 / 108, 134 / 120.
constexpr uint32_t kPrrPushIters = 3;
constexpr uint32_t kPrrChunk = 512;  // pairs per warp of the gather
constexpr uint32_t kPrrBatch = 12;   // iterations issued between two reads of the deltas
constexpr uint32_t kPrrSteps = 4;    // 32-pair steps whose loads are in flight together

// Live edges per target of the range (fill false), or the pairs written at
// their targets' positions, the counts used up as cursors (fill true).  A key
// outside the range (a range that is not closed under edges) is skipped and
// reported as MK_DEVERR_INVALID_ID.  An edge that was not counted (the member
// changed under the call) is left out (row_place).
template <bool kW, bool kFill>
__global__ void k_prr_turn(GraphView g, uint32_t lo, uint32_t n, uint32_t b0, uint32_t nb,
                           uint32_t *__restrict__ cnt, const unsigned long long *__restrict__ rp,
                           uint2 *__restrict__ pairs) {
  const Lanes L = lanes();
  const uint32_t group = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const uint32_t ngroups = (gridDim.x * blockDim.x) >> 3;
  for (uint64_t i0 = (uint64_t)group * 4; i0 < nb; i0 += (uint64_t)ngroups * 4) {
    const uint32_t b = b0 + (uint32_t)i0, m = nb - i0 < 4 ? (uint32_t)(nb - i0) : 4u;
    const uint32_t own = kFill && L.gl < m ? __ldg(g.bowner + b + L.gl) - lo : 0u;
    uint32_t src[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) src[j] = kFill ? __shfl_sync(L.gmask, own, L.gbase + j) : 0u;
    walk4_levels(g, L, b, m, [&](uint32_t j, const uint4 q) {
      const uint32_t u = j == 0 ? src[0] : j == 1 ? src[1] : j == 2 ? src[2] : src[3];
      uint32_t k[4], w[4], at[4];
      lane_keys<kW>(q, L.gl, k, w);
#pragma unroll
      for (int t = 0; t < keys_per_lane<kW>(); ++t) {
        const uint32_t v = k[t] - lo;
        if (k[t] >= kTombKey) {
          k[t] = kEmptyKey;
        } else if (k[t] < lo || v >= n) {
          k[t] = kEmptyKey;
          if (!kFill) atomicOr(g.err, kErrInvalidId);
        } else if (!kFill) {
          atomicAdd(cnt + v, 1u);
        } else {
          at[t] = row_place(atomicSub(cnt + v, 1u), rp[v + 1] - rp[v]);
          if (at[t] == kNoPlace) k[t] = kEmptyKey;
        }
      }
      if (!kFill) return;
#pragma unroll
      for (int t = 0; t < keys_per_lane<kW>(); ++t)
        if (k[t] != kEmptyKey) pairs[rp[k[t] - lo] + at[t]] = make_uint2(u, k[t] - lo);
    });
  }
}

// *most = the largest number of live edges of any window of w vertices (rp:
// the running sum of the degrees).
__global__ void k_prr_window(const unsigned long long *__restrict__ rp, uint32_t V, uint32_t w,
                             unsigned long long *most) {
  unsigned long long m = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= V - w; i += gridDim.x * blockDim.x)
    m = max(m, rp[i + w] - rp[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if ((threadIdx.x & 31u) == 0 && m) atomicMax(most, m);
}

// PR = x, the first contributions, empty sums, the first dangling mass; and
// the places that the fill left open (edges that went between the count and
// the fill) get no target, so the gather never follows an old word.
__global__ void k_prr_start(double *__restrict__ pr, double *__restrict__ c, double *__restrict__ sum,
                            const uint32_t *__restrict__ deg, uint32_t n, double x, double d,
                            double *dang, const uint32_t *__restrict__ cnt,
                            const unsigned long long *__restrict__ rp, uint2 *__restrict__ pairs) {
  double lost = 0.0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t dg = deg[i];
    pr[i] = x;
    sum[i] = 0.0;
    c[i] = dg ? d * x / (double)dg : 0.0;
    if (!dg) lost += x;
    const uint32_t left = cnt[i];
    if (left) {
      const unsigned long long r0 = rp[i], gap = row_gap(left, rp[i + 1] - r0);
      for (unsigned long long j = 0; j < gap; ++j) pairs[r0 + j] = make_uint2(0u, kEmptyKey);
    }
  }
  block_add(lost, dang);
}

// Whether the iteration before this one (its |delta| in *before; null: none)
// ended the solve.  An iteration that did not run leaves its delta at zero,
// so every later one sees it as ended too.
__device__ __forceinline__ bool prr_done(const double *before, double d, double stop) {
  return before && *before * d / (1.0 - d) <= stop;
}

__global__ void __launch_bounds__(256)
    k_prr_gather(const uint2 *__restrict__ pairs, unsigned long long E, const double *__restrict__ c,
                 double *sum, const double *before, double d, double stop) {
  if (prr_done(before, d, stop)) return;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t e0 = warp * kPrrChunk; e0 < E; e0 += nwarps * kPrrChunk) {
    const uint32_t len = E - e0 < kPrrChunk ? (uint32_t)(E - e0) : kPrrChunk;
    const uint2 *__restrict__ chunk = pairs + e0;
    uint32_t ckey = kEmptyKey;  // target whose run is open, and its sum so far
    double cval = 0.0;
    for (uint32_t s0 = 0; s0 < len; s0 += 32u * kPrrSteps) {
      uint2 p[kPrrSteps];
      double val[kPrrSteps];
#pragma unroll
      for (uint32_t r = 0; r < kPrrSteps; ++r) {
        const uint32_t e = s0 + 32u * r + lane;
        p[r] = e < len ? __ldg(chunk + e) : make_uint2(0u, kEmptyKey);
      }
#pragma unroll
      for (uint32_t r = 0; r < kPrrSteps; ++r) val[r] = p[r].y != kEmptyKey ? __ldg(c + p[r].x) : 0.0;
#pragma unroll
      for (uint32_t r = 0; r < kPrrSteps; ++r) {
        if (s0 + 32u * r >= len) break;
        const uint32_t key = p[r].y;  // kEmptyKey: no edge here, val 0
        double v = val[r];
        if (lane == 0) {
          if (key == ckey)
            v += cval;
          else if (ckey != kEmptyKey)
            atomicAdd(sum + ckey, cval);
        }
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
          const double y = __shfl_up_sync(0xFFFFFFFFu, v, o);
          const uint32_t ky = __shfl_up_sync(0xFFFFFFFFu, key, o);
          if (lane >= o && ky == key) v += y;
        }
        const uint32_t next = __shfl_down_sync(0xFFFFFFFFu, key, 1);
        if (lane < 31 && key != next && key != kEmptyKey) atomicAdd(sum + key, v);
        ckey = __shfl_sync(0xFFFFFFFFu, key, 31);  // kEmptyKey when the chunk ended in this step
        cval = __shfl_sync(0xFFFFFFFFu, v, 31);
      }
    }
    if (lane == 0 && ckey != kEmptyKey) atomicAdd(sum + ckey, cval);
  }
}

// PR' from the gathered sums (emptied again), the next contributions;
// *delta += |PR' - PR|, dang[1] += the dangling mass of PR'.
__global__ void __launch_bounds__(256)
    k_prr_step(double *__restrict__ pr, double *__restrict__ c, double *__restrict__ sum,
               const uint32_t *__restrict__ deg, uint32_t n, double *dang, double *delta,
               const double *before, double d, double stop) {
  if (prr_done(before, d, stop)) return;
  const double base = (1.0 - d) / n + d * dang[0] / n;
  double moved = 0.0, lost = 0.0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double nv = base + sum[i];
    const uint32_t dg = deg[i];
    moved += fabs(nv - pr[i]);
    pr[i] = nv;
    sum[i] = 0.0;
    c[i] = dg ? d * nv / (double)dg : 0.0;
    if (!dg) lost += nv;
  }
  block_add(moved, delta);
  block_add(lost, dang + 1);
}

// acc[1] += sum |nx - pr|
__global__ void k_prr_delta(const double *__restrict__ pr, const double *__restrict__ nx,
                            uint32_t n, double *acc) {
  double x = 0.0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x += fabs(nx[i] - pr[i]);
  block_add(x, acc + 1);
}

__global__ void k_prr_out(const double *__restrict__ pr, uint32_t n, float *__restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = (float)pr[i];
}

int flat_blocks(uint64_t n, int device) {
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(n / 256 + 1, (uint64_t)device_sm_count(device) * 8));
}

}  // namespace
}  // namespace mk

using namespace mk;

struct mk_pagerank_range {
  mk_graph *g = nullptr;
  uint32_t cap = 0;  // vertices
  double *a = nullptr, *b = nullptr;
  // push form: [0] dangling, [1] delta; else the dangling mass before every
  // iteration of a batch and after it, then the iterations' deltas
  double *acc = nullptr;
  DevBuf<uint2> pairs;  // (source, target) of every live edge, by target
  bool fixed = false;   // the pairs do not grow (mk_pagerank_range_reserve)
  DevBuf<double> c;     // contributions d PR / outdeg
  DevBuf<uint32_t> cnt;
  DevBuf<unsigned long long> rp, tmp;
  float *out = nullptr;
  uint32_t n = 0;  // vertices of the last run
  uint32_t iters = 0;
  float delta = 0.f;
  Timer timer;
};

// Sizes what a run needs for the graph as it is, so that no run allocates
// inside its timed window unless the member grows (262,144 vertices, 4.1 M
// edges: a handle's first run 2.29 ms when it allocated, 1.25 now, later ones
// 1.22).  Whatever does not fit here is tried again by the runs.
static mk_status prr_presize(mk_pagerank_range *p) {
  mk_graph *g = p->g;
  const uint32_t w = std::min(p->cap, g->V);
  MK_CHECK(p->cnt.reserve(w));
  MK_CHECK(p->rp.reserve((size_t)w + 1));
  MK_CHECK(p->c.reserve(w));
  struct Rows {
    unsigned long long *ptr = nullptr;
    ~Rows() { cudaFree(ptr); }
  } rows;
  MK_CUDA(cudaMalloc(&rows.ptr, ((size_t)g->V + 1) * 8));
  MK_CHECK(scan_u32_to_u64(g->deg, rows.ptr, g->V, p->tmp, nullptr));
  unsigned long long most = 0, *d_most = reinterpret_cast<unsigned long long *>(p->acc);
  MK_CUDA(cudaMemset(d_most, 0, 8));
  k_prr_window<<<flat_blocks(g->V - w + 1, g->device), 256>>>(rows.ptr, g->V, w, d_most);
  MK_CUDA(cudaMemcpy(&most, d_most, 8, cudaMemcpyDeviceToHost));
  return most ? p->pairs.reserve(most) : MK_OK;
}

extern "C" {

mk_status mk_pagerank_range_create(mk_graph *g, uint32_t max_vertices, mk_pagerank_range **out) {
  if (!g || !out || max_vertices == 0)
    return fail(MK_ERR_INVALID, "mk_pagerank_range_create: bad argument");
  if (g->reverse) return fail(MK_ERR_INVALID, "mk_pagerank_range_create: needs an out-edge graph");
  *out = nullptr;
  DeviceGuard dg(g->device);
  mk_pagerank_range *p = new mk_pagerank_range();
  p->g = g;
  p->cap = max_vertices;
  cudaError_t e = cudaMalloc(&p->a, (size_t)max_vertices * 8);
  if (e == cudaSuccess) e = cudaMalloc(&p->b, (size_t)max_vertices * 8);
  if (e == cudaSuccess) e = cudaMalloc(&p->acc, (2 * kPrrBatch + 1) * 8);
  if (e == cudaSuccess) e = cudaMalloc(&p->out, (size_t)max_vertices * 4);
  if (e != cudaSuccess) {
    mk_pagerank_range_destroy(p);
    return cuda_fail(e, "mk_pagerank_range_create");
  }
  if (prr_presize(p) != MK_OK) (void)cudaGetLastError();
  *out = p;
  return MK_OK;
}

}  // extern "C"

// Turns the range's edges around (p->pairs); *edges their number.  MK_ERR_OOM
// when they do not fit, on the device or in the scratch that the caller fixed.
static mk_status prr_turn(mk_pagerank_range *p, uint32_t lo, uint32_t n, uint32_t b0, uint32_t nb,
                          cudaStream_t s, unsigned long long *edges) {
  mk_graph *g = p->g;
  MK_CHECK(p->cnt.reserve(n));
  MK_CHECK(p->rp.reserve((size_t)n + 1));
  MK_CHECK(p->c.reserve(n));
  const GraphView v = g->view();
  const int gb = (int)std::min<uint64_t>((uint64_t)nb * 2 / 256 + 1, (uint64_t)device_sm_count(g->device) * 8);
  MK_CUDA(cudaMemsetAsync(p->cnt.ptr, 0, (size_t)n * 4, s));
  if (g->weighted)
    k_prr_turn<true, false><<<gb, 256, 0, s>>>(v, lo, n, b0, nb, p->cnt.ptr, nullptr, nullptr);
  else
    k_prr_turn<false, false><<<gb, 256, 0, s>>>(v, lo, n, b0, nb, p->cnt.ptr, nullptr, nullptr);
  MK_CHECK(scan_u32_to_u64(p->cnt.ptr, p->rp.ptr, n, p->tmp, s));
  MK_CUDA(cudaMemcpyAsync(edges, p->rp.ptr + n, 8, cudaMemcpyDeviceToHost, s));
  MK_CUDA(cudaStreamSynchronize(s));
  if (p->fixed && *edges > p->pairs.cap) return MK_ERR_OOM;
  MK_CHECK(p->pairs.reserve(std::max<unsigned long long>(*edges, 1)));
  if (g->weighted)
    k_prr_turn<true, true><<<gb, 256, 0, s>>>(v, lo, n, b0, nb, p->cnt.ptr, p->rp.ptr, p->pairs.ptr);
  else
    k_prr_turn<false, true><<<gb, 256, 0, s>>>(v, lo, n, b0, nb, p->cnt.ptr, p->rp.ptr, p->pairs.ptr);
  MK_CUDA(cudaGetLastError());
  return MK_OK;
}

// The iterations over the turned edges; the ranks end in p->a.
static mk_status prr_gather_solve(mk_pagerank_range *p, uint32_t lo, uint32_t n, unsigned long long E,
                                  double d, double stop, uint32_t max_iter, cudaStream_t s,
                                  uint32_t *iters, double *last) {
  mk_graph *g = p->g;
  const uint32_t *deg = g->deg + lo;
  const int fb = flat_blocks(n, g->device);
  const uint64_t chunks = (E + kPrrChunk - 1) / kPrrChunk;
  const int eb = (int)std::max<uint64_t>(
      1, std::min<uint64_t>((chunks + 7) / 8, (uint64_t)device_sm_count(g->device) * 8));
  double *dang = p->acc, *delta = p->acc + kPrrBatch + 1;
  MK_CUDA(cudaMemsetAsync(p->acc, 0, (2 * kPrrBatch + 1) * 8, s));
  k_prr_start<<<fb, 256, 0, s>>>(p->a, p->c.ptr, p->b, deg, n, 1.0 / n, d, dang, p->cnt.ptr, p->rp.ptr,
                                 p->pairs.ptr);
  MK_CUDA(cudaGetLastError());
  uint32_t it = 0;
  double h[kPrrBatch];
  while (it < max_iter) {
    const uint32_t k = std::min(kPrrBatch, max_iter - it);
    for (uint32_t i = 0; i < k; ++i) {
      const double *before = i ? delta + i - 1 : nullptr;
      k_prr_gather<<<eb, 256, 0, s>>>(p->pairs.ptr, E, p->c.ptr, p->b, before, d, stop);
      k_prr_step<<<fb, 256, 0, s>>>(p->a, p->c.ptr, p->b, deg, n, dang + i, delta + i, before, d, stop);
    }
    MK_CUDA(cudaGetLastError());
    MK_CUDA(cudaMemcpyAsync(h, delta, sizeof(double) * k, cudaMemcpyDeviceToHost, s));
    MK_CUDA(cudaStreamSynchronize(s));
    for (uint32_t i = 0; i < k; ++i) {
      ++it;
      *last = h[i];
      if (h[i] * d / (1.0 - d) <= stop) {
        *iters = it;
        return MK_OK;
      }
    }
    if (it < max_iter) {  // the next batch starts from the dangling mass this one left
      MK_CUDA(cudaMemcpyAsync(dang, dang + kPrrBatch, 8, cudaMemcpyDeviceToDevice, s));
      MK_CUDA(cudaMemsetAsync(dang + 1, 0, 2 * kPrrBatch * 8, s));
    }
  }
  *iters = it;
  return MK_OK;
}

extern "C" {

mk_status mk_pagerank_range_reserve(mk_pagerank_range *p, uint64_t max_edges) {
  if (!p) return fail(MK_ERR_INVALID, "mk_pagerank_range_reserve: null handle");
  DeviceGuard dg(p->g->device);
  p->fixed = max_edges != 0;
  if (!p->fixed) return MK_OK;
  MK_CUDA(cudaDeviceSynchronize());  // queued runs may still read the old scratch
  p->pairs.release();
  return p->pairs.reserve(max_edges);
}

mk_status mk_pagerank_range_run(mk_pagerank_range *p, uint32_t v_begin, uint32_t v_end,
                                float damping, float tol, uint32_t max_iter, void *stream,
                                float *ms_out) {
  if (!p) return fail(MK_ERR_INVALID, "mk_pagerank_range_run: null handle");
  mk_graph *g = p->g;
  if (v_begin >= v_end || v_end > g->V)
    return fail(MK_ERR_INVALID, "mk_pagerank_range_run: bad vertex range");
  if (v_end - v_begin > p->cap)
    return fail(MK_ERR_INVALID, "mk_pagerank_range_run: range larger than max_vertices");
  if (!(damping > 0.f && damping < 1.f) || !(tol > 0.f))
    return fail(MK_ERR_INVALID, "mk_pagerank_range_run: damping must be in (0,1), tol > 0");
  DeviceGuard dg(g->device);
  cudaStream_t s = as_stream(stream);
  MK_CHECK(p->timer.start(s, ms_out != nullptr));
  const uint32_t n = v_end - v_begin;
  const uint32_t b0 = g->h_boff[v_begin], nb = g->h_boff[v_end] - b0;
  const double d = damping;
  const int fb = flat_blocks(n, g->device);
  const int gb = (int)std::min<uint64_t>((uint64_t)nb * 8 / 256 + 1, (uint64_t)device_sm_count(g->device) * 8);
  const GraphView v = g->view();
  double *pr = p->a, *nx = p->b;
  uint32_t it = 0;
  double delta = 0.0;
  unsigned long long E = 0;
  bool push = max_iter <= kPrrPushIters;
  if (!push) {
    const mk_status turned = prr_turn(p, v_begin, n, b0, nb, s, &E);
    push = turned == MK_ERR_OOM;  // the pairs do not fit beside what the process holds
    if (push)
      (void)cudaGetLastError();
    else
      MK_CHECK(turned);
  }
  if (!push) {
    MK_CHECK(prr_gather_solve(p, v_begin, n, E, d, 0.5 * tol, max_iter, s, &it, &delta));
  } else {
    k_prr_fill<<<fb, 256, 0, s>>>(pr, n, 1.0 / n);
    while (it < max_iter) {
      MK_CUDA(cudaMemsetAsync(p->acc, 0, 16, s));
      k_prr_dangling<<<fb, 256, 0, s>>>(pr, g->deg + v_begin, n, p->acc);
      k_prr_base<<<fb, 256, 0, s>>>(nx, n, p->acc, d);
      if (g->weighted)
        k_prr_push<true><<<gb, 256, 0, s>>>(v, v_begin, n, b0, nb, pr, nx, d);
      else
        k_prr_push<false><<<gb, 256, 0, s>>>(v, v_begin, n, b0, nb, pr, nx, d);
      k_prr_delta<<<fb, 256, 0, s>>>(pr, nx, n, p->acc);
      MK_CUDA(cudaGetLastError());
      MK_CUDA(cudaMemcpyAsync(&delta, p->acc + 1, 8, cudaMemcpyDeviceToHost, s));
      MK_CUDA(cudaStreamSynchronize(s));
      std::swap(pr, nx);
      ++it;
      if (delta * d / (1.0 - d) <= 0.5 * tol) break;
    }
  }
  k_prr_out<<<fb, 256, 0, s>>>(pr, n, p->out);
  MK_CUDA(cudaGetLastError());
  p->n = n;
  p->iters = it;
  p->delta = (float)delta;
  return p->timer.stop(ms_out);
}

mk_status mk_pagerank_range_values(mk_pagerank_range *p, float *h_out) {
  if (!p || !h_out) return fail(MK_ERR_INVALID, "mk_pagerank_range_values: null argument");
  DeviceGuard dg(p->g->device);
  MK_CUDA(cudaDeviceSynchronize());
  MK_CUDA(cudaMemcpy(h_out, p->out, (size_t)p->n * 4, cudaMemcpyDeviceToHost));
  return MK_OK;
}

mk_status mk_pagerank_range_stats(mk_pagerank_range *p, uint32_t *h_iters, float *h_delta) {
  if (!p) return fail(MK_ERR_INVALID, "mk_pagerank_range_stats: null handle");
  if (h_iters) *h_iters = p->iters;
  if (h_delta) *h_delta = p->delta;
  return MK_OK;
}

mk_status mk_pagerank_range_destroy(mk_pagerank_range *p) {
  if (!p) return MK_OK;
  DeviceGuard dg(p->g->device);
  cudaFree(p->a);
  cudaFree(p->b);
  cudaFree(p->acc);
  cudaFree(p->out);
  p->pairs.release();
  p->c.release();
  p->cnt.release();
  p->rp.release();
  p->tmp.release();
  delete p;
  return MK_OK;
}

}  // extern "C"
