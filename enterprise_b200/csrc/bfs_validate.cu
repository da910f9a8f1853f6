// Graph500-style validation of a traversal's result on the GPU.
//
// The reference checks one random vertex per source on the host (validate(),
// validate.h:34-103: its depth is one more than some neighbour's and no
// neighbour is two levels shallower). This file checks every vertex and edge
// with two certificates, rule for rule the ones the CPU oracle states:
//  * depth certificate (codes as oracle_check_depths):
//      -1 depth[src] != 0;  for each vertex v in ascending order:
//      -2 depth[v] < -1;  -3 depth[v] == 0 and v != src;  then its row in CSR
//      order, at the first edge (v, u) that breaks a rule: -4 exactly one of
//      v, u reached, -5 both reached with depths more than one apart; then
//      -6 a reached v > 0 deep with no neighbour one level up;
//  * parent certificate (codes as oracle_check_parents):
//      -1 parent[src] != src or depth[src] != 0; for each v != src in
//      ascending order: -2 unreached v with a parent, -3 parent out of range,
//      -4 depth[parent] != depth[v] - 1, -5 (parent, v) is not an edge.
// Every vertex's first broken rule is computed independently; the smallest
// such vertex wins (atomicMin on vertex << 8 | rule), so the answer is the
// oracle's (rule, vertex) exactly, whatever the launch order.
//
// Nearly every call finds nothing wrong, and that takes less: k_val_rows looks
// for any broken depth rule, over the rows in traversal order, where
// neighbouring rows have equal lengths and a lane takes one. Only when it
// finds one does k_val_depth go through the caller's rows for the answer.
#include <cub/cub.cuh>

#include "dev_common.cuh"
#include "dev_graph.h"

namespace ent {
namespace {

constexpr int VT = 256;

__device__ __forceinline__ void report(unsigned long long* slot, int64_t v, int code) {
  atomicMin(slot, ((unsigned long long)v << 8) | (unsigned)(-code));
}

// One warp per vertex; lanes walk the row 32 edges at a time in CSR order.
__global__ void __launch_bounds__(VT) k_val_depth(const int64_t* __restrict__ off, const int32_t* __restrict__ adj,
                                                  int64_t V, int32_t src, const int32_t* __restrict__ depth,
                                                  unsigned long long* slot) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)VT + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * VT) >> 5;
  for (int64_t v = gw; v < V; v += nw) {
    const int dv = depth[v];
    int code = 0;
    if (dv < -1) code = -2;
    else if (dv == 0 && v != src) code = -3;
    if (!code) {
      const int64_t b = off[v], e = off[v + 1];
      bool has_parent = false;
      for (int64_t k0 = b; k0 < e && !code; k0 += 32) {
        const int64_t k = k0 + lane;
        int c = 0;
        if (k < e) {
          const int du = depth[adj[k]];
          if ((du == -1) != (dv == -1)) c = -4;
          else if (dv != -1 && (du > dv + 1 || du < dv - 1)) c = -5;
          if (dv > 0 && du == dv - 1) has_parent = true;
        }
        const unsigned bad = __ballot_sync(FULL, c != 0);
        if (bad) code = __shfl_sync(FULL, c, __ffs(bad) - 1);  // the first broken edge in row order
      }
      has_parent = __any_sync(FULL, has_parent);
      if (!code && dv > 0 && !has_parent) code = -6;
    }
    if (code && lane == 0) report(slot, v, code);
  }
}

// Whether a vertex of depth dv breaks a depth rule with the smallest and largest
// depth among its neighbours, all compared unsigned (unreached is the largest).
// Depths below -1, and depth 0 off the source, are found vertex by vertex.
__device__ __forceinline__ bool row_breaks(unsigned dv, unsigned mn, unsigned mx) {
  if (dv == ~0u) return mn != ~0u;
  return mx > dv + 1 || (dv > 0 && mn != dv - 1);
}

constexpr int VAL_CTA = 2048;  // degree from which a CTA takes a row
constexpr int VAL_WARP = 32;   // ... and a warp, down to a lane per row
constexpr int VAL_ILP = 4;     // neighbours a lane has in flight together

// First traversal id whose degree is below d (degrees descend): 32 probes a step.
__device__ __forceinline__ int64_t first_below(const int32_t* deg, int64_t n, int d) {
  int64_t lo = 0, hi = n;
  const int lane = threadIdx.x & 31;
  while (lo < hi) {
    const int64_t step = (hi - lo + 31) / 32, at = lo + step * lane;
    const unsigned ge = __ballot_sync(FULL, at < hi && deg[at] >= d);
    if (!ge) return lo;
    const int last = 31 - __clz(ge);
    hi = min(hi, lo + step * (last + 1));
    lo = lo + step * last + 1;
  }
  return lo;
}

// Sets *broken if any row breaks a depth rule. dt: depths by traversal id.
// Bound by the scattered depth reads, a line each where neighbours share none
// (ER 2^22 d16: 67M of them), and by its longest rows where hubs are: a warp
// per row took 0.66 ms there and 16.6 ms on R-MAT s22, whose hubs hold 10^5
// entries (whole calls, with the traversal: 1.90 -> 1.00 and 18.3 -> 1.12 ms).
__global__ void __launch_bounds__(VT) k_val_rows(const int64_t* __restrict__ off, const int32_t* __restrict__ rows,
                                                 const int32_t* __restrict__ deg, int64_t n_active,
                                                 const uint32_t* __restrict__ dt, int short_rows,
                                                 unsigned long long* broken) {
  __shared__ int64_t s_bound[2];
  __shared__ unsigned s_mn[VT / 32], s_mx[VT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (short_rows) {  // in any order
    if (threadIdx.x < 2) s_bound[threadIdx.x] = 0;
  } else if (warp < 2) {
    const int64_t b = first_below(deg, n_active, warp == 0 ? VAL_CTA : VAL_WARP);
    if (lane == 0) s_bound[warp] = b;
  }
  __syncthreads();
  const int64_t n_cta = s_bound[0], n_warp = s_bound[1];
  bool bad = false;
  // entries [at, end) of a row, `step` apart per lane and round
  const auto scan = [&](int64_t at, int64_t step, int64_t end, unsigned& mn, unsigned& mx) {
    for (; at < end; at += step * VAL_ILP) {
      int u[VAL_ILP];
#pragma unroll
      for (int i = 0; i < VAL_ILP; ++i) u[i] = at + step * i < end ? __ldg(rows + at + step * i) : -1;
#pragma unroll
      for (int i = 0; i < VAL_ILP; ++i)
        if (u[i] >= 0) {
          const unsigned du = __ldg(dt + u[i]);
          mn = min(mn, du);
          mx = max(mx, du);
        }
    }
  };
  for (int64_t v = blockIdx.x; v < n_cta; v += gridDim.x) {
    unsigned mn = ~0u, mx = 0;
    scan(off[v] + threadIdx.x, VT, off[v + 1], mn, mx);
    mn = __reduce_min_sync(FULL, mn);
    mx = __reduce_max_sync(FULL, mx);
    __syncthreads();
    if (lane == 0) s_mn[warp] = mn, s_mx[warp] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < VT / 32; ++w) mn = min(mn, s_mn[w]), mx = max(mx, s_mx[w]);
      bad |= row_breaks(dt[v], mn, mx);
    }
  }
  const int64_t gw = (blockIdx.x * (int64_t)VT + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * VT) >> 5;
  for (int64_t v = n_cta + gw; v < n_warp; v += nw) {
    unsigned mn = ~0u, mx = 0;
    scan(off[v] + lane, 32, off[v + 1], mn, mx);
    mn = __reduce_min_sync(FULL, mn);
    mx = __reduce_max_sync(FULL, mx);
    bad |= row_breaks(dt[v], mn, mx);
  }
  for (int64_t v = n_warp + gw * 32 + lane; v < n_active; v += nw * 32) {
    unsigned mn = ~0u, mx = 0;
    const int64_t b = off[v];
    scan(b, 1, b + deg[v], mn, mx);
    bad |= row_breaks(dt[v], mn, mx);
  }
  if (bad) *broken = 1;
}

__device__ __forceinline__ bool row_has(const int64_t* off, const int32_t* rows, int32_t p, int32_t v) {
  int64_t lo = off[p], hi = off[p + 1];  // rows sorted ascending
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    const int32_t x = rows[mid];
    if (x == v) return true;
    if (x < v) lo = mid + 1;
    else hi = mid;
  }
  return false;
}

__device__ __forceinline__ int parent_code(const int64_t* off, const int32_t* rows_sorted, int64_t V, int32_t v,
                                           const int32_t* depth, int dv, int p, bool symmetric = false) {
  if (dv == -1) return p != -1 ? -2 : 0;
  if (p < 0 || p >= V) return -3;
  if (depth[p] != dv - 1) return -4;
  return (symmetric ? row_has(off, rows_sorted, v, p) : row_has(off, rows_sorted, p, v)) ? 0 : -5;
}

__global__ void __launch_bounds__(VT) k_val_parent(const int64_t* __restrict__ off,
                                                   const int32_t* __restrict__ rows_sorted, int64_t V, int32_t src,
                                                   const int32_t* __restrict__ depth,
                                                   const int32_t* __restrict__ parent, unsigned long long* slot) {
  for (int64_t v = blockIdx.x * (int64_t)VT + threadIdx.x; v < V; v += (int64_t)gridDim.x * VT) {
    if (v == src) continue;
    const int code = parent_code(off, rows_sorted, V, (int32_t)v, depth, depth[v], parent[v]);
    if (code) report(slot, v, code);
  }
}

// The rules that need no row, over caller ids: depths of their own, the rules
// of the source, and (with parents and sorted rows) the parent certificate;
// and the depths by traversal id, for k_val_rows. Where every edge is known to
// be there both ways, the vertex looks for its parent in its own row, which
// lies beside its neighbour thread's, instead of for itself in the parent's
// row, a random one: a traversal of ER 2^22 x 16 with its certificates 1018 us, 890 so.
__global__ void __launch_bounds__(VT) k_val_vertex(const int64_t* __restrict__ off, const int32_t* __restrict__ adj,
                                                   const int32_t* __restrict__ inv, int64_t V, int64_t n_active,
                                                   int32_t src, const int32_t* __restrict__ depth,
                                                   const int32_t* __restrict__ parent, bool symmetric,
                                                   int32_t* __restrict__ dt, unsigned long long* words) {
  for (int64_t v = blockIdx.x * (int64_t)VT + threadIdx.x; v < V; v += (int64_t)gridDim.x * VT) {
    const int dv = depth[v], i = inv ? inv[v] : (int)v, p = parent ? parent[v] : -1;
    if (inv) dt[i] = dv;
    if (dv < -1 || (dv == 0 && v != src) || (dv > 0 && i >= n_active)) words[3] = 1;
    if (v == src) {
      if (dv != 0) words[4] = 1;
      if (parent && (p != src || dv != 0)) words[5] = 1;
    } else if (parent) {
      const int code = parent_code(off, adj, V, (int32_t)v, depth, dv, p, symmetric);
      if (code) report(words + 1, v, code);
    }
  }
}

__global__ void k_rows_unsorted(const int64_t* __restrict__ off, const int32_t* __restrict__ adj, int64_t V,
                                unsigned long long* n_bad) {
  for (int64_t v = blockIdx.x * (int64_t)VT + threadIdx.x; v < V; v += (int64_t)gridDim.x * VT)
    for (int64_t k = off[v] + 1; k < off[v + 1]; ++k)
      if (adj[k - 1] > adj[k]) {
        atomicAdd(n_bad, 1ull);
        break;
      }
}

__global__ void k_val_src(int32_t src, const int32_t* depth, const int32_t* parent, unsigned long long* words) {
  if (blockIdx.x || threadIdx.x) return;
  if (depth[src] != 0) words[4] = 1;
  if (parent && (parent[src] != src || depth[src] != 0)) words[5] = 1;
}

void decode(unsigned long long key, int32_t* code, int64_t* bad) {
  if (key == ~0ull) {
    *code = 0;
    *bad = -1;
  } else {
    *code = -(int32_t)(key & 0xff);
    *bad = (int64_t)(key >> 8);
  }
}

}  // namespace
}  // namespace ent

using namespace ent;

extern "C" int ent_validate(ent_graph* g, int32_t src, const int32_t* depth_dev, const int32_t* parent_dev,
                            int32_t* depth_code, int64_t* depth_bad, int32_t* parent_code, int64_t* parent_bad) {
  ent::NvtxRange nvtx_range("ent_validate");
  clear_error();
  if (!g || !depth_dev || !depth_code || !depth_bad) return fail(ENT_ERR_INVALID_ARG, "null argument");
  if (parent_dev && (!parent_code || !parent_bad)) return fail(ENT_ERR_INVALID_ARG, "null parent result");
  if (src < 0 || src >= g->V) return fail(ENT_ERR_INVALID_ARG, "source %d out of range", src);
  std::lock_guard<std::mutex> lk(g->mu);
  DeviceGuard dg(g->device);
  cudaStream_t s = g->stream;
  const int64_t V = g->V, E = g->E;
  // [0] depth certificate, [1] parent certificate (smallest vertex << 8 | rule),
  // [2] unsorted rows, [3] some depth rule broken, [4], [5] the source's own
  // depth and parent rules (the oracle checks them first: they win)
  constexpr int NW = 6;
  unsigned long long h[NW];
  if (!g->val) {
    const cudaError_t ea = dev_alloc(&g->val, 256 + sizeof(int32_t) * (g->perm ? V : 0));
    if (ea != cudaSuccess) {
      g->val = nullptr;
      return fail(ENT_ERR_OOM, "validation scratch: %s", cudaGetErrorString(ea));
    }
  }
  unsigned long long* words = (unsigned long long*)g->val;
  int32_t* dt = (int32_t*)((char*)g->val + 256);
  int32_t* sorted = nullptr;
  void* tmp = nullptr;
  int rc = ENT_OK;
  const int grid = g->num_sms * 8;
  const auto launched = [] {
    g_kernel_launches++;
    return cudaGetLastError();
  };
  const auto read_words = [&] {
    cudaError_t x = cudaMemcpyAsync(h, words, sizeof(h), cudaMemcpyDeviceToHost, s);
    return x == cudaSuccess ? cudaStreamSynchronize(s) : x;
  };
  cudaError_t e = cudaMemsetAsync(words, 0xFF, 2 * sizeof(unsigned long long), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(words + 2, 0, (NW - 2) * sizeof(unsigned long long), s);
  const bool fast = g->perm || g->road;               // else the rows are in caller order, of any lengths
  const bool fast_parent = fast && g->rows_sorted;
  if (e == cudaSuccess && fast) {
    k_val_vertex<<<grid, VT, 0, s>>>(g->off, g->adj, g->inv, V, g->n_active, src, depth_dev,
                                     fast_parent ? parent_dev : nullptr, g->symmetric, dt, words);
    e = launched();
    if (e == cudaSuccess) {
      k_val_rows<<<grid, VT, 0, s>>>(g->toff, g->trav, g->deg, g->n_active,
                                       (const uint32_t*)(g->perm ? dt : depth_dev), g->road, words + 3);
      e = launched();
    }
    if (e == cudaSuccess) e = read_words();
  }
  if (e == cudaSuccess && (!fast || h[3] || (parent_dev && !fast_parent))) {
    if (!fast || h[3]) {
      k_val_depth<<<grid, VT, 0, s>>>(g->off, g->adj, V, src, depth_dev, words);
      e = launched();
    }
    const int32_t* rows = g->adj;
    if (e == cudaSuccess && parent_dev && !fast_parent) {
      // binary search needs sorted rows: check, and sort a copy if a caller's
      // CSR came with unsorted rows
      k_rows_unsorted<<<grid, VT, 0, s>>>(g->off, g->adj, V, words + 2);
      e = launched();
      if (e == cudaSuccess) e = read_words();
      if (e == cudaSuccess && h[2] != 0) {
        if (E > 0x7fffffffll) {
          rc = fail(ENT_ERR_UNSUPPORTED, "parent validation of unsorted rows needs E < 2^31");
        } else {
          size_t tmp_bytes = 0;
          e = cudaMallocAsync(&sorted, sizeof(int32_t) * E, s);
          if (e == cudaSuccess)
            e = cub::DeviceSegmentedSort::SortKeys(nullptr, tmp_bytes, g->adj, sorted, (int)E, (int)V, g->off,
                                                   g->off + 1, s);
          if (e == cudaSuccess) e = cudaMallocAsync(&tmp, tmp_bytes, s);
          if (e == cudaSuccess)
            e = cub::DeviceSegmentedSort::SortKeys(tmp, tmp_bytes, g->adj, sorted, (int)E, (int)V, g->off,
                                                   g->off + 1, s);
          rows = sorted;
        }
      }
      if (e == cudaSuccess && rc == ENT_OK) {
        k_val_parent<<<grid, VT, 0, s>>>(g->off, rows, V, src, depth_dev, parent_dev, words + 1);
        e = launched();
      }
    }
    if (e == cudaSuccess && rc == ENT_OK) {
      k_val_src<<<1, 32, 0, s>>>(src, depth_dev, parent_dev, words);
      e = launched();
    }
    if (e == cudaSuccess && rc == ENT_OK) e = read_words();
  }
  if (sorted) cudaFreeAsync(sorted, s);
  if (tmp) cudaFreeAsync(tmp, s);
  const cudaError_t e2 = rc != ENT_OK || e != cudaSuccess || sorted ? cudaStreamSynchronize(s) : cudaSuccess;
  if (rc != ENT_OK) return rc;
  if (e != cudaSuccess || e2 != cudaSuccess)
    return fail(ENT_ERR_CUDA, "validation failed: %s", cudaGetErrorString(e != cudaSuccess ? e : e2));
  decode(h[4] ? ((unsigned long long)src << 8 | 1u) : h[0], depth_code, depth_bad);
  if (parent_dev) decode(h[5] ? ((unsigned long long)src << 8 | 1u) : h[1], parent_code, parent_bad);
  return ENT_OK;
}
