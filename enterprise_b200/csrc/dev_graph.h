// Device-resident graph handle and the traversal workspaces hanging off it.
#pragma once
#include <cuda_runtime.h>
#include <mutex>
#include <stdint.h>
#include "ent_internal.h"

namespace ent {
struct BfsWorkspace;    // single-source direction-optimising traversal
struct BatchWorkspace;  // bitwise multi-source traversal
struct DeepLanes;       // concurrent single-source traversals of a batch on a deep graph
void destroy_bfs_workspace(BfsWorkspace* w);
void destroy_batch_workspace(BatchWorkspace* w);
void destroy_deep_lanes(DeepLanes* l);
}  // namespace ent

// Device memory layout of one graph (all on `device`):
//   off  int64[V+1]   row offsets (reference strt_pos + adj_card, allocator.cuh:107-114)
//   adj  int32[E]     column ids, rows ascending (reference adj_list, allocator.cuh:116-120)
// and the traversal's own arrays (one slab), in traversal ids: vertices by
// descending degree, ties by caller id. The vertices without a row come last,
// so a bottom-up sweep covers the first n_active ids without idle lanes; a
// warp's 32 vertices have (nearly) equal degrees and adjacent rows; and the
// hubs, which most probes hit, share a few cache lines of every per-vertex
// array. Caller ids appear only where sources come in and results go out.
//   perm int32[V]     caller id of each traversal id (null: caller order, when
//                     E >= 2^31 or E == 0 and on road-like graphs; toff and trav
//                     are then off and adj)
//   inv  int32[V]     traversal id of each caller id
//   toff int64[V+1]   row offsets
//   trav int32[E]     the rows, ascending: the highest-degree neighbours first.
//                     A bottom-up check then meets the likeliest parent, a hub,
//                     first.
//   deg  int32[V]     degrees, read by the classifier (reference adj_card)
//   active uint32[V/32] bit v set iff deg(v) > 0 (bottom-up skips isolated vertices)
//   lead int4[V]      first 4 entries of each trav row (the highest-degree
//                     neighbours), -1 past the row's end: a bottom-up sweep
//                     reads them coalesced instead of a random row sector per
//                     vertex, and most light vertices need nothing else.
struct ent_graph {
  int device = 0;
  int num_sms = 0;
  int64_t V = 0, E = 0;
  int64_t* off = nullptr;
  int32_t* adj = nullptr;
  void* slab = nullptr;  // the arrays below (toff and trav may alias off and adj)
  int32_t* perm = nullptr;
  int32_t* inv = nullptr;
  int64_t* toff = nullptr;
  int32_t* trav = nullptr;
  int32_t* deg = nullptr;
  uint32_t* active = nullptr;
  int4* lead = nullptr;
  int64_t n_active = 0;  // vertices with a row are traversal ids [0, n_active); V in caller order
  bool road = false;         // low mean degree and no hub: keeps the caller's order
  bool symmetric = false;  // every edge is there both ways (rows built here from undirected edges)
  bool rows_sorted = false;  // every adj row is ascending (known with an order of its own, and for road-like graphs)
  cudaStream_t stream = nullptr;
  ent_bfs_opts opts;
  std::mutex mu;
  ent::BfsWorkspace* ws = nullptr;
  ent::BatchWorkspace* bws = nullptr;
  ent::DeepLanes* lanes = nullptr;
  int32_t deep = -1;          // whether traversals have many small levels (-1: not yet known)
  int32_t probe_levels = -1;  // depth of the graph as probed by its first auto-mode batch (-1: not yet)
  void* stage = nullptr;      // device rows of batches whose results go to host memory
  size_t stage_cap = 0;
  void* val = nullptr;        // ent_validate's scratch: its result words, a depth per vertex
};

namespace ent {

// RAII device guard: switches to `dev`, restores the previous device.
struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    int cur;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

// Whether stream s is being captured into a graph (events of other streams
// then have no place in it).
inline bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) cudaGetLastError();
  return cap != cudaStreamCaptureStatusNone;
}

#define ENT_CUDA(call)                                                                      \
  do {                                                                                      \
    cudaError_t _e = (call);                                                                \
    if (_e != cudaSuccess)                                                                  \
      return ::ent::fail(_e == cudaErrorMemoryAllocation ? ENT_ERR_OOM : ENT_ERR_CUDA,      \
                         "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e), __FILE__, \
                         __LINE__);                                                         \
  } while (0)

// Device memory of the library's own, from a pool (memory.cpp), on the current
// device and ready for any stream. dev_free: no work may still use the memory.
cudaError_t dev_alloc(void** out, size_t bytes);
void dev_free(void* ptr);
template <class T>
cudaError_t dev_alloc(T** out, size_t bytes) { return dev_alloc(reinterpret_cast<void**>(out), bytes); }
// cudaMalloc, for memory whose address a caller may get (it can be shared with
// peers and other processes, which pool memory cannot); frees what the pool
// keeps before it fails.
cudaError_t dev_malloc(void** out, size_t bytes);
template <class T>
cudaError_t dev_malloc(T** out, size_t bytes) { return dev_malloc(reinterpret_cast<void**>(out), bytes); }
// A page-locked block of at most 512 bytes, for copies from any device; null
// when there is no memory. host_slot_free: no copy may still use it.
void* host_slot(size_t bytes);
void host_slot_free(void* p);
// Copies on stream s between the device and host memory of any kind. Pageable
// memory has been read, or holds the data, when the call returns (after the
// stream got there); page-locked memory is copied asynchronously.
cudaError_t to_device(void* dst, const void* src, size_t bytes, cudaStream_t s);
cudaError_t to_host(void* dst, const void* src, size_t bytes, cudaStream_t s);
// `rows` rows of `width` bytes, `pitch` apart on the device, to a contiguous host array.
cudaError_t rows_to_host(void* dst, const void* src, size_t width, size_t pitch, size_t rows, cudaStream_t s);

int graph_alloc(ent_graph* g, int64_t V, int64_t E);
int graph_finish(ent_graph* g);  // computes deg, creates stream
int run_bfs_single(ent_graph* g, int32_t src, int32_t* depth_dev, int32_t* parent_dev, cudaStream_t stream,
                   ent_stats* stats);
int run_bfs_batch(ent_graph* g, const int32_t* src, int32_t n_src, int32_t* depth_dev, cudaStream_t stream,
                  ent_stats* stats, bool bytes = false);
// Depth (levels) of g seen from the given candidate sources: single-source
// traversals from up to three of them (the deepest answer wins; a source that
// reaches a quarter of the graph ends the search). Synchronous, on g->stream;
// the caller holds g->mu.
int probe_graph_levels(ent_graph* g, const int32_t* src, int32_t n_src, int32_t* levels);
// A batch on a deep graph as concurrent single-source traversals, one per
// lane; rows as run_bfs_batch writes them (int32, or bytes with 255 for
// unreached). Ordered after and before `stream` like a launch on it; stats
// (n_src entries) synchronise. The caller holds g->mu.
int run_bfs_deep(ent_graph* g, const int32_t* src, int32_t n_src, void* depth_dev, bool bytes, cudaStream_t stream,
                 ent_stats* stats);

}  // namespace ent
