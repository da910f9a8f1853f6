// Breadth-first search that allocates no memory at all.
//
// Some callers cannot allocate GPU memory when they need a traversal: code on
// a latency-critical request path, where a cudaMalloc/cudaFree may
// synchronise the whole device and stall unrelated streams; plug-ins inside
// a host process whose GPU memory is already owned by another allocator (a
// framework's caching allocator or a fixed, pre-reserved budget); and code
// that must not fail half-way with an out-of-memory error. For them this file
// provides ent_bfs_noalloc: the caller passes the CSR and the depth output,
// both already on the GPU, and the traversal's scratch lives in a file-scope
// __device__ array that exists on every GPU that loads this library, for the
// lifetime of the process.
//
// The scratch holds a visited bitmap, two frontier queues and a control block
// for at most NOALLOC_MAX_VERTICES vertices (about 8.5 MB per GPU). Larger
// graphs are rejected with ENT_ERR_INVALID_ARG. The traversal is level-
// synchronous top-down (the caller's rows need not hold both directions of an
// edge, which bottom-up levels would rely on) and gives exactly the depths
// every other entry point of this library produces.
//
// The whole traversal is one cooperative launch: its CTAs go from level to
// level through a grid-wide barrier (bounded waits), so the host neither
// launches nor waits per level. While the frontier is small, CTA 0 runs the
// levels alone with its frontier in shared memory and the others wait at the
// barrier.
//
// Sharing: every call uses the same array and leaves its last contents
// behind; each call clears the visited bitmap and the counters before it
// starts. Two calls whose work overlaps on the same GPU (for example from two
// host threads at once, or on two streams) race on the shared scratch and
// produce wrong results: callers must serialise them.
#include <algorithm>
#include <cuda_runtime.h>
#include <mutex>
#include <stdint.h>
#include <vector>

#include "dev_common.cuh"
#include "ent_internal.h"

namespace ent {

constexpr int64_t NOALLOC_MAX_VERTICES = 1 << 20;
constexpr int64_t NOALLOC_WORDS = NOALLOC_MAX_VERTICES / 32;

// Layout inside the scratch array (all offsets 256-byte aligned):
//   [0]                       uint32 visited[NOALLOC_WORDS]
//   [NOALLOC_WORDS*4]         int32  queue[2][NOALLOC_MAX_VERTICES]
//   [.. + 8*MAX]              NaCtl
// A queue holds light vertices from its front and heavy ones from its back
// (together at most V entries).
constexpr size_t NA_OFF_QUEUE = NOALLOC_WORDS * 4;
constexpr size_t NA_OFF_CTL = NA_OFF_QUEUE + 2 * NOALLOC_MAX_VERTICES * 4;

constexpr int NA_T = 1024;        // threads per CTA, one per SM
constexpr int NA_ILP = 4;         // entries a lane has in flight together
constexpr int NA_HEAVY = 256;     // degree from which a CTA takes a vertex's row
constexpr int NA_HUGE = 1 << 15;  // ... and from which all CTAs share it
constexpr int NA_HUGE_CAP = 1024; // listed ones per level (more are rows of one CTA)
constexpr int NA_SOLO = 1024;     // light frontier vertices up to which CTA 0 runs alone
constexpr int NA_SOLO_M = 4096;   // ... and the sum of their degrees; it leaves above twice that
constexpr int NA_SOLO_CAP = 2048; // frontier entries it keeps in shared memory
constexpr int NA_SOLO_LEVELS = 4096;  // levels it runs before it meets the others again

struct NaCtl {
  uint32_t arrived;   // barrier arrivals, all barriers of a launch together
  int32_t err;        // a wait ran out
  int32_t level[2];   // per phase (mod 2): the level CTA 0 reached running alone
  int32_t n[3][4];    // per phase (mod 3): light, heavy, huge frontier vertices; degree sum of the light
  int32_t huge[2][NA_HUGE_CAP];
};
constexpr size_t NA_BYTES = (NA_OFF_CTL + sizeof(NaCtl) + 255) / 256 * 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];

struct NaArgs {
  uint32_t* visited;
  int32_t* queue[2];
  NaCtl* ctl;
  const int64_t* off;
  const int32_t* adj;
  int32_t* depth;
  int64_t V;
  int32_t src;
};

// Where the claimed vertices of a level go.
struct NaOut {
  int32_t* q;        // the next level's queue
  int32_t* n;        // its global counts
  int32_t* huge;     // its huge list
  // CTA 0 alone: light vertices go to shared memory while they fit
  int4* s_q;
  int32_t* s_n;      // [3]: light, heavy, huge
};

// Claims the neighbours v[] (negative: none) of frontier vertices for `ln` and
// queues the won ones by degree. One warp, converged. my_m: the lane's sum of the
// light ones' degrees (CTA 0 alone adds them beside the count instead: the sums
// at the level's end would lengthen its chain).
template <bool SOLO>
__device__ __forceinline__ void na_claim(const NaArgs& a, const int (&v)[NA_ILP], int ln, const NaOut& o,
                                         unsigned& my_m) {
  const int lane = threadIdx.x & 31;
  bool open[NA_ILP], mine[NA_ILP];
  int64_t st[NA_ILP];
  int d[NA_ILP];
  // A look through L1 saves most atomics (a stale word only costs one); a
  // small frontier claims at once: the look would lengthen its chain.
#pragma unroll
  for (int i = 0; i < NA_ILP; ++i)
    open[i] = v[i] >= 0 && (SOLO || !((__ldca(a.visited + (v[i] >> 5)) >> (v[i] & 31)) & 1u));
#pragma unroll
  for (int i = 0; i < NA_ILP; ++i) {
    mine[i] = false;
    st[i] = 0;
    d[i] = 0;
    if (open[i]) {  // the row is read beside the claim
      const int64_t o0 = __ldg(a.off + v[i]), o1 = __ldg(a.off + v[i] + 1);
      const uint32_t b = 1u << (v[i] & 31);
      mine[i] = !(atomicOr(a.visited + (v[i] >> 5), b) & b);
      st[i] = o0;
      d[i] = (int)min(o1 - o0, (int64_t)INT32_MAX);
    }
  }
  int n_light = 0;
  unsigned m_light = 0;
#pragma unroll
  for (int i = 0; i < NA_ILP; ++i) {
    if (mine[i]) a.depth[v[i]] = ln;
    const bool light = mine[i] && d[i] > 0 && d[i] < NA_HEAVY;
    n_light += __popc(__ballot_sync(FULL, light));
    m_light += light ? d[i] : 0;
  }
  int base = 0;
  if (n_light) {
    if (SOLO) {
      m_light = __reduce_add_sync(FULL, m_light);
      if (lane < 2) base = atomicAdd(o.s_n + 3 * lane, lane ? (int)m_light : n_light);
    } else {
      if (lane == 0) base = atomicAdd(o.n, n_light);
      my_m += m_light;
    }
    base = __shfl_sync(FULL, base, 0);
  }
#pragma unroll
  for (int i = 0; i < NA_ILP; ++i) {
    const bool light = mine[i] && d[i] > 0 && d[i] < NA_HEAVY;
    const unsigned m = __ballot_sync(FULL, light);
    if (light) {
      const int at = base + __popc(m & lanemask_lt());
      if (SOLO && at < NA_SOLO_CAP)
        o.s_q[at] = make_int4(v[i], d[i], (int)(uint32_t)st[i], (int)(uint32_t)((uint64_t)st[i] >> 32));
      else
        o.q[at] = v[i];
    }
    base += __popc(m);
    if (mine[i] && d[i] >= NA_HEAVY) {  // few: one atomic each
      const int h = d[i] >= NA_HUGE ? atomicAdd((SOLO ? o.s_n : o.n) + 2, 1) : NA_HUGE_CAP;
      if (h < NA_HUGE_CAP) o.huge[h] = v[i];
      else o.q[NOALLOC_MAX_VERTICES - 1 - atomicAdd((SOLO ? o.s_n : o.n) + 1, 1)] = v[i];
    }
  }
}

// The concatenated rows of a warp's light vertices (lane: one row of d entries
// from st, d = 0: none), NA_ILP rounds of 32 entries together.
template <bool SOLO>
__device__ __forceinline__ void na_rows(const NaArgs& a, int d, int64_t st, int ln, const NaOut& o, unsigned& my_m) {
  const int lane = threadIdx.x & 31;
  int incl = d;
#pragma unroll
  for (int ofs = 1; ofs < 32; ofs <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, ofs);
    if (lane >= ofs) incl += y;
  }
  const int total = __shfl_sync(FULL, incl, 31), excl = incl - d;
  for (int r0 = 0; r0 < total; r0 += 32 * NA_ILP) {
    int v[NA_ILP];
#pragma unroll
    for (int i = 0; i < NA_ILP; ++i) {
      v[i] = -1;
      if (r0 + 32 * i < total) {  // warp-uniform
        const int k = r0 + 32 * i + lane;
        int j = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const int ev = __shfl_sync(FULL, excl, (j + step) & 31);
          if (j + step < 32 && ev <= k) j += step;
        }
        const int64_t sj = __shfl_sync(FULL, st, j);
        const int ej = __shfl_sync(FULL, excl, j);
        if (k < total) v[i] = __ldg(a.adj + sj + (k - ej));
      }
    }
    na_claim<SOLO>(a, v, ln, o, my_m);
  }
}

// Entries first, first + step, ... below end of one long row, 32 * NA_ILP
// consecutive ones per warp and turn.
__device__ __forceinline__ void na_slice(const NaArgs& a, int64_t first, int64_t step, int64_t end, int ln,
                                         const NaOut& o, unsigned& my_m) {
  const int lane = threadIdx.x & 31;
  for (int64_t e0 = first; e0 < end; e0 += step) {
    int v[NA_ILP];
#pragma unroll
    for (int i = 0; i < NA_ILP; ++i) {
      const int64_t e = e0 + 32 * i + lane;
      v[i] = e < end ? __ldg(a.adj + e) : -1;
    }
    na_claim<false>(a, v, ln, o, my_m);
  }
}

// CTA 0 alone, from level L on: runs levels while all frontier vertices are
// light and fit and their rows are few, at most NA_SOLO_LEVELS, and leaves the
// next frontier in the queues, its counts in `out` and its level in *level. It
// walks about 1.2 entries a ns: without the bound on the rows a band graph of
// 1000-vertex levels took 147 us a level at degree 200 and 19 at 20, and 12 and 8
// so. The bound costs 2% where it never applies (700 x 700 grid 4.12 -> 4.20 ms,
// R-MAT s18 221 -> 225 us; sums at the level's end cost the grid 3%).
__device__ void na_solo(const NaArgs& a, int L, int n, int4 (*s_q)[NA_SOLO_CAP], int32_t (*s_n)[4], int32_t* out,
                        int32_t* level) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NWARP = NA_T / 32;
  const int32_t* q0 = a.queue[L & 1];
  for (int i = tid; i < n; i += NA_T) {
    const int u = __ldcg(q0 + i);
    const int64_t st = a.off[u];
    s_q[L & 1][i] = make_int4(u, (int)(a.off[u + 1] - st), (int)(uint32_t)st, (int)(uint32_t)((uint64_t)st >> 32));
  }
  if (tid < 4) s_n[0][tid] = s_n[1][tid] = 0;
  __syncthreads();
  int n2 = 0, n3 = 0, m = 0;
  for (int run = 0;; ++run) {
    const int cur = L & 1, nxt = cur ^ 1;
    const NaOut o{a.queue[nxt], nullptr, a.ctl->huge[nxt], s_q[nxt], s_n[nxt]};
    // up to 32 rows per warp, spread over all warps
    const int k = min(32, (n + NWARP - 1) / NWARP);
    unsigned unused = 0;
    for (int first = warp * k; first < n; first += NWARP * k) {
      int d = 0;
      int64_t st = 0;
      if (lane < k && first + lane < n) {
        const int4 e = s_q[cur][first + lane];
        d = e.y;
        st = (int64_t)(((uint64_t)(uint32_t)e.w << 32) | (uint32_t)e.z);
      }
      na_rows<true>(a, d, st, L + 1, o, unused);
    }
    __syncthreads();
    n = s_n[nxt][0];
    n2 = s_n[nxt][1];
    n3 = s_n[nxt][2];
    ++L;
    m = s_n[nxt][3];
    if (n == 0 || n > NA_SOLO_CAP || m > 2 * NA_SOLO_M || n2 || n3 || run + 1 >= NA_SOLO_LEVELS) break;
    if (tid < 4) s_n[cur][tid] = 0;  // takes the counts of the level after
    __syncthreads();
  }
  // hand over: stored entries to the queue (the rest are there), counts
  int32_t* q = a.queue[L & 1];
  for (int i = tid; i < min(n, NA_SOLO_CAP); i += NA_T) q[i] = s_q[L & 1][i].x;
  if (tid == 0) {
    out[0] = n;
    out[1] = n2;
    out[2] = n3;
    out[3] = m;
    *level = L;
  }
}

// The whole traversal (cooperative launch; the control block is zeroed before).
// Bound by the atomics and scattered reads of the entries on wide levels and
// by the barrier and the chain entry -> row -> claim on narrow ones. R-MAT
// s18: 0.23 ms; a 700 x 700 grid: 4.2 ms, 2.6 us a level (a launch and a host
// wait per level, a warp per vertex: 1.17 and 18.8 ms). 1024 threads and one
// CTA per SM beat two of 512 (grid 5.2 ms: CTA 0 alone has more lanes); rows
// of one CTA from 256 entries beat 64 and 1024 (0.28 ms at s18), four entries
// per lane two (0.27 ms).
// A phase is one level of all CTAs, or several of CTA 0 alone; a barrier ends
// it. Phase p reads the counts n[p % 3], fills n[(p + 1) % 3] and clears
// n[(p + 2) % 3], which no CTA reads any more once it is past the barrier
// before: a CTA that is late to read n[p % 3] still finds it unchanged.
__global__ void __launch_bounds__(NA_T, 1) k_na_run(NaArgs a) {
  extern __shared__ int4 s_dyn[];
  int4(*s_q)[NA_SOLO_CAP] = reinterpret_cast<int4(*)[NA_SOLO_CAP]>(s_dyn);
  __shared__ int32_t s_n[2][4];
  __shared__ unsigned s_m;
  if (threadIdx.x == 0) s_m = 0;
  NaCtl* c = a.ctl;
  const int64_t tid = blockIdx.x * (int64_t)NA_T + threadIdx.x, nth = (int64_t)gridDim.x * NA_T;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NWARP = NA_T / 32;
  const int64_t W = (a.V + 31) >> 5;
  for (int64_t i = tid; i < W; i += nth) a.visited[i] = i == (a.src >> 5) ? 1u << (a.src & 31) : 0u;
  for (int64_t i = tid; i < a.V; i += nth) a.depth[i] = i == a.src ? 0 : -1;
  if (tid == 0) {
    const int64_t d = a.off[a.src + 1] - a.off[a.src];
    if (d > 0 && d < NA_HEAVY) {
      a.queue[0][0] = a.src;
      c->n[0][0] = 1;
      c->n[0][3] = (int32_t)d;
    } else if (d >= NA_HEAVY) {
      a.queue[0][NOALLOC_MAX_VERTICES - 1] = a.src;
      c->n[0][1] = 1;
    }
  }
  uint32_t target = 0;
  if (!grid_barrier(&c->arrived, &c->err, target += gridDim.x, [] {})) return;
  int L = 0;
  for (int p = 0; L <= a.V; ++p) {
    const int32_t* cnt = c->n[p % 3];
    int32_t* next = c->n[(p + 1) % 3];
    const int n_l = __ldcg(cnt), n_h = __ldcg(cnt + 1), n_g = min(__ldcg(cnt + 2), NA_HUGE_CAP);
    if (n_l + n_h + n_g == 0) return;
    if (tid < 4) c->n[(p + 2) % 3][tid] = 0;
    if (n_l <= NA_SOLO && __ldcg(cnt + 3) <= NA_SOLO_M && n_h + n_g == 0) {
      if (blockIdx.x == 0) na_solo(a, L, n_l, s_q, s_n, next, &c->level[p & 1]);
      if (!grid_barrier(&c->arrived, &c->err, target += gridDim.x, [] {})) return;
      L = __ldcg(&c->level[p & 1]);
      continue;
    }
    const int32_t* q = a.queue[L & 1];
    const NaOut o{a.queue[(L + 1) & 1], next, c->huge[(L + 1) & 1], nullptr, nullptr};
    const int64_t gw = (int64_t)blockIdx.x * NWARP + warp, nw = (int64_t)gridDim.x * NWARP;
    unsigned my_m = 0;
    for (int i = 0; i < n_g; ++i) {  // rows shared by all CTAs
      const int u = __ldcg(c->huge[L & 1] + i);
      const int64_t beg = a.off[u], end = a.off[u + 1];
      na_slice(a, beg + gw * 32 * NA_ILP, nw * 32 * NA_ILP, end, L + 1, o, my_m);
    }
    for (int i = blockIdx.x; i < n_h; i += gridDim.x) {  // rows of one CTA
      const int u = __ldcg(q + NOALLOC_MAX_VERTICES - 1 - i);
      const int64_t beg = a.off[u], end = a.off[u + 1];
      na_slice(a, beg + warp * 32 * NA_ILP, NWARP * 32 * NA_ILP, end, L + 1, o, my_m);
    }
    // up to 32 light rows per warp, spread over all warps
    const int k = (int)min((int64_t)32, (n_l + nw - 1) / nw);
    for (int64_t first = gw * k; first < n_l; first += nw * k) {
      int d = 0;
      int64_t st = 0;
      if (lane < k && first + lane < n_l) {
        const int u = __ldcg(q + first + lane);
        st = a.off[u];
        d = (int)(a.off[u + 1] - st);
      }
      na_rows<false>(a, d, st, L + 1, o, my_m);
    }
    my_m = __reduce_add_sync(FULL, my_m);
    if (lane == 0 && my_m) atomicAdd(&s_m, my_m);
    __syncthreads();
    if (threadIdx.x == 0 && s_m) {
      atomicAdd(next + 3, (int)s_m);
      s_m = 0;
    }
    ++L;
    if (!grid_barrier(&c->arrived, &c->err, target += gridDim.x, [] {})) return;
  }
  if (tid == 0) c->err = 2;  // more levels than vertices
}

// Device address of the scratch array, looked up once per device and CUDA
// context with that device current (in host code the symbol's name is only a
// stand-in). An address is valid only in the context it was looked up in, so
// a caller that switches between the runtime's primary context and a context
// of its own (a driver-API plug-in) gets one lookup in each.
typedef int (*CtxGetCurrentFn)(void**);  // cuCtxGetCurrent, from the driver
struct NaEntry {
  int dev;
  void* ctx;
  unsigned char* ptr;
};
static std::mutex g_na_mu;
static std::vector<NaEntry> g_na_cache;
static CtxGetCurrentFn g_ctx_get = nullptr;

static int na_scratch_for_current_device(unsigned char** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(ENT_ERR_CUDA, "cudaGetDevice failed: %s", cudaGetErrorString(e));
  std::lock_guard<std::mutex> lk(g_na_mu);
  if (!g_ctx_get) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    e = cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn)
      return fail(ENT_ERR_CUDA, "driver entry point cuCtxGetCurrent unavailable: %s", cudaGetErrorString(e));
    g_ctx_get = reinterpret_cast<CtxGetCurrentFn>(fn);
  }
  void* ctx = nullptr;
  if (g_ctx_get(&ctx) != 0) return fail(ENT_ERR_CUDA, "cuCtxGetCurrent failed on device %d", dev);
  if (ctx)
    for (const NaEntry& n : g_na_cache)
      if (n.dev == dev && n.ctx == ctx) {
        *out = n.ptr;
        return ENT_OK;
      }
  // Not seen in this context (or no context is bound to this thread yet: the
  // lookup binds the device's primary context, as any runtime call does).
  void* p = nullptr;
  e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess || !p)
    return fail(ENT_ERR_CUDA, "cudaGetSymbolAddress(scratch) failed on device %d: %s", dev, cudaGetErrorString(e));
  if (!ctx && (g_ctx_get(&ctx) != 0 || !ctx)) return fail(ENT_ERR_CUDA, "no current CUDA context on device %d", dev);
  g_na_cache.push_back(NaEntry{dev, ctx, static_cast<unsigned char*>(p)});
  *out = static_cast<unsigned char*>(p);
  return ENT_OK;
}

}  // namespace ent

using namespace ent;

extern "C" int ent_bfs_noalloc(const int64_t* beg_pos_dev, const int32_t* csr_dev, int64_t vert_count, int32_t src,
                               int32_t* depth_dev, void* stream) {
  clear_error();
  if (!beg_pos_dev || !csr_dev || !depth_dev) return fail(ENT_ERR_INVALID_ARG, "null device pointer");
  if (vert_count < 1) return fail(ENT_ERR_INVALID_ARG, "vert_count must be >= 1");
  if (vert_count > NOALLOC_MAX_VERTICES)
    return fail(ENT_ERR_INVALID_ARG,
                "vert_count %lld exceeds the no-allocation limit of %lld vertices (use ent_bfs_device instead)",
                (long long)vert_count, (long long)NOALLOC_MAX_VERTICES);
  if (src < 0 || src >= vert_count) return fail(ENT_ERR_INVALID_ARG, "source %d out of range [0,%lld)", src, (long long)vert_count);
  unsigned char* scratch = nullptr;
  int rc = na_scratch_for_current_device(&scratch);
  if (rc != ENT_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  int dev = 0, sms = 148, per_sm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  constexpr size_t smem = 2 * NA_SOLO_CAP * sizeof(int4);
  cudaError_t e = cudaFuncSetAttribute(k_na_run, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_na_run, NA_T, smem);
  if (e != cudaSuccess) return fail(ENT_ERR_CUDA, "kernel setup failed: %s", cudaGetErrorString(e));
  NaArgs a;
  a.visited = reinterpret_cast<uint32_t*>(scratch);
  a.queue[0] = reinterpret_cast<int32_t*>(scratch + NA_OFF_QUEUE);
  a.queue[1] = a.queue[0] + NOALLOC_MAX_VERTICES;
  a.ctl = reinterpret_cast<NaCtl*>(scratch + NA_OFF_CTL);
  a.off = beg_pos_dev;
  a.adj = csr_dev;
  a.depth = depth_dev;
  a.V = vert_count;
  a.src = src;
  e = cudaMemsetAsync(a.ctl, 0, sizeof(NaCtl), s);
  if (e != cudaSuccess) return fail(ENT_ERR_CUDA, "control reset failed: %s", cudaGetErrorString(e));
  // Every CTA must be resident (they wait on one another): as many as fit, fewer
  // for small graphs, whose barriers are then cheaper. Where part of the GPU is
  // set aside (MPS, a partition) the launch is refused and tried smaller.
  void* args[1] = {&a};
  int grid = (int)std::min<int64_t>((int64_t)sms * std::max(1, std::min(per_sm, 1)), (vert_count + 255) / 256);
  for (;; grid >>= 1) {
    e = cudaLaunchCooperativeKernel((const void*)k_na_run, dim3(grid), dim3(NA_T), args, smem, s);
    if (e != cudaErrorCooperativeLaunchTooLarge || grid <= 1) break;
    cudaGetLastError();
  }
  if (e != cudaSuccess) return fail(ENT_ERR_CUDA, "traversal launch failed: %s", cudaGetErrorString(e));
  g_kernel_launches++;
  int32_t err = 0;
  // 4-byte read of the status into a host variable (no allocation)
  e = cudaMemcpyAsync(&err, &a.ctl->err, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(ENT_ERR_CUDA, "traversal failed: %s", cudaGetErrorString(e));
  if (err == 1) return fail(ENT_ERR_TIMEOUT, "a wait between the traversal's CTAs ran out");
  if (err) return fail(ENT_ERR_INTERNAL, "level loop did not terminate");
  return ENT_OK;
}
