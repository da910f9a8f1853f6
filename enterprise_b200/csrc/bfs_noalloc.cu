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
// The whole traversal is one launch, whose CTAs go from level to level together
// (a Crew, dev_common.cuh; all waits bounded), so the host neither launches nor
// waits per level. While the frontier is small, the first CTA runs the levels
// alone with its frontier in shared memory and the others wait at the barrier;
// after NA_DISMISS such levels they leave, and if a larger frontier follows, the
// host, which waits for the end anyway, launches all of them once more.
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
constexpr int NA_SOLO = 1024;     // light frontier vertices up to which the leader runs alone
constexpr int NA_SOLO_M = 4096;   // ... and the sum of their degrees; it leaves above twice that
constexpr int NA_SOLO_CAP = 2048; // frontier entries it keeps in shared memory
constexpr int64_t NA_SHORT = 1 << 15;  // vertices up to which a traversal is short
constexpr int NA_DISMISS = 64;    // levels of a run after which it sends the others away

// A phase is one level of all members, a run of levels of the leader alone, a wait
// for more members, or the fills of CTAs that started late.
enum { NA_ALL, NA_ALONE, NA_DONE, NA_GATHER, NA_FILL };
struct NaState {
  int32_t p, kind, then, L;     // then: the kind of the phase after NA_GATHER and NA_FILL
  int32_t n_l, n_h, n_g, m_l;   // frontier: light, heavy, huge vertices; degree sum of the light
};

struct NaCtl {
  Crew<NaState> crew;
  int32_t err;        // a wait ran out
  int32_t again;      // the leader had sent the others away, and `resume` needs them
  int32_t level[2];   // per phase (mod 2): the level the leader reached running alone
  int32_t n[3][4];    // per phase (mod 3): light, heavy, huge frontier vertices; degree sum of the light
  // what a launch that resumes finds (all before it is zeroed for every launch)
  NaState resume;
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
  int32_t resume;  // goes on from ctl->resume
};

// Where the claimed vertices of a level go.
struct NaOut {
  int32_t* q;        // the next level's queue
  int32_t* n;        // its global counts
  int32_t* huge;     // its huge list
  // the leader alone: light vertices go to shared memory while they fit
  int4* s_q;
  int32_t* s_n;      // [3]: light, heavy, huge
};

// Claims the neighbours v[] (negative: none) of frontier vertices for `ln` and
// queues the won ones by degree. One warp, converged. my_m: the lane's sum of the
// light ones' degrees (the leader alone adds them beside the count instead: the sums
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

// The leader alone, from level L on: runs levels while all frontier vertices are
// light and fit and their rows are few, and leaves the next frontier in the queues,
// its counts in `out` and its level in *level. In a long run it sends the others
// away (returns true): a 700 x 700 grid is 1000 levels of one CTA, and a server's
// clusters got 190 queries a second done beside such calls, not 1400, while the
// waiting CTAs held the SMs. It
// walks about 1.2 entries a ns: without the bound on the rows a band graph of
// 1000-vertex levels took 147 us a level at degree 200 and 19 at 20, and 12 and 8
// so. The bound costs 2% where it never applies (700 x 700 grid 4.12 -> 4.20 ms,
// R-MAT s18 221 -> 225 us; sums at the level's end cost the grid 3%).
__device__ bool na_solo(const NaArgs& a, int L, int n, int4 (*s_q)[NA_SOLO_CAP], int32_t (*s_n)[4], int32_t* out,
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
  int run = 0;
  for (;; ++run) {
    if (run == NA_DISMISS && tid == 0) crew_dismiss(&a.ctl->crew);
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
    if (n == 0 || n > NA_SOLO_CAP || m > 2 * NA_SOLO_M || n2 || n3 || L > a.V) break;
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
  return run >= NA_DISMISS;
}

// The row entries, about, of a level of all members.
__device__ __forceinline__ int64_t na_work(const NaState& s) {
  return s.m_l + (int64_t)s.n_h * (4 * NA_HEAVY) + (int64_t)s.n_g * (2 * NA_HUGE);
}
// What follows for the phase to come from its frontier.
__device__ __forceinline__ void na_choose(NaState& s, const CrewSeat& seat) {
  if (s.n_l + s.n_h + s.n_g == 0) {
    s.kind = NA_DONE;
  } else if (s.n_l <= NA_SOLO && s.m_l <= NA_SOLO_M && s.n_h + s.n_g == 0) {
    s.kind = NA_ALONE;
  } else {
    s.kind = seat.size < gridDim.x && crew_short(seat, na_work(s)) ? NA_GATHER : NA_ALL;
    s.then = NA_ALL;
  }
}

// The whole traversal (the control block is zeroed before). Bound by the atomics and scattered reads of the entries on wide
// levels and by the barrier and the chain entry -> row -> claim on narrow ones.
// R-MAT s18: 0.22 ms; a 700 x 700 grid: 4.2 ms, 4.2 us a level (a launch and a
// host wait per level, a warp per vertex: 1.04 and 20.3 ms). 1024 threads and one
// CTA per SM beat two of 512 (grid 5.2 ms: the leader alone has more lanes); rows
// of one CTA from 256 entries beat 64 and 1024 (0.28 ms at s18), four entries
// per lane two (0.27 ms).
// Phase p reads the counts n[p % 3], fills n[(p + 1) % 3] and clears
// n[(p + 2) % 3], which no CTA reads any more once it is past the barrier
// before: a CTA that is late to read n[p % 3] still finds it unchanged.
__global__ void __launch_bounds__(NA_T, 1) k_na_run(NaArgs a) {
  extern __shared__ int4 s_dyn[];
  int4(*s_q)[NA_SOLO_CAP] = reinterpret_cast<int4(*)[NA_SOLO_CAP]>(s_dyn);
  __shared__ int32_t s_n[2][4];
  __shared__ unsigned s_m;
  __shared__ NaState s_st;
  __shared__ CrewSeat s_seat;
  if (threadIdx.x == 0) s_m = 0;
  NaCtl* c = a.ctl;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NWARP = NA_T / 32;
  const auto advance = [&] {  // what every member concludes from an opened barrier
    NaState& s = s_st;
    if (s.kind >= NA_GATHER) {
      s.p += 1;
      s.kind = s.then;
      return;
    }
    const int32_t* cnt = c->n[(s.p + 1) % 3];
    s.n_l = __ldcg(cnt);
    s.n_h = __ldcg(cnt + 1);
    s.n_g = min(__ldcg(cnt + 2), NA_HUGE_CAP);
    s.m_l = __ldcg(cnt + 3);
    s.L = s.kind == NA_ALONE ? __ldcg(&c->level[s.p & 1]) : s.L + 1;
    s.p += 1;
    na_choose(s, s_seat);
  };
  const auto fill = [&](uint32_t share) {  // one CTA's share of the fills
    if (a.resume) return;
    const int64_t tid = (int64_t)share * NA_T + threadIdx.x, nth = (int64_t)gridDim.x * NA_T;
    const int64_t W = (a.V + 31) >> 5;
    for (int64_t i = tid; i < W; i += nth) a.visited[i] = i == (a.src >> 5) ? 1u << (a.src & 31) : 0u;
    for (int64_t i = tid; i < a.V; i += nth) a.depth[i] = i == a.src ? 0 : -1;
  };
  const int in = crew_join(&c->crew, &c->err, s_seat, s_st, fill, advance);
  if (!in) return;
  const int rank = s_seat.rank;
  if (in == 1 && threadIdx.x == 0) {
    const int64_t d = a.off[a.src + 1] - a.off[a.src];
    NaState s = {};
    if (a.resume) {
      s = c->resume;
      s.p = 0;
    } else {
      s.n_l = d > 0 && d < NA_HEAVY;
      s.n_h = d >= NA_HEAVY;
      s.m_l = s.n_l ? (int32_t)d : 0;
      if (rank == 0) {
        if (s.n_l) a.queue[0][0] = a.src;
        if (s.n_h) a.queue[0][NOALLOC_MAX_VERTICES - 1] = a.src;
      }
    }
    na_choose(s, s_seat);
    if (s_seat.size < gridDim.x && !a.resume) {  // some shares are nobody's
      if (s.kind != NA_GATHER) s.then = s.kind;
      s.kind = NA_FILL;
    }
    s_st = s;
  }
  __syncthreads();
  for (;;) {
    const NaState& s = s_st;  // thread 0 changes it inside the barrier only
    if (s.kind == NA_DONE) break;
    if (s.L > a.V) {  // more levels than vertices
      if (rank == 0 && threadIdx.x == 0) c->err = 2;
      break;
    }
    const int L = s.L;
    int32_t* next = c->n[(s.p + 1) % 3];
    if (rank == 0 && threadIdx.x < 4) c->n[(s.p + 2) % 3][threadIdx.x] = 0;
    if (s.kind == NA_GATHER) {
      crew_gather(&c->crew, s_seat, na_work(s));
    } else if (s.kind == NA_FILL) {
      for (uint32_t i = s_seat.size + rank; i < gridDim.x; i += s_seat.size) fill(i);
    } else if (s.kind == NA_ALONE) {
      if (rank == 0 && na_solo(a, L, s.n_l, s_q, s_n, next, &c->level[s.p & 1])) {
        // alone from here: the end, or the host launches all of them again
        if (threadIdx.x == 0) {
          advance();
          if (s_st.kind != NA_DONE) {
            c->resume = s_st;
            c->again = 1;
          }
          if (s_st.L > a.V) c->err = 2;
        }
        return;
      }
    } else {
      const int32_t* q = a.queue[L & 1];
      const NaOut o{a.queue[(L + 1) & 1], next, c->huge[(L + 1) & 1], nullptr, nullptr};
      const int64_t gw = (int64_t)rank * NWARP + warp, nw = (int64_t)s_seat.size * NWARP;
      unsigned my_m = 0;
      for (int i = 0; i < s.n_g; ++i) {  // rows shared by all CTAs
        const int u = __ldcg(c->huge[L & 1] + i);
        const int64_t beg = a.off[u], end = a.off[u + 1];
        na_slice(a, beg + gw * 32 * NA_ILP, nw * 32 * NA_ILP, end, L + 1, o, my_m);
      }
      for (int i = rank; i < s.n_h; i += s_seat.size) {  // rows of one CTA
        const int u = __ldcg(q + NOALLOC_MAX_VERTICES - 1 - i);
        const int64_t beg = a.off[u], end = a.off[u + 1];
        na_slice(a, beg + warp * 32 * NA_ILP, NWARP * 32 * NA_ILP, end, L + 1, o, my_m);
      }
      // up to 32 light rows per warp, spread over all warps
      const int n_l = s.n_l;
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
    }
    if (!crew_barrier(&c->crew, &c->err, s_seat, s_st, advance)) break;
  }
  crew_close(&c->crew, s_seat);
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
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  constexpr size_t smem = 2 * NA_SOLO_CAP * sizeof(int4);
  cudaError_t e = cudaFuncSetAttribute(k_na_run, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
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
  a.resume = 0;
  // one CTA per SM, fewer for small graphs, whose barriers are then cheaper
  const int grid = (int)std::min<int64_t>(std::min(sms, CREW_MAX), (vert_count + 255) / 256);
  int32_t state[2] = {0, 0};  // err, again
  do {
    e = cudaMemsetAsync(a.ctl, 0, offsetof(NaCtl, resume), s);
    if (e != cudaSuccess) return fail(ENT_ERR_CUDA, "control reset failed: %s", cudaGetErrorString(e));
    k_na_run<<<grid, NA_T, smem, s>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(ENT_ERR_CUDA, "traversal launch failed: %s", cudaGetErrorString(e));
    g_kernel_launches++;
    // 8-byte read of the status into a host variable (no allocation). On the legacy
    // stream a pageable copy that has to wait for a kernel keeps other threads
    // from launching theirs (a server beside 4 ms traversals: 160 queries a second
    // instead of 1400): there the end is waited for first, except on small graphs,
    // whose traversals are short and would take 8 us of 70 more.
    if ((!s || s == cudaStreamLegacy) && vert_count > NA_SHORT) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(state, &a.ctl->err, sizeof(state), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(ENT_ERR_CUDA, "traversal failed: %s", cudaGetErrorString(e));
    a.resume = 1;
  } while (state[1] && !state[0]);
  const int32_t err = state[0];
  if (err == 1) return fail(ENT_ERR_TIMEOUT, "a wait between the traversal's CTAs ran out");
  if (err) return fail(ENT_ERR_INTERNAL, "level loop did not terminate");
  return ENT_OK;
}
