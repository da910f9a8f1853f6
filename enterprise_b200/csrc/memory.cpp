// Device memory from a pool, and host copies through page-locked staging.
//
// cudaMalloc and cudaFree map and unmap memory and wait for the device: 0.3 to
// 0.5 ms each at tens of MB, with outliers of tens of ms, and building a graph
// and traversing it once made 15 of each (R-MAT s18 edge list: 11 of 19 ms).
// dev_alloc takes memory from a pool of the library's own that keeps up to
// POOL_KEEP bytes of what was given back for the next allocation. Whatever is
// above goes back to the device at once, and all of it when ent_release_memory is
// called or an allocation, of this library or of another in the process, finds too
// little (the driver takes from pools what they do not use; measured with 160 MB
// free and 420 kept: 300 MB by cudaMalloc succeed). Blocks of POOL_MAX and more
// bypass it.
//
// Programs with CUDA contexts of their own (driver-API plug-ins) get memory from
// the device there, and page-locked memory made in the same context.
//
// A copy between the device and pageable host memory runs through the driver's
// own staging on one host thread (about 10 GB/s, first touch of fresh pages
// included). Here two page-locked chunks take turns: the DMA of one overlaps
// the copying of the other by several threads.
#include <algorithm>
#include <cuda_runtime.h>
#include <mutex>
#include <omp.h>
#include <string.h>
#include <vector>

#include "dev_graph.h"

namespace ent {
namespace {

constexpr uint64_t POOL_KEEP = 512ull << 20;  // per device
constexpr size_t CHUNK = 4 << 20;             // bytes per staging chunk
constexpr size_t STAGED_MIN = 1 << 20;        // shorter copies go to the driver
constexpr int COPY_THREADS = 8;
// Larger blocks come from the device and go back to it: the pool would keep none
// of them, and maps and unmaps them far more slowly (making R-MAT s22 58 ms at
// best and up to 750, 29 so; s24 246 and up to seconds, 116 so; from 32 MB on
// s20 10 -> 25).
constexpr size_t POOL_MAX = 256ull << 20;

struct DevicePool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;  // orders the pool's own allocations and frees
  uint64_t ctx = 0;               // the primary context it was made in
};
std::mutex g_mu;
std::vector<DevicePool> g_pools;      // by device
std::vector<void*> g_large;           // blocks that bypassed the pools
// What is kept belongs to the CUDA context it was made in and ends with it: it is
// used in that context only, by an id that no later context has again.
struct Chunks {
  uint64_t ctx = 0;
  char* idle[2];  // page-locked pairs of chunks not in use
  int n_idle = 0;
  int n = 0;      // ... and all of them
};
std::vector<Chunks> g_chunks;
constexpr int MAX_PAIRS = 2;          // 16 MB; further copies at the same time go to the driver

// Small page-locked blocks (a traversal's status words): a slot of an arena, for
// a call of cudaHostAlloc and cudaFreeHost each takes as long as a small graph's
// whole build. Arenas stay; their number follows the most slots in use at once.
constexpr size_t SLOT = 512, ARENA = 64 << 10;
struct Arena {
  uint64_t ctx;
  char* base;
  std::vector<char*> free;
};
std::vector<Arena> g_arenas;

// The current context's id (0: unknown), and whether it is its device's primary
// one. Only that one has a pool: memory of another context goes with it, and a
// pool's would stay.
struct Context {
  uint64_t id = 0;
  bool primary = true;
};
Context context() {
  typedef int (*GetCurrent)(void**);
  typedef int (*GetId)(void*, unsigned long long*);
  typedef int (*GetState)(int, unsigned*, int*);
  typedef int (*Retain)(void**, int);
  typedef int (*Release)(int);
  static const auto entry = [](const char* name) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint(name, &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return fn;
  };
  static const auto current = (GetCurrent)entry("cuCtxGetCurrent");
  static const auto id_of = (GetId)entry("cuCtxGetId");
  static const auto state = (GetState)entry("cuDevicePrimaryCtxGetState");
  static const auto retain = (Retain)entry("cuDevicePrimaryCtxRetain");
  static const auto release = (Release)entry("cuDevicePrimaryCtxRelease");
  static std::mutex mu;
  static std::vector<Context> known;
  Context c;
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (!current || !id_of || !state || !retain || !release) return c;
  if (current(&ctx) != 0) return c;
  if (!ctx && (cudaFree(nullptr) != cudaSuccess || current(&ctx) != 0 || !ctx)) return c;  // binds the primary one
  if (id_of(ctx, &id) != 0) return c;
  c.id = id + 1;
  std::lock_guard<std::mutex> lk(mu);
  for (const Context& k : known)
    if (k.id == c.id) return k;
  int dev = 0, active = 0;
  unsigned flags = 0;
  cudaGetDevice(&dev);
  void* p = nullptr;
  if (state(dev, &flags, &active) == 0 && active && retain(&p, dev) == 0) release(dev);
  c.primary = p == ctx;
  known.push_back(c);
  return c;
}

// The current device's pool; pool null where it cannot have one.
DevicePool device_pool() {
  const Context c = context();
  if (!c.primary) return {};
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_mu);
  if ((int)g_pools.size() <= dev) g_pools.resize(dev + 1);
  DevicePool& p = g_pools[dev];
  if (!p.stream || p.ctx != c.id) {
    p = DevicePool{};
    p.ctx = c.id;
    int ok = 0;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    uint64_t keep = POOL_KEEP;
    if (cudaDeviceGetAttribute(&ok, cudaDevAttrMemoryPoolsSupported, dev) != cudaSuccess ||
        cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess || !ok ||
        cudaMemPoolCreate(&p.pool, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
      cudaGetLastError();
      p.pool = nullptr;
    }
  }
  return p;
}

struct Staging {
  char* buf = nullptr;  // two chunks
  uint64_t ctx = 0;
  cudaEvent_t done[2] = {nullptr, nullptr};
  static Chunks& of(uint64_t ctx) {
    for (Chunks& c : g_chunks)
      if (c.ctx == ctx) return c;
    g_chunks.emplace_back();
    g_chunks.back().ctx = ctx;
    return g_chunks.back();
  }
  Staging() {
    ctx = context().id;
    {
      std::lock_guard<std::mutex> lk(g_mu);
      Chunks& c = of(ctx);
      if (c.n_idle > 0) {
        buf = c.idle[--c.n_idle];
      } else if (c.n < MAX_PAIRS) {
        if (cudaHostAlloc((void**)&buf, 2 * CHUNK, cudaHostAllocPortable) == cudaSuccess) {
          ++c.n;
        } else {
          buf = nullptr;
          cudaGetLastError();
        }
      }
    }
    for (cudaEvent_t& e : done)
      if (buf && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        e = nullptr;
        cudaGetLastError();
      }
  }
  bool ok() const { return buf && done[0] && done[1]; }
  ~Staging() {
    for (cudaEvent_t e : done)
      if (e) {
        cudaEventSynchronize(e);  // no DMA may still use the chunk
        cudaEventDestroy(e);
      }
    if (!buf) return;
    std::lock_guard<std::mutex> lk(g_mu);
    Chunks& c = of(ctx);
    c.idle[c.n_idle++] = buf;
  }
};

// memcpy by several threads (first touch of the destination's pages included).
void copy_host(char* dst, const char* src, size_t n) {
  const int t = (int)std::min<size_t>(std::min(COPY_THREADS, omp_get_max_threads()), n / (256 << 10) + 1);
  if (t <= 1) {
    memcpy(dst, src, n);
    return;
  }
#pragma omp parallel for num_threads(t) schedule(static)
  for (int i = 0; i < t; ++i) {
    const size_t a = n * i / t, b = n * (i + 1) / t;
    memcpy(dst + a, src + a, b - a);
  }
}

bool pageable(const void* host) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

}  // namespace

// Memory from the device itself, which dev_free gives back to it.
static cudaError_t alloc_large(void** out, size_t bytes) {
  const cudaError_t e = dev_malloc(out, bytes);
  if (e == cudaSuccess) {
    std::lock_guard<std::mutex> lk(g_mu);
    g_large.push_back(*out);
  }
  return e;
}

cudaError_t dev_alloc(void** out, size_t bytes) {
  *out = nullptr;
  bytes = std::max<size_t>(bytes, 1);
  if (bytes >= POOL_MAX) return alloc_large(out, bytes);
  const DevicePool p = device_pool();
  if (!p.pool) return alloc_large(out, bytes);
  cudaError_t e = cudaMallocFromPoolAsync(out, bytes, p.pool, p.stream);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    cudaMemPoolTrimTo(p.pool, 0);
    e = cudaMallocFromPoolAsync(out, bytes, p.pool, p.stream);
  }
  // usable on any stream once the pool's stream has reached it
  if (e == cudaSuccess) e = cudaStreamSynchronize(p.stream);
  if (e != cudaSuccess) *out = nullptr;
  return e;
}

cudaError_t dev_malloc(void** out, size_t bytes) {
  cudaError_t e = cudaMalloc(out, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  const DevicePool p = device_pool();
  if (p.pool) cudaMemPoolTrimTo(p.pool, 0);
  return cudaMalloc(out, bytes);
}

void dev_free(void* ptr) {
  if (!ptr) return;
  bool large = false;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    const auto it = std::find(g_large.begin(), g_large.end(), ptr);
    if ((large = it != g_large.end())) g_large.erase(it);
  }
  if (large) {
    cudaFree(ptr);
    return;
  }
  const DevicePool p = device_pool();
  if (p.pool) cudaFreeAsync(ptr, p.stream);
  else cudaFree(ptr);
}

void* host_slot(size_t bytes) {
  if (bytes > SLOT) return nullptr;
  const uint64_t ctx = context().id;
  std::lock_guard<std::mutex> lk(g_mu);
  Arena* a = nullptr;
  for (Arena& x : g_arenas)
    if (x.ctx == ctx && !x.free.empty()) a = &x;
  if (!a) {
    char* base = nullptr;
    if (cudaHostAlloc((void**)&base, ARENA, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    g_arenas.push_back({ctx, base, {}});
    a = &g_arenas.back();
    for (size_t at = 0; at < ARENA; at += SLOT) a->free.push_back(base + at);
  }
  char* p = a->free.back();
  a->free.pop_back();
  return p;
}

void host_slot_free(void* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_mu);
  for (auto a = g_arenas.rbegin(); a != g_arenas.rend(); ++a)  // an address may be a dead context's too: the latest
    if ((char*)p >= a->base && (char*)p < a->base + ARENA) {
      a->free.push_back((char*)p);
      return;
    }
}

cudaError_t to_device(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  if (bytes < STAGED_MIN || !pageable(src)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
  Staging st;
  if (!st.ok()) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
  cudaError_t e = cudaSuccess;
  for (size_t at = 0, k = 0; at < bytes && e == cudaSuccess; at += CHUNK, ++k) {
    const size_t n = std::min(CHUNK, bytes - at);
    char* buf = st.buf + (k & 1) * CHUNK;
    if (k >= 2) e = cudaEventSynchronize(st.done[k & 1]);
    if (e != cudaSuccess) break;
    copy_host(buf, (const char*)src + at, n);
    e = cudaMemcpyAsync((char*)dst + at, buf, n, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaEventRecord(st.done[k & 1], s);
  }
  return e;
}

cudaError_t rows_to_host(void* dst, const void* src, size_t width, size_t pitch, size_t rows, cudaStream_t s) {
  if (width == 0 || rows == 0) return cudaSuccess;
  const size_t bytes = width * rows;
  const auto direct = [&] {
    return pitch == width ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s)
                          : cudaMemcpy2DAsync(dst, width, src, pitch, width, rows, cudaMemcpyDeviceToHost, s);
  };
  // whole rows per chunk, or one run of bytes; other shapes go to the driver
  const bool flat = pitch == width;
  if (bytes < STAGED_MIN || (!flat && width > CHUNK) || !pageable(dst)) return direct();
  Staging st;
  if (!st.ok()) return direct();
  const size_t unit = flat ? 1 : width, per = flat ? CHUNK : CHUNK / width * width;
  struct Part {
    size_t at = 0, n = 0;
  } part[2];
  cudaError_t e = cudaSuccess;
  size_t at = 0;
  for (size_t k = 0;; ++k) {
    Part& p = part[k & 1];
    if (p.n) {  // the DMA of two turns ago: copy it out (the other chunk's is in flight)
      e = cudaEventSynchronize(st.done[k & 1]);
      if (e != cudaSuccess) break;
      copy_host((char*)dst + p.at, st.buf + (k & 1) * CHUNK, p.n);
      p.n = 0;
    }
    if (at < bytes) {
      const size_t n = std::min(per, bytes - at);
      char* buf = st.buf + (k & 1) * CHUNK;
      e = flat ? cudaMemcpyAsync(buf, (const char*)src + at, n, cudaMemcpyDeviceToHost, s)
               : cudaMemcpy2DAsync(buf, width, (const char*)src + at / unit * pitch, pitch, width, n / unit,
                                   cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaEventRecord(st.done[k & 1], s);
      if (e != cudaSuccess) break;
      p.at = at;
      p.n = n;
      at += n;
    } else if (!part[0].n && !part[1].n) {
      break;
    }
  }
  return e;
}

cudaError_t to_host(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  return rows_to_host(dst, src, bytes, bytes, 1, s);
}

}  // namespace ent

extern "C" int ent_release_memory(int32_t gpu) {
  using namespace ent;
  clear_error();
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || gpu < 0 || gpu >= n)
    return fail(ENT_ERR_INVALID_ARG, "no GPU %d (%d present)", gpu, n);
  cudaMemPool_t pool = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if ((size_t)gpu < g_pools.size()) pool = g_pools[gpu].pool;
  }
  if (pool) ENT_CUDA(cudaMemPoolTrimTo(pool, 0));
  return ENT_OK;
}
