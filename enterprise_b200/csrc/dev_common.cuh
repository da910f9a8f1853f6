// Device utilities shared by the traversal kernels: acquire/release accessors,
// warp/block scans and the single-pass decoupled look-back prefix sum
// (Merrill & Garland, "Single-pass Parallel Prefix Scan with Decoupled
// Look-back", NVIDIA TR 2016). The look-back replaces the reference's
// two-kernel Blelloch scan over 65,536 per-thread bin counts
// (scan.cuh:484-685, driven by insp_scan, scan.cuh:895-938).
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

namespace ent {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ void st_release(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_cg(const uint32_t* p) { return __ldcg(p); }
__device__ __forceinline__ void red_or(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Look-back status word: [63:34] epoch, [33:32] flag, [31:0] value.
constexpr unsigned long long LB_INVALID = 0, LB_AGG = 1, LB_PREFIX = 2;
__device__ __forceinline__ unsigned long long lb_pack(uint32_t epoch, unsigned long long flag, uint32_t value) {
  return ((unsigned long long)(epoch & 0x3fffffffu) << 34) | (flag << 32) | value;
}
__device__ __forceinline__ unsigned long long lb_flag(unsigned long long w, uint32_t epoch) {
  return ((uint32_t)(w >> 34) == (epoch & 0x3fffffffu)) ? ((w >> 32) & 3ull) : LB_INVALID;
}

// Spin limit for any wait in these kernels: a wait that exceeds it records
// an error bit and gives up, so a bug can never hang the GPU. An iteration
// (an acquire load, a load of the error word, a short sleep) takes about a
// microsecond, so a wait gives up after roughly a second; a predecessor
// tile is always held by a running CTA and publishes within microseconds.
constexpr int SPIN_LIMIT = 1 << 20;

// A crew: the CTAs of one ordinary launch that go from phase to phase of some
// work together. A CTA takes part from the phase after the one in which it
// started, and none is waited for that has not started. So the work begins as
// soon as one SM is free and grows onto the others as they come free, where a
// cooperative launch begins when all its CTAs fit at once. Beside a server with
// eight deep queries in flight, whose clusters hold some SMs for milliseconds at a
// time, an R-MAT s16 traversal took 5.7 ms when launched so and takes 81 us (66 on
// an idle GPU), s24 7.0 and 0.49 ms, and the server kept a third of its queries
// and keeps all. On an idle GPU the seats cost 0 to 3 us a launch: R-MAT s12 47.4 us
// a traversal (46.9 as a cooperative launch), s20 83.3 (81-84), s22 136 (133), s24, whose
// traversals have two such launches, 337 (328).
//
// Ranks are given in the order of starting. Rank 0 leads. It founds the crew with
// those that have started within a moment, nearly always the whole grid; from then
// on, before it arrives at the barrier that ends a phase, it admits those that
// have started since and leaves them the phase's state. They wait for that
// barrier too (without an arrival) and draw the same conclusions from it as
// everyone. While the size is the whole grid none of this costs anything.
//
// State is what every member knows about the phase; its `p` counts phases. Posts
// and sizes alternate between two places: the leader writes one again two
// barriers later, and those who read it have arrived at the barrier between.
constexpr int CREW_MAX = 256;  // CTAs of a launch at most
constexpr uint32_t CREW_FOUNDED = 1u << 31;
constexpr uint32_t CREW_DISMISSED = 1u << 30;  // more arrivals than any launch has
template <class State>
struct Crew {  // zeroed before the launch
  unsigned long long arrived;  // arrivals, all barriers of the launch together; << 32: members of the first phase
  uint32_t joined;    // CTAs that have started, and CREW_FOUNDED
  uint32_t closed;    // the work is over: CTAs that have not been admitted leave
  uint32_t size[2];   // members of a phase, by its parity
  struct {
    State state;
    uint32_t target, size;
  } post[2];
  uint32_t when[CREW_MAX];  // by rank: 1 + the post it was admitted with, or 0
};
struct CrewSeat {  // one CTA's, in shared memory
  uint32_t rank, size;  // of the phase that is running
  uint32_t target;      // arrivals at which its barrier opens
};

__device__ __forceinline__ uint32_t ld_acquire32(const uint32_t* p) {
  uint32_t x;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
  return x;
}
__device__ __forceinline__ void st_release32(uint32_t* p, uint32_t x) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(x) : "memory");
}

// One thread's wait until test() holds, bounded (`limit` polls of half a
// microsecond; one that runs out means a bug): false when it ran out here, or
// when *err says that another did.
template <class Test>
__device__ __forceinline__ bool crew_wait(int32_t* err, int limit, Test test) {
  for (int spins = 0;; ++spins) {
    if (test()) return true;
    if (spins > 64) __nanosleep(64);
    if (spins >= limit || ((spins & 63) == 63 && *(volatile int32_t*)err)) {
      *(volatile int32_t*)err = 1;
      return false;
    }
  }
}

// Thread 0, once a phase's barrier has opened: the next phase's size and target
// (s.p still counts the one that ended).
template <class State>
__device__ __forceinline__ void crew_next(Crew<State>* c, CrewSeat& seat, const State& s) {
  if (seat.size < gridDim.x) seat.size = __ldcg(&c->size[(s.p + 1) & 1]);
  seat.target += seat.size;
}

// Takes a seat: 0, there is nothing left to do; 1, a founder, whose own share
// begin(rank) of what comes before the first phase is done and visible, like that
// of the other founders (ranks from seat.size on have had none); 2, a member of
// the phase that begins, its state in s. advance(): thread 0's conclusions from an
// opened barrier, s.p included.
template <class State, class Begin, class F>
__device__ int crew_join(Crew<State>* c, int32_t* err, CrewSeat& seat, State& s, Begin begin, F advance) {
  __shared__ int s_in;
  if (threadIdx.x == 0) {
    const uint32_t ticket = atomicAdd(&c->joined, 1u);
    seat.rank = ticket & ~CREW_FOUNDED;
    s_in = ticket & CREW_FOUNDED ? 2 : 1;
    if (ticket == gridDim.x - 1) atomicAdd(&c->arrived, (unsigned long long)gridDim.x << 32);  // all are there
  }
  __syncthreads();
  const uint32_t rank = seat.rank;
  if (s_in == 1) {
    begin(rank);
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(&c->arrived, 1ull);
      uint32_t n = 0;  // founders, once known
      const auto all = [&] {
        const unsigned long long now = ld_acquire(&c->arrived);
        n = (uint32_t)(now >> 32);
        return n != 0 && (uint32_t)now >= n;
      };
      if (rank == 0) {  // the CTAs of an idle GPU start within a microsecond or two
        for (const long long t0 = clock64(); !all() && clock64() - t0 < 4096;) {
        }
        if (n == 0) {
          const uint32_t there = atomicOr(&c->joined, CREW_FOUNDED);
          if (there < gridDim.x) atomicAdd(&c->arrived, (unsigned long long)there << 32);
        }
      }
      const bool ok = crew_wait(err, SPIN_LIMIT * 4, all);
      __threadfence();
      seat.size = n;
      seat.target = 2 * n;
      s_in = ok;
    }
  } else if (threadIdx.x == 0) {
    uint32_t w = 0;
    // as long as a phase of the others lasts, and they may still be few
    bool in = crew_wait(err, SPIN_LIMIT * 64, [&] {
      w = ld_acquire32(&c->when[rank]);
      return w != 0 || ld_acquire32(&c->closed) != 0;
    });
    in = in && w != 0;
    if (in) {
      const auto& post = c->post[w - 1];
      s = post.state;
      seat.target = post.target;
      in = crew_wait(err, SPIN_LIMIT * 4, [&] { return (uint32_t)ld_acquire(&c->arrived) >= seat.target; });
      __threadfence();
      seat.size = post.size;
      seat.target += seat.size;
      if (in) advance();
    }
    s_in = in ? 2 : 0;
  }
  __syncthreads();
  return s_in;
}

// Ends a phase: every member's work of it is visible to all, and thread 0 has
// run advance(). False when a wait ran out anywhere, or when the leader dismissed
// the others; the CTA then leaves.
template <class State, class F>
__device__ bool crew_barrier(Crew<State>* c, int32_t* err, CrewSeat& seat, const State& s, F advance) {
  __shared__ int s_ok;
  __shared__ uint32_t s_joined;
  __syncthreads();
  if (seat.rank == 0 && seat.size < gridDim.x) {
    if (threadIdx.x == 0) {
      s_joined = *(volatile uint32_t*)&c->joined & ~CREW_FOUNDED;
      auto& post = c->post[s.p & 1];
      post.state = s;
      post.target = seat.target;
      post.size = s_joined;
      c->size[(s.p + 1) & 1] = s_joined;
      __threadfence();
    }
    __syncthreads();
    for (uint32_t r = seat.size + threadIdx.x; r < s_joined; r += blockDim.x)
      st_release32(&c->when[r], 1 + (s.p & 1));
  }
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&c->arrived, 1ull);
    const uint32_t target = seat.target;
    uint32_t now = 0;
    bool ok = crew_wait(err, SPIN_LIMIT * 4, [&] {
      now = (uint32_t)ld_acquire(&c->arrived);
      return now >= target;
    });
    __threadfence();
    ok = ok && now < CREW_DISMISSED;
    s_ok = ok;
    if (ok) {
      crew_next(c, seat, s);
      advance();
    }
  }
  __syncthreads();
  return s_ok != 0;
}

// Whether a phase of `work` row entries is worth waiting for more members (a CTA
// walks about one entry a nanosecond): a phase of its own then, in which the
// leader waits for them, up to a quarter of what they would save.
__device__ __forceinline__ bool crew_short(const CrewSeat& seat, int64_t work) {
  return work / seat.size - work / gridDim.x > 4096;
}
template <class State>
__device__ void crew_gather(Crew<State>* c, const CrewSeat& seat, int64_t work) {
  if (seat.rank != 0 || threadIdx.x != 0) return;
  const int64_t limit = min((work / seat.size - work / gridDim.x) / 2, (int64_t)1 << 30);  // cycles, two a nanosecond
  for (const long long t0 = clock64(); clock64() - t0 < limit && (*(volatile uint32_t*)&c->joined & ~CREW_FOUNDED) < gridDim.x;)
    __nanosleep(100);
}

// Sends every other member away, from the barrier of the running phase: their SMs
// are free for other work while the leader goes on alone (its thread 0 calls
// this). It meets nobody at a barrier again.
template <class State>
__device__ __forceinline__ void crew_dismiss(Crew<State>* c) {
  st_release32(&c->closed, 1u);
  atomicAdd(&c->arrived, (unsigned long long)CREW_DISMISSED);
}

// The leader's last word, whichever way it leaves.
template <class State>
__device__ __forceinline__ void crew_close(Crew<State>* c, const CrewSeat& seat) {
  if (seat.rank == 0 && threadIdx.x == 0) st_release32(&c->closed, 1u);
}

// Inclusive warp scan of K lanes' values (each lane holds v[k]).
template <int K>
__device__ __forceinline__ void warp_incl_scan(uint32_t (&v)[K]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      uint32_t y = __shfl_up_sync(FULL, v[k], o);
      if (lane >= o) v[k] += y;
    }
  }
}

// Exclusive block scan of K values per thread. smem: [32][K] words.
// Returns per-thread exclusive prefix in v and block totals in total.
template <int K>
__device__ __forceinline__ void block_excl_scan(uint32_t (&v)[K], uint32_t (&total)[K], uint32_t* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t orig[K];
#pragma unroll
  for (int k = 0; k < K; ++k) orig[k] = v[k];
  warp_incl_scan<K>(v);
  if (lane == 31) {
#pragma unroll
    for (int k = 0; k < K; ++k) smem[warp * K + k] = v[k];
  }
  __syncthreads();
  if (warp == 0) {
    uint32_t w[K];
#pragma unroll
    for (int k = 0; k < K; ++k) w[k] = lane < nw ? smem[lane * K + k] : 0u;
    warp_incl_scan<K>(w);
    if (lane < nw) {
#pragma unroll
      for (int k = 0; k < K; ++k) smem[lane * K + k] = w[k];
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    uint32_t before = warp > 0 ? smem[(warp - 1) * K + k] : 0u;
    total[k] = smem[(nw - 1) * K + k];
    v[k] = before + v[k] - orig[k];
  }
  __syncthreads();
}

// Decoupled look-back for tile `tile` with K independent chains. status is
// this segment's array [tiles][KS] (KS >= K). agg: tile aggregates (valid in
// every thread). On return excl[k] (valid in every thread) is the exclusive
// prefix of chain k. *err gets bit 1 set if a wait timed out.
template <int K, int KS>
__device__ void lookback(unsigned long long* status, uint32_t tile, uint32_t epoch, const uint32_t (&agg)[K],
                         uint32_t (&excl)[K], uint32_t* s_excl, int* err, bool hold_first = false) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    if (tile == 0) {
      if (!hold_first) {  // fault-injection hook: tile 0 never publishes, the others time out
#pragma unroll
        for (int k = 0; k < K; ++k) st_release(status + k, lb_pack(epoch, LB_PREFIX, agg[k]));
      }
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) st_release(status + (size_t)tile * KS + k, lb_pack(epoch, LB_AGG, agg[k]));
    }
  }
  if (tile == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) excl[k] = 0;
    return;
  }
  if (threadIdx.x < 32) {
#pragma unroll 1
    for (int k = 0; k < K; ++k) {
      uint32_t acc = 0;
      long pred = (long)tile - 1;
      int spins = 0;
      while (true) {
        long idx = pred - lane;
        unsigned long long w = idx >= 0 ? ld_acquire(status + (size_t)idx * KS + k) : lb_pack(epoch, LB_PREFIX, 0);
        unsigned long long f = idx >= 0 ? lb_flag(w, epoch) : LB_PREFIX;
        if (__any_sync(FULL, f == LB_INVALID)) {
          // give up (warp-uniformly) on timeout or once another tile timed out
          if (__any_sync(FULL, ++spins > SPIN_LIMIT || (*(volatile int*)err & 2))) {
            if (lane == 0) atomicOr(err, 2);
            break;
          }
          __nanosleep(32);
          continue;
        }
        unsigned pmask = __ballot_sync(FULL, f == LB_PREFIX);
        uint32_t val = (uint32_t)w;
        int stop = pmask ? (__ffs(pmask) - 1) : 31;
        uint32_t contrib = lane <= stop ? val : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(FULL, contrib, o);
        acc += contrib;
        if (pmask) break;
        pred -= 32;
      }
      if (lane == 0) {
        s_excl[k] = acc;
        st_release(status + (size_t)tile * KS + k, lb_pack(epoch, LB_PREFIX, acc + agg[k]));
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) excl[k] = s_excl[k];
  __syncthreads();
}

}  // namespace ent
