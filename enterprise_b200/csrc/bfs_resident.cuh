// The whole single-source traversal as one kernel, for graphs that the level
// kernels of bfs_single.cu cannot keep busy (included there).
//
// On a small graph the level loop costs more than the levels: a level is three
// kernel nodes and half a while-node iteration, about 20 us whatever it does
// (R-MAT s12: 124 us a traversal, 16 us of them in kernels; s20: 138 us). Here
// the CTAs stay resident and go from level to level together (a Crew,
// dev_common.cuh), and each takes the level's decision by itself from the counts
// that the barrier published, so no level ends in one CTA's chain.
//
// A phase is one of
//   * a top-down level: a warp takes up to 32 light rows together, heavy rows
//     get as many warps each as there are for them; a claim queues its vertex
//     by degree and sets its frontier bit, so that either direction can follow;
//   * a bottom-up level: a warp per status word, as in k_expand;
//   * a queue build, from the frontier bitmap, where a bottom-up level hands
//     over to top-down;
//   * a run of small top-down levels by the leader alone, its frontier in shared
//     memory (counted as small-frontier levels), while the others wait;
//   * where other work holds some SMs, a wait for more members before a long phase,
//     or the fills of CTAs that had not started.
// Phase p reads the counts n[p % 3] and acc[p % 3], fills those of p + 1 and
// clears those of p + 2, which no CTA reads any more once it is past the
// barrier before; frontier bitmaps rotate the same way per level. All waits
// are bounded: one that runs out sets the error word and every CTA leaves; the
// traversal's status, an error from its start on, is then never cleared.
//
// On large graphs the bottom-up levels are most of the time and want k_expand's
// occupancy, twice this kernel's (R-MAT s24 0.355 -> 0.31 ms, ER 2^24 d32 2.43 ->
// 1.69). The traversal then runs in parts: a head up to the first bottom-up
// level, R_BU_LEVELS kernels of one level each (those not
// needed leave at once; the last CTA of each takes the decision), and a tail
// for whatever is left.
//
// With parents (PAR) a claim also stores the caller's id of the vertex in whose row
// it was found, and a bottom-up find its neighbour's: instantiations of their own,
// so that traversals without them keep their registers.
//
// Not here: hub tables, runs with the small-frontier mode off, parents of small
// graphs, and graphs of many small levels (meshes, bands) stay with the level
// kernels.
#pragma once

constexpr int RT = 1024;          // threads per CTA, one per SM (64 registers a thread)
constexpr int RW = RT / 32;
constexpr int R_ILP = 4;          // row entries a lane has in flight together
constexpr int R_BW_WORDS = 4;     // bottom-up: words a warp up to which it takes them two by two
constexpr int R_HEAVY = 256;      // degree from which warps take a row alone, or share it
constexpr int R_HUGE = 16384;     // ... and from which at least R_SHARE warps do
constexpr int R_SHARE = 32;
constexpr int R_SOLO = 2048;      // frontier up to which the leader starts to run alone
constexpr int R_SOLO_M = 16384;   // ... and its degree sum; it leaves above twice that
constexpr int R_SOLO_CAP = 4096;  // frontier entries it keeps in shared memory
constexpr int R_SOLO_LEVELS = 4096;  // levels it runs before it meets the others again

enum { RK_TD, RK_BU, RK_QUEUE, RK_SOLO, RK_DONE, RK_GATHER, RK_FILL };

// What every member knows about the phase to come (thread 0 keeps it current).
struct ResState {
  int32_t kind, L, f, p;      // f: fb index of the frontier
  int32_t then;               // RK_GATHER, RK_FILL: the kind of the phase after
  int32_t n_l, n_h, n_g;
  int32_t td_levels, bu_levels, narrow_levels, mid_levels, err;
  int64_t n_f, m_f, n_vis, m_vis;
};

// Frontiers, by degree sum, that the cluster of k_narrow takes in less time.
constexpr int64_t RES_MID_MIN = 64, RES_MID_MAX = 40000;
__device__ __forceinline__ int res_mid(int64_t m_f) { return m_f >= RES_MID_MIN && m_f <= RES_MID_MAX; }


struct ResCtl {
  Crew<ResState> crew[2];  // of the head (or the whole), and of the tail
  int32_t err;       // a wait ran out
  uint32_t finished; // CTAs of a bottom-up kernel that are done
  ResState state;    // between the kernels of a traversal in parts
  int32_t n[3][4];   // light, heavy, huge frontier vertices of a phase
  unsigned long long acc[3][2];  // vertices and degree sum that a phase found
  struct {
    int64_t n_f, m_f, n_vis, m_vis;
    int32_t level, mid_levels;
  } solo[2];         // where the leader got to alone, by phase parity
};

struct ResArgs {
  ResCtl* rc;
  uint32_t* fb[3];
  int32_t* queue[2];  // light vertices from the front, heavy ones from the back (V entries)
  int32_t* huge[2];
  int32_t* parent;    // PAR
};

__device__ __forceinline__ int64_t ldcg64(const void* p) {
  return (int64_t)__ldcg(reinterpret_cast<const long long*>(p));
}

// The kind of a top-down level over the queued frontier.
__device__ __forceinline__ int res_td_kind(const LevelArgs& a, const ResState& s) {
  return s.n_h + s.n_g == 0 && s.n_l <= R_SOLO && s.n_f <= a.narrow_f && s.m_f <= min(a.narrow_m, (int64_t)R_SOLO_M)
             ? RK_SOLO
             : RK_TD;
}

// After phase s.p (thread 0): the next one, from the counts the barrier
// published. The rules are k_inspect's.
__device__ void res_advance(const LevelArgs& a, const ResArgs& r, ResState& s) {
  const ResCtl* c = r.rc;
  const int q = (s.p + 1) % 3;
  const int kind = s.kind;
  const int32_t n_l = __ldcg(&c->n[q][0]), n_h = __ldcg(&c->n[q][1]), n_g = __ldcg(&c->n[q][2]);
  int64_t n_next = 0, m_next = 0;
  if (kind == RK_SOLO) {
    const auto* so = &c->solo[s.p & 1];
    const int L = __ldcg(&so->level);
    n_next = ldcg64(&so->n_f);
    m_next = ldcg64(&so->m_f);
    s.n_vis = ldcg64(&so->n_vis);
    s.m_vis = ldcg64(&so->m_vis);
    s.td_levels += L - s.L;
    s.narrow_levels += L - s.L;
    s.mid_levels += __ldcg(&so->mid_levels);
    s.L = L;
  } else if (kind != RK_QUEUE) {
    n_next = ldcg64(&c->acc[q][0]);
    m_next = ldcg64(&c->acc[q][1]);
    s.n_vis += n_next;
    s.m_vis += m_next;
    s.L += 1;
    s.mid_levels += res_mid(s.m_f);
    if (kind == RK_TD) s.td_levels += 1;
    else s.bu_levels += 1;
  }
  s.p += 1;
  s.n_l = n_l;
  s.n_h = n_h;
  s.n_g = n_g;
  if (kind == RK_QUEUE) {
    s.kind = res_td_kind(a, s);
    return;
  }
  const int64_t n_before = s.n_f;
  s.f = (s.f + 1) % 3;
  s.n_f = n_next;
  s.m_f = m_next;
  bool done = n_next == 0;
  if (s.L >= a.max_levels && !done) {
    s.err |= 4;
    done = true;
  }
  if (s.n_vis > a.V) {
    s.err |= 8;
    done = true;
  }
  if (done) {
    s.kind = RK_DONE;
    return;
  }
  if (kind == RK_BU) {
    const bool to_td = a.policy == ENT_POLICY_BEAMER && (double)n_next < (double)a.V / a.beta && n_next < n_before;
    s.kind = to_td ? RK_QUEUE : RK_BU;
    return;
  }
  bool bu = a.policy == ENT_POLICY_BU_ONLY;
  if (a.policy == ENT_POLICY_BEAMER) bu = (double)m_next > (double)(a.E - s.m_vis) / a.alpha;
  if (a.policy == ENT_POLICY_REFERENCE) bu = (double)m_next >= a.ref_ratio * (double)a.E;
  s.kind = bu ? RK_BU : res_td_kind(a, s);
}

// Where the claims of a top-down phase go, and what they add up to.
struct ResOut {
  uint32_t* fb;      // the next frontier's bits (not while the leader runs alone)
  int32_t* q;
  int32_t* huge;
  int32_t* n;        // counts: global, or the leader's own in shared memory
  int4* s_q;         // the leader alone: entries in shared memory while they fit
  int32_t* parent;   // PAR
};

// Where vertices queue by degree: 0 light, 1 heavy, 2 huge.
__device__ __forceinline__ int res_class(int d) { return d < R_HEAVY ? 0 : (d < R_HUGE ? 1 : 2); }

// Queues vertices of a converged warp, N per lane (cls < 0: none): one atomic
// per class for all of them (one each for the heavy ones took 40 us on R-MAT
// s24's second level, whose 23k finds are mostly hubs). put(i, at) stores the
// lane's i-th light vertex at position `at`.
template <int N, class Put>
__device__ __forceinline__ void res_queue_up(const LevelArgs& a, const ResOut& o, const int (&v)[N],
                                             const int (&cls)[N], Put put) {
  const int lane = threadIdx.x & 31;
  int cnt[3] = {0, 0, 0};
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int c = 0; c < 3; ++c) cnt[c] += __popc(__ballot_sync(FULL, cls[i] == c));
  if (cnt[0] + cnt[1] + cnt[2] == 0) return;
  const int mine = lane == 0 ? cnt[0] : (lane == 1 ? cnt[1] : (lane == 2 ? cnt[2] : 0));
  int at = 0;
  if (mine) at = atomicAdd(o.n + lane, mine);
  int base[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) base[c] = __shfl_sync(FULL, at, c);
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const unsigned m = __ballot_sync(FULL, cls[i] == c);
      const int pos = base[c] + __popc(m & lanemask_lt());
      base[c] += __popc(m);
      if (cls[i] == c) {
        if (c == 0) put(i, pos);
        else if (c == 1) o.q[a.V - 1 - pos] = v[i];
        else o.huge[pos] = v[i];
      }
    }
}

// from (PAR): the caller's id of the vertex in whose row each v was found.
template <class DT, bool SOLO, bool PAR>
__device__ __forceinline__ void res_claim(const LevelArgs& a, const int (&v)[R_ILP], const int (&from)[R_ILP], int ln,
                                          DT* depth, const ResOut& o, unsigned& my_n, unsigned long long& my_m) {
  bool open[R_ILP], mine[R_ILP];
  int64_t st[R_ILP];
  int d[R_ILP], id[R_ILP];
#pragma unroll
  for (int i = 0; i < R_ILP; ++i)
    open[i] = v[i] >= 0 && (SOLO || !((__ldca(a.vis + (v[i] >> 5)) >> (v[i] & 31)) & 1u));
#pragma unroll
  for (int i = 0; i < R_ILP; ++i) {
    mine[i] = false;
    st[i] = 0;
    d[i] = id[i] = 0;
    if (open[i]) {  // row and degree, or degree and caller id, are read beside the claim
      if (SOLO) {
        st[i] = __ldg(a.off + v[i]);
        d[i] = (int)(__ldg(a.off + v[i] + 1) - st[i]);
      } else {
        d[i] = __ldg(a.deg + v[i]);
      }
      if (!SOLO || PAR) id[i] = out_id(a, v[i]);
      const uint32_t b = 1u << (v[i] & 31);
      mine[i] = !(atomicOr(a.vis + (v[i] >> 5), b) & b);
    }
  }
  int cls[R_ILP];
#pragma unroll
  for (int i = 0; i < R_ILP; ++i) {
    cls[i] = mine[i] ? res_class(d[i]) : -1;
    if (mine[i]) {
      if (!SOLO) {  // alone, depths and bits are written later: off the level's chain
        depth[id[i]] = (DT)ln;
        red_or(o.fb + (v[i] >> 5), 1u << (v[i] & 31));
      }
      if (PAR) o.parent[id[i]] = from[i];
      my_n += 1;
      my_m += (unsigned)d[i];
    }
  }
  res_queue_up<R_ILP>(a, o, v, cls, [&](int i, int at) {
    if (SOLO && at < R_SOLO_CAP)
      o.s_q[at] = make_int4(v[i], d[i], (int)(uint32_t)st[i], (int)(uint32_t)((uint64_t)st[i] >> 32));
    else
      o.q[at] = v[i];
  });
}

// The concatenated rows of a warp's light vertices (lane: d entries from st, of
// the vertex with the caller's id `own`).
template <class DT, bool SOLO, bool PAR>
__device__ __forceinline__ void res_rows(const LevelArgs& a, int d, int64_t st, int own, int ln, DT* depth,
                                         const ResOut& o, unsigned& my_n, unsigned long long& my_m) {
  const int lane = threadIdx.x & 31;
  int incl = d;
#pragma unroll
  for (int ofs = 1; ofs < 32; ofs <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, ofs);
    if (lane >= ofs) incl += y;
  }
  const int total = __shfl_sync(FULL, incl, 31), excl = incl - d;
  for (int r0 = 0; r0 < total; r0 += 32 * R_ILP) {
    int v[R_ILP], from[R_ILP];
#pragma unroll
    for (int i = 0; i < R_ILP; ++i) {
      v[i] = from[i] = -1;
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
        if (PAR) from[i] = __shfl_sync(FULL, own, j);
        if (k < total) v[i] = __ldg(a.adj + sj + (k - ej));
      }
    }
    res_claim<DT, SOLO, PAR>(a, v, from, ln, depth, o, my_n, my_m);
  }
}

// Entries first, first + step, ... of one long row, 32 * R_ILP per warp and turn.
template <class DT, bool PAR>
__device__ __forceinline__ void res_slice(const LevelArgs& a, int64_t first, int64_t step, int64_t end, int own,
                                          int ln, DT* depth, const ResOut& o, unsigned& my_n,
                                          unsigned long long& my_m) {
  const int lane = threadIdx.x & 31;
  for (int64_t e0 = first; e0 < end; e0 += step) {
    int v[R_ILP], from[R_ILP];
#pragma unroll
    for (int i = 0; i < R_ILP; ++i) {
      const int64_t e = e0 + 32 * i + lane;
      v[i] = e < end ? __ldg(a.adj + e) : -1;
      from[i] = own;
    }
    res_claim<DT, false, PAR>(a, v, from, ln, depth, o, my_n, my_m);
  }
}

template <class DT, bool PAR>
__device__ void res_td(const LevelArgs& a, const ResArgs& r, const ResState& s, const CrewSeat& seat, DT* depth,
                       const ResOut& o, unsigned& my_n, unsigned long long& my_m) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t* q = r.queue[s.L & 1];
  const int ln = s.L + 1;
  const int64_t gw = (int64_t)seat.rank * RW + warp, nw = (int64_t)seat.size * RW;
  // Long rows: `share` warps each, in turn over the rows. A CTA per row left
  // R-MAT s24's second level (four rows of 24k entries in all) at 60 us and
  // spent 2.1 ms on s22 top-down throughout; a list of equal chunks is as fast
  // there but costs 100 us to make on levels whose next one is bottom-up.
  const auto long_rows = [&](int n, int64_t share, auto row) {
    for (int64_t k = gw; k < n * share; k += nw) {
      const int u = row((int)(k % n));
      const int64_t end = a.off[u + 1];
      res_slice<DT, PAR>(a, a.off[u] + k / n * (32 * R_ILP), share * (32 * R_ILP), end, PAR ? out_id(a, u) : -1, ln,
                         depth, o, my_n, my_m);
    }
  };
  if (s.n_g) long_rows(s.n_g, max((int64_t)R_SHARE, nw / s.n_g), [&](int i) { return __ldcg(r.huge[s.L & 1] + i); });
  if (s.n_h) long_rows(s.n_h, max((int64_t)1, nw / s.n_h), [&](int i) { return __ldcg(q + a.V - 1 - i); });
  // up to 32 light rows per warp, spread over all warps
  const int k = (int)min((int64_t)32, (s.n_l + nw - 1) / nw);
  for (int64_t first = gw * k; first < s.n_l; first += nw * k) {
    int d = 0, own = -1;
    int64_t st = 0;
    if (lane < k && first + lane < s.n_l) {
      const int u = __ldcg(q + first + lane);
      st = a.off[u];
      d = a.deg[u];
      if (PAR) own = out_id(a, u);
    }
    res_rows<DT, false, PAR>(a, d, st, own, ln, depth, o, my_n, my_m);
  }
}

// One bottom-up level over the words of vertices that have rows (bu_expand
// with nothing to list), BW words of a warp in flight together, and ILP row
// entries of each vertex per step.
template <class DT, bool PAR, int BW, int ILP>
__device__ void res_bu_words(const LevelArgs& a, const ResArgs& r, const ResState& s, const CrewSeat& seat, DT* depth,
                             unsigned& my_n, unsigned long long& my_m) {
  const uint32_t* fbc = r.fb[s.f];
  uint32_t* fbn = r.fb[(s.f + 1) % 3];
  // read through L1: the barrier before this phase made it current
  const auto is_front = [&](int u) { return (__ldca(fbc + (u >> 5)) >> (u & 31)) & 1u; };
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gw = seat.rank * RW + warp, nw = seat.size * RW;
  const int W = (int)((a.n_active + 31) >> 5);  // below 2^26: ids are int32
  // BW words at a time through every stage together: a CTA of 64-register
  // threads holds half the warps of k_expand, so each has to keep more reads in
  // flight.
  for (int w0 = gw; w0 < W; w0 += BW * nw) {
    uint32_t vis[BW], mask[BW];
    int4 ld[BW];
    int d[BW], id[BW];
    bool todo[BW];  // still to be found
    bool found[BW];
    [[maybe_unused]] int by[BW];  // the neighbour that found it
#pragma unroll
    for (int t = 0; t < BW; ++t) {
      const int wi = w0 + t * nw;
      vis[t] = wi < W ? __ldcg(a.vis + wi) : 0u;
      mask[t] = wi < W ? a.active[wi] & ~vis[t] : 0u;
    }
#pragma unroll
    for (int t = 0; t < BW; ++t) {
      ld[t] = make_int4(-1, -1, -1, -1);
      d[t] = id[t] = 0;
      todo[t] = (mask[t] >> lane) & 1u;
      if (todo[t]) {
        const int v = (w0 + t * nw) * 32 + lane;
        ld[t] = __ldcs(a.lead + v);
        d[t] = __ldcs(a.deg + v);
        id[t] = a.perm ? __ldcs(a.perm + v) : v;
      }
    }
#pragma unroll
    for (int t = 0; t < BW; ++t) {
      found[t] = todo[t] && is_front(ld[t].x);
      todo[t] &= !found[t];
      by[t] = ld[t].x;
    }
#pragma unroll
    for (int t = 0; t < BW; ++t)
      if (todo[t] && d[t] > 1) {
        const bool fy = is_front(ld[t].y), fz = ld[t].z >= 0 && is_front(ld[t].z);
        found[t] = fy | fz | (ld[t].w >= 0 && is_front(ld[t].w));
        todo[t] = !found[t];
        by[t] = fy ? ld[t].y : (fz ? ld[t].z : ld[t].w);
      }
    uint32_t e0[BW];
#pragma unroll
    for (int t = 0; t < BW; ++t) {
      todo[t] &= d[t] > 4;  // shorter rows have been looked through
      e0[t] = 0;
      if (todo[t]) e0[t] = (uint32_t)__ldcs(a.off + (w0 + t * nw) * 32 + lane);
    }
    // light rows: ILP entries of each word per step
    for (int k = 4;; k += ILP) {
      bool more = false;
      int u[BW][ILP];
#pragma unroll
      for (int t = 0; t < BW; ++t) {
        const bool go = todo[t] && d[t] < a.small_max && k < d[t];
        more |= go;
#pragma unroll
        for (int i = 0; i < ILP; ++i) u[t][i] = go && k + i < d[t] ? __ldg(a.adj + e0[t] + k + i) : -1;
      }
      if (!more) break;
#pragma unroll
      for (int t = 0; t < BW; ++t) {
        bool f = false;
#pragma unroll
        for (int i = 0; i < ILP; ++i) {
          const bool fi = u[t][i] >= 0 && is_front(u[t][i]);
          f |= fi;
          if (PAR && fi) by[t] = u[t][i];
        }
        if (f) found[t] = true, todo[t] = false;
      }
    }
    // Heavy rows: the warp together, four rows at a time while there are four.
    // In the order by degree whole words hold them, and a row at a time took 32
    // trips for rows just above small_max (ER 2^19, mean degree 40: 145 -> 100 us a
    // traversal, 29: 216 -> 184).
#pragma unroll
    for (int t = 0; t < BW; ++t) {
      unsigned heavy = __ballot_sync(FULL, todo[t] && d[t] >= a.small_max);
      while (__popc(heavy) >= 4) {  // four rows at a time, eight lanes each
        const unsigned h1 = heavy & (heavy - 1), h2 = h1 & (h1 - 1), h3 = h2 & (h2 - 1);
        const int sub = lane >> 3;
        const int j = __ffs(sub == 0 ? heavy : (sub == 1 ? h1 : (sub == 2 ? h2 : h3))) - 1;
        heavy = h3 & (h3 - 1);
        const uint32_t beg = __shfl_sync(FULL, e0[t], j);
        const int n = __shfl_sync(FULL, d[t], j);
        bool hit = false;
        int hit_by = -1;  // PAR
        for (int b0 = lane & 7;; b0 += 32) {
          int u[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) u[i] = !hit && b0 + 8 * i < n ? __ldg(a.adj + beg + b0 + 8 * i) : -1;
          bool f = false;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const bool fi = u[i] >= 0 && is_front(u[i]);
            f |= fi;
            if (PAR && fi) u[0] = u[i];
          }
          const unsigned any = __ballot_sync(FULL, f);
          const unsigned hits = (any >> (8 * sub)) & 0xFFu;  // none once the row is found
          if (PAR && any) {
            const int x = __shfl_sync(FULL, u[0], hits ? 8 * sub + __ffs(hits) - 1 : lane);
            if (hits) hit_by = x;
          }
          hit |= hits != 0;
          if (__all_sync(FULL, hit || b0 + 32 - (lane & 7) >= n)) break;
        }
        const unsigned rows = __reduce_or_sync(FULL, hit ? 1u << j : 0u);
        if (rows >> lane & 1u) found[t] = true;
        if (PAR && rows)
#pragma unroll
          for (int r4 = 0; r4 < 4; ++r4) {
            const int row = __shfl_sync(FULL, hit ? j : -1, 8 * r4), x = __shfl_sync(FULL, hit_by, 8 * r4);
            if (lane == row) by[t] = x;
          }
      }
      while (heavy) {
        const int j = __ffs(heavy) - 1;
        heavy &= heavy - 1;
        const uint32_t beg = __shfl_sync(FULL, e0[t], j);
        const int n = __shfl_sync(FULL, d[t], j);
        bool hit = false;
        for (int b0 = 0; b0 < n && !hit; b0 += 64) {
          const int e = b0 + lane;
          const int u0 = e < n ? __ldg(a.adj + beg + e) : -1, u1 = e + 32 < n ? __ldg(a.adj + beg + e + 32) : -1;
          const bool f0 = u0 >= 0 && is_front(u0), f1 = u1 >= 0 && is_front(u1);
          const unsigned hits = __ballot_sync(FULL, f0 || f1);
          hit = hits != 0;
          if (PAR && hit) {
            const int x = __shfl_sync(FULL, f0 ? u0 : u1, __ffs(hits) - 1);
            if (lane == j) by[t] = x;
          }
        }
        if (lane == j) found[t] = hit;
      }
    }
#pragma unroll
    for (int t = 0; t < BW; ++t) {
      if (found[t]) {
        st_keep(depth + id[t], (DT)(s.L + 1));
        if (PAR) st_keep(r.parent + id[t], out_id(a, by[t]));
        my_n += 1;
        my_m += (unsigned)d[t];
      }
      const unsigned fm = __ballot_sync(FULL, found[t]);
      const int wi = w0 + t * nw;
      if (lane == 0 && fm) {  // this warp is the only writer of word wi during the level
        a.vis[wi] = vis[t] | fm;
        fbn[wi] = fm;
      }
    }
  }
}

// Three words of a warp and three entries a step; on small graphs, where a warp
// has few words and its last group would be mostly empty, two and four. us a
// traversal, words x entries 3 x 2, 3 x 3, 2 x 4: ER 2^19 of mean degree 16 108, 105,
// 100, of 29 184, 180, 172; R-MAT s16 66.6, 65.6, 63.5; ER 2^22 d16 291, 283, 301;
// ER 3M d6 305, 303, 323; R-MAT s22 155, 153, 153.
template <class DT, bool PAR>
__device__ void res_bu(const LevelArgs& a, const ResArgs& r, const ResState& s, const CrewSeat& seat, DT* depth,
                       unsigned& my_n, unsigned long long& my_m) {
  if ((a.n_active + 31) >> 5 <= (int64_t)seat.size * RW * R_BW_WORDS)
    res_bu_words<DT, PAR, 2, 4>(a, r, s, seat, depth, my_n, my_m);
  else
    res_bu_words<DT, PAR, 3, 3>(a, r, s, seat, depth, my_n, my_m);
}

// Queues the frontier in fb[s.f], left by a bottom-up level (vertices with rows).
__device__ void res_queue(const LevelArgs& a, const ResArgs& r, const ResState& s, const CrewSeat& seat,
                          const ResOut& o) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t gw = (int64_t)seat.rank * RW + warp, nw = (int64_t)seat.size * RW;
  const int64_t W = (a.n_active + 31) >> 5;
  for (int64_t w0 = gw * 32; w0 < W; w0 += nw * 32) {
    uint32_t bits = w0 + lane < W ? __ldcg(r.fb[s.f] + w0 + lane) : 0u;
    while (__any_sync(FULL, bits != 0)) {
      const int v = bits ? (int)((w0 + lane) * 32 + __ffs(bits) - 1) : -1;
      bits &= bits - 1;
      const int vs[1] = {v}, cls[1] = {v >= 0 ? res_class(__ldg(a.deg + v)) : -1};
      res_queue_up<1>(a, o, vs, cls, [&](int, int at) { o.q[at] = v; });
    }
  }
}

// The leader alone: top-down levels while the frontier is light and small, at most
// R_SOLO_LEVELS and no further than the direction rule allows; leaves the next
// frontier queued, its bits set in fbn, its counts in `n` and the totals in so.
template <class DT, bool PAR, class Solo>
__device__ void res_solo(const LevelArgs& a, const ResArgs& r, const ResState& s0, DT* depth, uint32_t* fbn, int32_t* n,
                         Solo* so, int4 (*s_q)[R_SOLO_CAP]) {
  __shared__ int32_t s_n[2][3];
  __shared__ unsigned long long s_m[2], s_v[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int L = s0.L, cnt = s0.n_l;
  int64_t n_vis = s0.n_vis, m_vis = s0.m_vis, n_f = s0.n_f, m_f = s0.m_f;
  for (int i = tid; i < cnt; i += RT) {
    const int u = __ldcg(r.queue[L & 1] + i);
    const int64_t st = a.off[u];
    s_q[L & 1][i] = make_int4(u, a.deg[u], (int)(uint32_t)st, (int)(uint32_t)((uint64_t)st >> 32));
  }
  if (tid < 3) s_n[0][tid] = s_n[1][tid] = 0;
  if (tid < 2) s_m[tid] = s_v[tid] = 0;
  __syncthreads();
  int n2 = 0, n3 = 0, mid = 0;
  for (int run = 0;; ++run) {
    const int cur = L & 1, nxt = cur ^ 1;
    mid += res_mid(m_f);
    const ResOut o{nullptr, r.queue[nxt], r.huge[nxt], s_n[nxt], s_q[nxt], r.parent};
    const int k = min(32, (cnt + RW - 1) / RW);
    unsigned my_n = 0;
    unsigned long long my_m = 0;
    for (int first = warp * k; first < cnt; first += RW * k) {
      int d = 0, id = -1;
      int64_t st = 0;
      if (lane < k && first + lane < cnt) {
        const int4 e = s_q[cur][first + lane];
        d = e.y;
        st = (int64_t)(((uint64_t)(uint32_t)e.w << 32) | (uint32_t)e.z);
        id = out_id(a, e.x);
      }
      res_rows<DT, true, PAR>(a, d, st, id, L + 1, depth, o, my_n, my_m);
      if (id >= 0) depth[id] = (DT)L;
    }
    my_n = __reduce_add_sync(FULL, my_n);
    if (my_n) {
      // a lane's claims in one level hold fewer than 2^32 entries of light rows; heavy ones may be any
#pragma unroll
      for (int ofs = 16; ofs > 0; ofs >>= 1) my_m += __shfl_xor_sync(FULL, my_m, ofs);
      if (lane == 0) {
        atomicAdd(&s_v[nxt], (unsigned long long)my_n);
        atomicAdd(&s_m[nxt], my_m);
      }
    }
    __syncthreads();
    cnt = s_n[nxt][0];
    n2 = s_n[nxt][1];
    n3 = s_n[nxt][2];
    n_f = (int64_t)s_v[nxt];
    m_f = (int64_t)s_m[nxt];
    n_vis += n_f;
    m_vis += m_f;
    ++L;
    const bool bu = (a.policy == ENT_POLICY_BEAMER && (double)m_f > (double)(a.E - m_vis) / a.alpha) ||
                    (a.policy == ENT_POLICY_REFERENCE && (double)m_f >= a.ref_ratio * (double)a.E);
    if (n_f == 0 || cnt > R_SOLO_CAP || n_f > 2 * (int64_t)a.narrow_f || m_f > min(a.exit_m, 2 * (int64_t)R_SOLO_M) || n2 || n3 || bu ||
        run + 1 >= R_SOLO_LEVELS || L >= a.max_levels)
      break;
    if (tid < 3) s_n[cur][tid] = 0;  // takes the counts of the level after
    if (tid == 3) s_m[cur] = s_v[cur] = 0;
    __syncthreads();
  }
  // hand over: stored entries to the queue (the rest are there), depths, bits, counts
  int32_t* q = r.queue[L & 1];
  for (int i = tid; i < min(cnt, R_SOLO_CAP); i += RT) q[i] = s_q[L & 1][i].x;
  __syncthreads();
  const auto hand = [&](int v) {
    depth[out_id(a, v)] = (DT)L;
    red_or(fbn + (v >> 5), 1u << (v & 31));
  };
  for (int i = tid; i < cnt; i += RT) hand(q[i]);
  for (int i = tid; i < n2; i += RT) hand(q[a.V - 1 - i]);
  for (int i = tid; i < n3; i += RT) hand(r.huge[L & 1][i]);
  if (tid == 0) {
    n[0] = cnt;
    n[1] = n2;
    n[2] = n3;
    so->n_f = n_f;
    so->m_f = m_f;
    so->n_vis = n_vis;
    so->m_vis = m_vis;
    so->level = L;
    so->mid_levels = mid;
  }
}

enum { RP_ALL, RP_HEAD, RP_TAIL };  // the part of the traversal a launch runs
// Bottom-up kernels between head and tail: R-MAT and uniform graphs take three
// or four such levels, and one that is not needed costs 6 us.
constexpr int R_BU_LEVELS = 4;

// The row entries, about, of a phase to come.
__device__ __forceinline__ int64_t res_work(const LevelArgs& a, const ResState& s, int kind) {
  switch (kind) {
    case RK_TD: return s.m_f;
    case RK_BU: return 2 * (a.n_active - s.n_vis);
    case RK_QUEUE: return a.n_active / 16;
    default: return 0;
  }
}

// A small crew waits for more members before a long phase.
__device__ __forceinline__ void res_gather(const LevelArgs& a, ResState& s, const CrewSeat& seat, int part) {
  if ((part == RP_HEAD && s.kind == RK_BU) || s.kind == RK_DONE || !crew_short(seat, res_work(a, s, s.kind))) return;
  s.then = s.kind;
  s.kind = RK_GATHER;
}

// The traversal's end, for the host (one thread).
__device__ void res_finish(const LevelArgs& a, const ResState& s, int32_t src, int part) {
  BfsCtl* k = a.ctl;
  k->src = src;
  k->level = s.L;
  k->done = 1;
  k->err = s.err;
  k->td_levels = s.td_levels;
  k->bu_levels = s.bu_levels;
  k->narrow_levels = s.narrow_levels;
  k->mid_levels = s.mid_levels;
  k->iters = 0;
  k->narrow_calls = 0;
  k->split_launches = part == RP_TAIL ? R_BU_LEVELS + 1 : 0;
  k->n_vis = s.n_vis;
  k->m_vis = s.m_vis;
}

template <class DT, bool PAR>
__global__ void __launch_bounds__(RT, 1) k_resident(LevelArgs a, ResArgs r, int32_t src, DT* depth, int part) {
  extern __shared__ int4 s_dyn[];
  int4(*s_q)[R_SOLO_CAP] = reinterpret_cast<int4(*)[R_SOLO_CAP]>(s_dyn);
  __shared__ ResState s_st;
  __shared__ CrewSeat s_seat;
  __shared__ unsigned long long s_red[2];
  ResCtl* c = r.rc;
  Crew<ResState>* crew = &c->crew[part == RP_TAIL];
  const int64_t W = (a.V + 31) >> 5;
  if (threadIdx.x == 0) s_red[0] = s_red[1] = 0;
  if (part == RP_TAIL && c->err) return;  // the head's error status stands
  if (part == RP_TAIL && c->state.kind == RK_DONE) {
    if (blockIdx.x == 0 && threadIdx.x == 0) res_finish(a, c->state, src, part);
    return;
  }
  const int32_t isrc = part == RP_TAIL ? 0 : (a.inv ? __ldg(a.inv + src) : src);
  // one CTA's share of the fills
  const auto fill = [&](uint32_t share) {
    const int64_t tid = (int64_t)share * RT + threadIdx.x, nth = (int64_t)gridDim.x * RT;
    fill_unreached(depth, a.V, tid, nth, src);
    if (PAR) fill_neg1(r.parent, a.V, tid, nth, src, src);
    for (int64_t i = tid; i < W; i += nth) {
      const uint32_t x = i == (isrc >> 5) ? 1u << (isrc & 31) : 0u;
      a.vis[i] = x;
      r.fb[0][i] = x;
      r.fb[1][i] = 0;
      r.fb[2][i] = 0;
    }
  };
  // what a founder does before the first phase, of which it knows the state
  const auto begin = [&](uint32_t rank) {
    if (threadIdx.x == 32) {
      ResState s;
      if (part == RP_TAIL) {
        s = c->state;
      } else {
        const int d = a.deg[isrc];
        s.L = s.f = s.p = s.then = 0;
        s.td_levels = s.bu_levels = s.narrow_levels = s.mid_levels = s.err = 0;
        s.n_f = s.n_vis = 1;
        s.m_f = s.m_vis = d;
        s.n_l = d < R_HEAVY;
        s.n_g = d >= R_HUGE;
        s.n_h = 1 - s.n_l - s.n_g;
        s.kind = a.policy == ENT_POLICY_BU_ONLY ? RK_BU : res_td_kind(a, s);
        if (rank == 0) {
          if (s.n_l) r.queue[0][0] = isrc;
          else if (s.n_h) r.queue[0][a.V - 1] = isrc;
          else r.huge[0][0] = isrc;
          // Until its end says otherwise the traversal has failed: whichever wait
          // runs out, and whichever CTAs notice, the host does not read the last
          // one's status.
          a.ctl->err = 2;
        }
      }
      s_st = s;
    }
    if (part != RP_TAIL) fill(rank);
  };
  // what every member concludes from an opened barrier
  const auto advance = [&] {
    ResState& s = s_st;
    if (s.kind >= RK_GATHER) {
      s.p += 1;
      s.kind = s.then;
      return;
    }
    res_advance(a, r, s);
    if (s_seat.size < gridDim.x) res_gather(a, s, s_seat, part);
  };
  const int in = crew_join(crew, &c->err, s_seat, s_st, begin, advance);
  if (!in) return;
  const int rank = s_seat.rank;
  if (in == 1 && s_seat.size < gridDim.x) {  // a small crew
    if (threadIdx.x == 0) {
      ResState& s = s_st;
      if (part == RP_TAIL) {
        res_gather(a, s, s_seat, part);
      } else {  // some shares are nobody's
        s.then = s.kind;
        s.kind = RK_FILL;
      }
    }
    __syncthreads();
  }
  for (;;) {
    const ResState& s = s_st;  // thread 0 changes it inside the barrier only
    if (s.kind == RK_DONE || (part == RP_HEAD && s.kind == RK_BU)) break;
    const CrewSeat seat = s_seat;
    const int64_t tid = (int64_t)rank * RT + threadIdx.x, nth = (int64_t)seat.size * RT;
    int32_t* n_next = c->n[(s.p + 1) % 3];
    unsigned long long* acc = c->acc[(s.p + 1) % 3];
    if (tid < 3) c->n[(s.p + 2) % 3][tid] = 0;
    if (tid < 2) c->acc[(s.p + 2) % 3][tid] = 0;
    if (s.kind != RK_QUEUE && s.kind < RK_DONE) {  // the bits of the frontier before this one
      uint32_t* old = r.fb[(s.f + 2) % 3];
      for (int64_t i = tid; i < W; i += nth) old[i] = 0;
    }
    unsigned my_n = 0;
    unsigned long long my_m = 0;
    uint32_t* fbn = r.fb[(s.f + 1) % 3];
    const int nq = s.kind == RK_QUEUE ? s.L & 1 : (s.L + 1) & 1;
    const ResOut o{fbn, r.queue[nq], r.huge[nq], n_next, nullptr, r.parent};
    if (s.kind == RK_TD) res_td<DT, PAR>(a, r, s, seat, depth, o, my_n, my_m);
    else if (s.kind == RK_BU) res_bu<DT, PAR>(a, r, s, seat, depth, my_n, my_m);
    else if (s.kind == RK_QUEUE) res_queue(a, r, s, seat, o);
    else if (s.kind == RK_GATHER) crew_gather(crew, seat, res_work(a, s, s.then));
    else if (s.kind == RK_FILL)
      for (uint32_t i = s_seat.size + rank; i < gridDim.x; i += s_seat.size) fill(i);
    else if (rank == 0) res_solo<DT, PAR>(a, r, s, depth, fbn, n_next, &c->solo[s.p & 1], s_q);
    if (s.kind <= RK_BU) {
      const unsigned wn = __reduce_add_sync(FULL, my_n);
      if (wn) {
#pragma unroll
        for (int ofs = 16; ofs > 0; ofs >>= 1) my_m += __shfl_xor_sync(FULL, my_m, ofs);
        if ((threadIdx.x & 31) == 0) {
          atomicAdd(&s_red[0], (unsigned long long)wn);
          atomicAdd(&s_red[1], my_m);
        }
      }
      __syncthreads();
      if (threadIdx.x == 0 && s_red[0]) {
        atomicAdd(&acc[0], s_red[0]);
        atomicAdd(&acc[1], s_red[1]);
        s_red[0] = s_red[1] = 0;
      }
    }
    // test hook: a CTA that never arrives (the others' waits run out)
    if (a.fault_inject && part == RP_ALL && rank > 0 && rank == (int)s_seat.size - 1) return;
    if (!crew_barrier(crew, &c->err, s_seat, s_st, advance)) {
      crew_close(crew, s_seat);
      return;
    }
  }
  crew_close(crew, s_seat);
  const int64_t tid = (int64_t)rank * RT + threadIdx.x;
  // test hook: a CTA that gave up just as the head's last barrier opened for the others
  if (a.fault_inject && part == RP_HEAD && threadIdx.x == 0 && rank == (int)s_seat.size - 1) c->err = 1;
  if (tid == 0 && part == RP_HEAD) c->state = s_st;
  if (tid == 0 && part != RP_HEAD) res_finish(a, s_st, src, part);
}

// One bottom-up level of a traversal in parts, if that is what comes next:
// k_expand's sweep, the old frontier's bits cleared beside it, and the decision
// by the last CTA to finish.
template <class DT, bool PAR>
__global__ void __launch_bounds__(BT, 8) k_res_bu_level(LevelArgs a, ResArgs r, DT* depth) {
  __shared__ unsigned long long s_red[BT / 32];
  __shared__ int s_last;
  ResCtl* c = r.rc;
  if (c->state.kind != RK_BU || c->err) return;
  const int f = c->state.f, p = c->state.p, L = c->state.L;
  {
    uint32_t* old = r.fb[(f + 2) % 3];
    const int64_t W = (a.V + 31) >> 5;
    for (int64_t i = blockIdx.x * (int64_t)BT + threadIdx.x; i < W; i += (int64_t)gridDim.x * BT) old[i] = 0;
  }
  const Front is_front{r.fb[f], nullptr, 0, 0};
  unsigned long long my_n = 0, my_m = 0;
  bu_words<DT>(a, is_front, r.fb[(f + 1) % 3], L + 1, depth, PAR ? r.parent : nullptr, nullptr, my_n, my_m);
  unsigned long long* acc = c->acc[(p + 1) % 3];
  if (__syncthreads_or(my_n != 0)) {
    unsigned long long x = block_sum(my_n, s_red);
    if (threadIdx.x == 0) atomicAdd(&acc[0], x);
    x = block_sum(my_m, s_red);
    if (threadIdx.x == 0) atomicAdd(&acc[1], x);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&c->finished, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last || threadIdx.x != 0) return;
  __threadfence();
  ResState s = c->state;
  res_advance(a, r, s);
  for (int i = 0; i < 3; ++i) c->n[(p + 2) % 3][i] = 0;
  c->acc[(p + 2) % 3][0] = c->acc[(p + 2) % 3][1] = 0;
  c->state = s;
  c->finished = 0;
}
