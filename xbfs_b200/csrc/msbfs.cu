// Batched multi-source BFS: up to 64*W sources traversed together, 64
// sources packed per uint64 word, W words per vertex (W = 1, 2, 4, 8; 512
// sources = 8 groups of 64 in one pass at W = 8).
//
// No counterpart in the reference (it runs one source per process). The
// bit-parallel formulation is the standard multi-source BFS: per vertex a
// visited word set vis[v] and a frontier word set F[v] (bits that arrived at
// the current level). Top-down pushes F[u] & ~vis[v] with atomic ORs;
// bottom-up lets every vertex that still lacks sources OR in the frontier
// words of its neighbours. Both directions are exact for every source,
// whatever the schedule.
//
// B200 layout and schedule:
//  * Levels are bit-sliced: plane k holds bit k of the level of every
//    (vertex, source), so a vertex that gains sources at level l ORs one word
//    set into the planes of l's set bits instead of storing one byte per
//    source. Planes are zeroed when a level first needs them, and
//    k_ms_expand turns visited words and planes into the int32 rows of the
//    API (four levels per step, spread to bytes by a multiply).
//  * Bottom-up takes W/2 lanes per vertex, two words (16 bytes) each: a
//    warp reads 8 (W = 8) to 32 neighbours' frontier words per load
//    instruction as whole sectors, eight loads in flight (four for high-degree
//    vertices below W = 8). Low-degree vertices of a ticket stream through the
//    lane groups from a per-warp list, higher degrees take a whole warp, and
//    the neighbour lists of degree above kMega are cut into chunks that any
//    warp of the grid takes, their gains meeting in an accumulator that the
//    chunk finishing last merges.
//  * Only sources that are alive (some vertex gained them at the last
//    level) are searched for: a source whose component is exhausted stops
//    holding up the early exit of every other vertex.
//  * Frontier, visited-by-frontier bitmap and queue counters are rings, so a
//    level costs one grid barrier (and one more when a bottom-up frontier
//    has to be turned into a queue); top-down expansion is edge-balanced over
//    the queue's exclusive edge offsets.
#include <string.h>

#include <algorithm>
#include <chrono>
#include <memory>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "internal.hpp"

namespace xbfs {

namespace ms {

typedef unsigned long long u64;
constexpr int kBlock = 512;
constexpr int kWarps = kBlock / 32;
constexpr int kLight = 64;     // bottom-up: up to this degree one lane group takes the vertex, above it a warp
constexpr int kMegaLog = 10;
constexpr int kMega = 1 << kMegaLog;  // bottom-up: above this degree the list is cut into chunks of kMega edges
constexpr int kStep = 8;       // neighbours a lane group reads per step (light vertices; heavy ones at W = 8)
constexpr int kExpand = 512;   // threads of an expansion CTA
constexpr int kTicketWords = 4;  // bitmap words (of 32 vertices) per bottom-up ticket, at most
constexpr int kLoPlanes = 8, kMaxPlanes = 16;
constexpr u64 kCountMask = (1ull << 31) - 1;

struct Ctl {
  GridBarrier bar;
  int depth;           // levels of the finished traversal (0 until then)
  int more;            // stopped before level 255: the planes above the low eight are needed
  u64 q[4];            // packed (edges << 31) | count, frontier queue ring
  u64 n_f[4], m_f[4];  // frontiers that bottom-up levels produced: vertices, degree sum
  u64 m_done[4];       // degree sum of vertices completed, per level
  u64 alive[4][8];     // sources with a frontier at each level
  unsigned tick[4];    // bottom-up work tickets
  int strat_count[2];
  unsigned n_mega, n_tasks;
  u64 msum;            // sum over sources of the degrees of reached vertices
  // loop state of a traversal that stopped for more planes
  long long r_level, r_done;
  int r_qv, r_qvp;
};

template <int W>
struct Params {
  const long long* beg;
  const int* csr;
  long long V, E;
  u64* vis;             // [V][W], padded to ps words
  u64* F[3];            // [V][W], ring by level; all zero outside the live frontiers
  uint32_t* fbm[3];     // vertices with frontier bits, ring by level like F
  long long ps;         // words from one plane to the next: V * W rounded up to even (16-byte alignment)
  u64* lo;              // planes 0-7, [8][ps]
  u64* hi;              // planes 8-15 (null until a traversal needs them)
  uint32_t* done;       // vertices that need no search any more (isolated + tail pre-set)
  int* qids[4];
  unsigned* qeb[4];     // exclusive edge offset within the queue
  unsigned* qbg[4];     // CSR offset of the vertex (E < 2^32)
  int* mega_v;          // vertices of degree > kMega
  uint2* tasks;         // (index into mega_v, chunk)
  unsigned* mega_n;     // chunks finished at this level, per mega vertex
  u64* mega_acc;        // [n_mega][W]: bits found at this level so far
  Ctl* ctl;
  long long nwords;
  long long m_active;   // degree sum of non-isolated vertices
  float alpha;          // top-down while m_f <= (m_u + bu_fixed) / alpha
  long long bu_fixed;
  int allow_bu;
  int force;            // -1: heuristic, 0: always top-down, 1: bottom-up whenever allowed
  int symmetric;        // done starts from the isolated-vertex bitmap
  int have_mega;
  int resume;
  int level_cap;        // stop before this level (255: more planes; 65535: levels do not fit)
  u64 timeout_ns;
  long long max_levels;
  const uint32_t* iso;
};

struct Seeds {
  int n;
  int v[512];
};

struct __align__(16) Smem {
  unsigned wbeg[kBlock + 1];
  unsigned web[kBlock + 1];
  int wu[kBlock + 1];
  // per warp: the vertices of a bottom-up ticket, light ones from the front,
  // heavy ones from the back
  int lv[kWarps][32 * kTicketWords];
  unsigned lb[kWarps][32 * kTicketWords];
  int ldeg[kWarps][32 * kTicketWords];
  u64 alive[8];       // sources with a frontier at this level
  u64 next_alive[8];  // and at the next, as far as this CTA found them
  int next_s;
  int decision;
  int few;            // bottom-up: few edges are left to search
  int sparse;         // bottom-up: look into the frontier's bitmap before reading a neighbour's words
  u64 cnt_m;          // packed size of this level's frontier queue
  long long red[3 * kWarps];
};

template <int W>
struct Geo {
  static constexpr int WL = W >= 2 ? 2 : 1;  // words per lane
  static constexpr int G = W / WL;           // lanes per vertex
  static constexpr int NG = 32 / G;          // vertices side by side in a warp
};

template <int WL>
__device__ __forceinline__ void ld_words(const u64* p, u64 (&x)[WL]) {
  if (WL == 2) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(p);
    x[0] = t.x;
    x[WL - 1] = t.y;
  } else {
    x[0] = *p;
  }
}
template <int WL>
__device__ __forceinline__ void st_words(u64* p, const u64 (&x)[WL]) {
  if (WL == 2)
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x[0], x[WL - 1]);
  else
    *p = x[0];
}

template <int W>
__device__ __forceinline__ u64* plane(const Params<W>& p, int k) {
  return k < kLoPlanes ? p.lo + (size_t)k * p.ps : p.hi + (size_t)(k - kLoPlanes) * p.ps;
}

// ORs the gained bits of word `idx` (= v * W + w) into the planes of `level`.
template <int W>
__device__ __forceinline__ void record(const Params<W>& p, size_t idx, u64 gained, int level) {
  for (int b = level; b; b &= b - 1) red_or_u64(plane(p, __ffs(b) - 1) + idx, gained);
}

// Warp-aggregated append to queue ring slot s (full warp).
template <int W>
__device__ __forceinline__ void warp_enqueue(const Params<W>& p, int s, bool have, int v, long long deg, unsigned b0) {
  const unsigned mask = __ballot_sync(0xffffffffu, have);
  if (!mask) return;
  const int lane = threadIdx.x & 31;
  const long long d = have ? deg : 0;
  const long long inc = warp_inclusive_scan(d);
  u64 old = 0;
  if (lane == 31) old = atomicAdd(&p.ctl->q[s], ((u64)inc << 31) | (u64)__popc(mask));
  old = __shfl_sync(0xffffffffu, old, 31);
  if (have) {
    const unsigned slot = (unsigned)(old & kCountMask) + __popc(mask & ((1u << lane) - 1));
    p.qids[s][slot] = v;
    p.qeb[s][slot] = (unsigned)((old >> 31) + (u64)(inc - d));
    p.qbg[s][slot] = b0;
  }
}

// One edge (owner -> v) of a top-down level: the owner's frontier words are
// offered to v, each source bit is won by exactly one atomic OR on vis[v],
// and won bits go into the next frontier and the planes. Returns whether
// this thread is the one that queues v (the first to set v's bit in the next
// frontier's bitmap). A vertex without edges gets its levels, no frontier.
template <int W>
__device__ __forceinline__ bool td_claim(const Params<W>& p, Smem& sm, const u64* Fc, u64* Fn, uint32_t* fbn, int owner,
                                         int v, int level, long long& deg, unsigned& b0, long long& m_done) {
  constexpr int WL = Geo<W>::WL;
  bool won = false;
  deg = -1;
#pragma unroll
  for (int w = 0; w < W; w += WL) {
    u64 f[WL], m[WL];
    ld_words<WL>(Fc + (size_t)owner * W + w, f);
    bool any = false;
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      m[i] = f[i] ? f[i] & ~ld_cg_u64(p.vis + (size_t)v * W + w + i) : 0ull;
      any |= m[i] != 0;
    }
    if (!any) continue;
    if (deg < 0) {
      const long long x = ld_nc_i64(p.beg + v);
      deg = ld_nc_i64(p.beg + v + 1) - x;
      b0 = (unsigned)x;
    }
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      if (!m[i]) continue;
      const size_t idx = (size_t)v * W + w + i;
      const u64 old = atomicOr(p.vis + idx, m[i]);
      const u64 g = m[i] & ~old;
      if (!g) continue;
      record(p, idx, g, level);
      if (W == 1 && !(sm.alive[0] & ~(old | m[i]))) {
        red_or_u32(p.done + (v >> 5), 1u << (v & 31));
        m_done += deg;
      }
      if (deg == 0) continue;
      red_or_u64(Fn + idx, g);
      if (g & ~*(volatile u64*)&sm.next_alive[w + i]) atomicOr(&sm.next_alive[w + i], g);
      won = true;
    }
  }
  if (!won) return false;
  const uint32_t bit = 1u << (v & 31);
  return !(atomicOr(fbn + (v >> 5), bit) & bit);
}

// Top-down level: the edges of frontier queue slot qs, shared equally between
// the CTAs. A small queue of low-degree vertices is cut by entries (each CTA
// loads its entries directly), any other by edges (each CTA searches the
// entry that owns its first edge and walks a window of entries).
template <int W>
__device__ void ms_td(const Params<W>& p, Smem& sm, int qs, int qn, const u64* Fc, u64* Fn, uint32_t* fbn, int level,
                      long long& m_done) {
  const int lane = threadIdx.x & 31;
  const unsigned cnt = (unsigned)(sm.cnt_m & kCountMask);
  const u64 M = sm.cnt_m >> 31;
  const u64 nb = gridDim.x, b = blockIdx.x;
  const int* ids = p.qids[qs];
  const unsigned* eb = p.qeb[qs];
  const unsigned* bgs = p.qbg[qs];
  if ((u64)cnt <= 32ull * nb && M <= 32ull * cnt) {
    const unsigned i0 = (unsigned)((u64)cnt * b / nb), i1 = (unsigned)((u64)cnt * (b + 1) / nb);
    if (i0 >= i1) return;
    const int n = (int)(i1 - i0);
    const unsigned base = eb[i0];
    const unsigned T = (unsigned)(((i1 < cnt) ? (u64)eb[i1] : M) - base);
    if (threadIdx.x < n) {
      const unsigned slot = i0 + threadIdx.x;
      sm.wu[threadIdx.x] = ids[slot];
      sm.wbeg[threadIdx.x] = bgs[slot];
      sm.web[threadIdx.x] = eb[slot] - base;
    }
    __syncthreads();
    for (unsigned e0 = 0; e0 < T; e0 += kBlock) {
      const unsigned e = e0 + threadIdx.x;
      if ((e & ~31u) >= T) break;  // whole warps leave together
      bool first = false;
      int v = 0;
      long long deg = 0;
      unsigned b0 = 0;
      if (e < T) {
        int a = 0, c = n;
        while (c - a > 1) {
          const int mid = (a + c) >> 1;
          if (sm.web[mid] <= e) a = mid; else c = mid;
        }
        v = ld_stream_i32(p.csr + sm.wbeg[a] + (e - sm.web[a]));
        first = td_claim<W>(p, sm, Fc, Fn, fbn, sm.wu[a], v, level, deg, b0, m_done);
      }
      warp_enqueue(p, qn, first, v, deg, b0);
    }
    return;
  }
  const u64 lo = M * b / nb, hi = M * (b + 1) / nb;
  if (lo >= hi) return;
  if (threadIdx.x < 32) {
    unsigned a = 0, c = cnt;
    while (c - a > 32) {
      const unsigned span = c - a;
      const unsigned piv = a + (unsigned)(((u64)span * lane) / 32);
      const unsigned m = __ballot_sync(0xffffffffu, (u64)eb[piv] <= lo);
      const int last = 31 - __clz(m);
      const unsigned na = a + (unsigned)(((u64)span * last) / 32);
      const unsigned nc = (last == 31) ? c : a + (unsigned)(((u64)span * (last + 1)) / 32);
      a = na;
      c = nc;
    }
    const unsigned idx = a + lane;
    const unsigned m = __ballot_sync(0xffffffffu, idx < c && (u64)eb[idx] <= lo);
    if (lane == 0) sm.next_s = (int)(a + 31 - __clz(m));
  }
  __syncthreads();
  unsigned s = (unsigned)sm.next_s;
  for (u64 r = lo; r < hi; r += kBlock) {
    const u64 rhi = (r + kBlock < hi) ? r + kBlock : hi;
    for (int i = threadIdx.x; i <= kBlock; i += kBlock) {
      const unsigned slot = s + (unsigned)i;
      unsigned e0 = 0xffffffffu;
      if (slot < cnt) {
        const unsigned x = eb[slot];
        if ((u64)x < rhi) {
          e0 = x;
          sm.wu[i] = ids[slot];
          sm.wbeg[i] = bgs[slot];
        }
      }
      sm.web[i] = e0;
    }
    __syncthreads();
    const u64 e = r + threadIdx.x;
    bool first = false;
    int v = 0;
    long long deg = 0;
    unsigned b0 = 0;
    if (e < rhi) {
      int a = 0, c = kBlock + 1;
      while (c - a > 1) {
        const int mid = (a + c) >> 1;
        if ((u64)sm.web[mid] <= e) a = mid; else c = mid;
      }
      v = ld_stream_i32(p.csr + sm.wbeg[a] + (unsigned)(e - sm.web[a]));
      first = td_claim<W>(p, sm, Fc, Fn, fbn, sm.wu[a], v, level, deg, b0, m_done);
    }
    warp_enqueue(p, qn, first, v, deg, b0);
    if (threadIdx.x == 0 && rhi < hi) {
      int a = 0, c = kBlock + 1;
      while (c - a > 1) {
        const int mid = (a + c) >> 1;
        if ((u64)sm.web[mid] <= rhi) a = mid; else c = mid;
      }
      sm.next_s = (int)(s + a);
    }
    __syncthreads();
    s = (unsigned)sm.next_s;
  }
}

// Per-lane state of a bottom-up level.
template <int W>
struct Bu {
  u64 al[Geo<W>::WL];  // alive sources, this lane's words
  u64 ga[Geo<W>::WL];  // OR of everything gained
  long long n_f, m_f, m_done;
};

// Closes the search of vertex v for the lane groups with `fin`: stores the
// gains (g: this lane's words, vv: its visited words before), marks v in the
// next frontier's bitmap and, when no alive source is missing any more, as
// done. Called by the full warp.
template <int W>
__device__ __forceinline__ void bu_close(const Params<W>& p, Bu<W>& st, bool fin, int v, unsigned deg,
                                         const u64 (&vv)[Geo<W>::WL], const u64 (&g)[Geo<W>::WL], u64* Fn,
                                         uint32_t* fbn, int level) {
  constexpr int WL = Geo<W>::WL, G = Geo<W>::G;
  const int lane = threadIdx.x & 31, gl = lane % G;
  const unsigned gmask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << (lane - gl);
  bool any = false, open = false;
#pragma unroll
  for (int i = 0; i < WL; ++i) {
    any |= g[i] != 0;
    open |= (st.al[i] & ~(vv[i] | g[i])) != 0;
  }
  const unsigned am = __ballot_sync(0xffffffffu, fin && any);
  const unsigned om = __ballot_sync(0xffffffffu, fin && open);
  if (!fin) return;
  if (am & gmask) {
    const size_t idx = (size_t)v * W + gl * WL;
    st_words<WL>(Fn + idx, g);
    if (any) {
      u64 vn[WL];
#pragma unroll
      for (int i = 0; i < WL; ++i) {
        vn[i] = vv[i] | g[i];
        st.ga[i] |= g[i];
        if (g[i]) record(p, idx + i, g[i], level);
      }
      st_words<WL>(p.vis + idx, vn);
    }
    if (gl == 0) {
      red_or_u32(fbn + (v >> 5), 1u << (v & 31));
      st.n_f += 1;
      st.m_f += deg;
    }
  }
  if (gl == 0 && !(om & gmask)) {
    red_or_u32(p.done + (v >> 5), 1u << (v & 31));
    st.m_done += deg;
  }
}

// v when it has frontier bits (its bit in the frontier's bitmap), else the
// zero row `none` (the bitmap is padded past it).
__device__ __forceinline__ int in_frontier(const uint32_t* fb, int v, int none) {
  return ((fb[v >> 5] >> (v & 31)) & 1u) ? v : none;
}

// The frontier words of `left` neighbours from CSR entry e on, ORed by the
// whole warp until none of the sources the vertex lacks (need, this lane's
// words) is open or the range ends; acc receives the union on every lane group. `sparse` is
// the frontier's bitmap on levels that look there first, else null.
//
// Bound by the latency of its two dependent reads (CSR entry, then frontier
// words) at 32 warps per SM, so it keeps K reads of 8 or 16 bytes per lane in
// flight and the next step's CSR entries on the way: K = 8 against 4 at W = 8
// is 5.86 against 6.04 ms per 512-source call on R-MAT scale 22 ef 16.
// `left` counts the entries from e on; offsets never pass e + left < 2^32.
template <int W>
__device__ __forceinline__ void warp_pull(const Params<W>& p, const u64* Fc, const uint32_t* sparse, unsigned e,
                                          int left, const u64 (&need)[Geo<W>::WL], u64 (&acc)[Geo<W>::WL]) {
  constexpr int WL = Geo<W>::WL, G = Geo<W>::G, NG = Geo<W>::NG;
  constexpr int K = W == 8 ? kStep : 4;  // neighbours per lane group and step
  constexpr int R = NG * K / 32;  // CSR entries per lane and step
  const int lane = threadIdx.x & 31, gl = lane % G, grp = lane / G, none = (int)p.V;
  const u64* Fl = Fc + gl * WL;
  int own[R];
#pragma unroll
  for (int r = 0; r < R; ++r) own[r] = (r * 32 + lane < left) ? ld_stream_i32(p.csr + (e + r * 32 + lane)) : none;
  for (;;) {
    if (sparse) {
#pragma unroll
      for (int r = 0; r < R; ++r) own[r] = in_frontier(sparse, own[r], none);
    }
    u64 f[K][WL];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int u = __shfl_sync(0xffffffffu, own[(k * NG) / 32], (k * NG + grp) & 31);
      ld_words<WL>(Fl + (size_t)(unsigned)u * W, f[k]);
    }
    e += NG * K;
    left -= NG * K;
#pragma unroll
    for (int r = 0; r < R; ++r) own[r] = (r * 32 + lane < left) ? ld_stream_i32(p.csr + (e + r * 32 + lane)) : none;
    bool open = false;
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      u64 a = f[0][i];
#pragma unroll
      for (int k = 1; k < K; ++k) a |= f[k][i];
#pragma unroll
      for (int o = G; o < 32; o <<= 1) a |= __shfl_xor_sync(0xffffffffu, a, o);
      acc[i] |= a;
      open |= (need[i] & ~acc[i]) != 0;
    }
    if (left <= 0 || !__any_sync(0xffffffffu, open)) break;
  }
}

// One chunk of a vertex whose list is cut up. The bits found go to the
// vertex's accumulator; the warp that finishes the vertex's last chunk closes
// its search.
template <int W>
__device__ void bu_chunk(const Params<W>& p, Bu<W>& st, const u64* Fc, const uint32_t* sparse, u64* Fn,
                         uint32_t* fbn, int level, uint2 tk, int v) {
  constexpr int WL = Geo<W>::WL, G = Geo<W>::G;
  const int lane = threadIdx.x & 31, gl = lane % G;
  const unsigned b0 = (unsigned)ld_nc_i64(p.beg + v), deg = (unsigned)(ld_nc_i64(p.beg + v + 1)) - b0;
  const size_t idx = (size_t)v * W + gl * WL;
  u64* ap = p.mega_acc + (size_t)tk.x * W + gl * WL;
  u64 vv[WL], need[WL], acc[WL];
  ld_words<WL>(p.vis + idx, vv);
#pragma unroll
  for (int i = 0; i < WL; ++i) {
    need[i] = st.al[i] & ~(vv[i] | ld_cg_u64(ap + i));  // what no other chunk has found yet
    acc[i] = 0;
  }
  const unsigned c0 = tk.y << kMegaLog;
  bool open = false;
#pragma unroll
  for (int i = 0; i < WL; ++i) open |= need[i] != 0;
  if (__any_sync(0xffffffffu, open))
    warp_pull<W>(p, Fc, sparse, b0 + c0, (int)min(deg - c0, (unsigned)kMega), need, acc);
#pragma unroll
  for (int i = 0; i < WL; ++i)
    if (lane < G && (acc[i] & need[i])) red_or_u64(ap + i, acc[i] & need[i]);
  __threadfence();
  __syncwarp();
  unsigned n = 0;
  if (lane == 0) n = atomicAdd(p.mega_n + tk.x, 1u) + 1;
  n = __shfl_sync(0xffffffffu, n, 0);
  if (n != (deg + kMega - 1) >> kMegaLog) return;
  __threadfence();
  u64 g[WL];
#pragma unroll
  for (int i = 0; i < WL; ++i) g[i] = ld_cg_u64(ap + i);
  __syncwarp();
  bu_close<W>(p, st, lane < G, v, deg, vv, g, Fn, fbn, level);
  if (lane < G) {
#pragma unroll
    for (int i = 0; i < WL; ++i) ap[i] = 0ull;
    if (lane == 0) p.mega_n[tk.x] = 0u;
  }
}

// Tasks [t0, t1), at most 32: the chunks whose vertex is not done (done bits
// are set at the end of a vertex's last chunk of a level, so all chunks of
// one vertex see the same).
template <int W>
__device__ __forceinline__ void bu_chunks(const Params<W>& p, Bu<W>& st, const u64* Fc, const uint32_t* sparse,
                                          u64* Fn, uint32_t* fbn, int level, unsigned t0, unsigned t1) {
  const int lane = threadIdx.x & 31;
  uint2 tk = make_uint2(0, 0);
  int v = 0;
  bool open = false;
  if (t0 + lane < t1) {
    tk = p.tasks[t0 + lane];
    v = p.mega_v[tk.x];
    open = !((ld_cg_u32(p.done + (v >> 5)) >> (v & 31)) & 1u);
  }
  for (unsigned m = __ballot_sync(0xffffffffu, open); m; m &= m - 1) {
    const int k = __ffs(m) - 1;
    const uint2 x = make_uint2(__shfl_sync(0xffffffffu, tk.x, k), __shfl_sync(0xffffffffu, tk.y, k));
    bu_chunk<W>(p, st, Fc, sparse, Fn, fbn, level, x, __shfl_sync(0xffffffffu, v, k));
  }
}

// The vertices of one ticket: light ones stream through the lane groups,
// each group taking the next vertex of the warp's list when it is through
// with one; the others take the whole warp one after another.
template <int W>
__device__ void bu_words(const Params<W>& p, Smem& sm, Bu<W>& st, const u64* Fc, const uint32_t* sparse, u64* Fn,
                         uint32_t* fbn, int level, long long w0, int nw) {
  constexpr int WL = Geo<W>::WL, G = Geo<W>::G;
  constexpr int R = kStep / G;  // CSR entries per lane and step
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, gl = lane % G, gbase = lane - gl;
  const unsigned gmask = ((G == 32) ? 0xffffffffu : ((1u << G) - 1u)) << gbase;
  const unsigned leaders = 0xffffffffu / ((1u << G) - 1u);  // bit of each group's first lane
  const unsigned below = (1u << gbase) - 1u;
  constexpr int kList = 32 * kTicketWords;
  const int none = (int)p.V;
  const u64* Fl = Fc + gl * WL;
  int* lv = sm.lv[wid];
  unsigned* lb = sm.lb[wid];
  int* ld = sm.ldeg[wid];
  const uint32_t td = lane < nw ? ~ld_cg_u32(p.done + w0 + lane) : 0u;  // vertices left, one word per lane
  unsigned nz = __ballot_sync(0xffffffffu, td != 0);
  while (nz) {
    int nl = 0, nh = 0;
    __syncwarp();  // the previous list is no longer read
    while (nz && nl + nh <= kList - 32) {
      const int k = __ffs(nz) - 1;
      nz &= nz - 1;
      const uint32_t todo = __shfl_sync(0xffffffffu, td, k);
      const bool mine = (todo >> lane) & 1u;
      const int v = (int)((w0 + k) * 32) + lane;
      unsigned b0 = 0, deg = 0;
      if (mine) {
        const long long x = ld_nc_i64(p.beg + v);
        b0 = (unsigned)x;
        deg = (unsigned)(ld_nc_i64(p.beg + v + 1) - x);
      }
      const unsigned lm = __ballot_sync(0xffffffffu, mine && deg <= kLight);
      const unsigned hm = __ballot_sync(0xffffffffu, mine && deg > kLight && deg <= kMega);
      const unsigned lt = (1u << lane) - 1u;
      int at = -1;
      if ((lm >> lane) & 1u) at = nl + __popc(lm & lt);
      if ((hm >> lane) & 1u) at = kList - 1 - nh - __popc(hm & lt);
      if (at >= 0) {
        lv[at] = v;
        lb[at] = b0;
        ld[at] = (int)deg;
      }
      nl += __popc(lm);
      nh += __popc(hm);
    }
    __syncwarp();
    // ---- light vertices
    int next = 0, v = 0;
    unsigned e = 0, deg = 0;
    int left = 0;
    bool act = false;
    u64 vv[WL], acc[WL];
#pragma unroll
    for (int i = 0; i < WL; ++i) vv[i] = acc[i] = 0ull;
    for (;;) {
      const unsigned idle = ~__ballot_sync(0xffffffffu, act) & leaders;
      if (idle && next < nl) {
        const int r = next + __popc(idle & below);
        if (!act && r < nl) {
          v = lv[r];
          e = lb[r];
          deg = (unsigned)ld[r];
          left = (int)deg;
          ld_words<WL>(p.vis + (size_t)v * W + gl * WL, vv);
#pragma unroll
          for (int i = 0; i < WL; ++i) acc[i] = 0ull;
          act = true;
        }
        next += __popc(idle);
      }
      if (!__any_sync(0xffffffffu, act)) break;
      int own[R];
#pragma unroll
      for (int r = 0; r < R; ++r) own[r] = (act && r * G + gl < left) ? __ldg(p.csr + (e + r * G + gl)) : none;
      if (sparse) {
#pragma unroll
        for (int r = 0; r < R; ++r) own[r] = in_frontier(sparse, own[r], none);
      }
      u64 f[kStep][WL];
#pragma unroll
      for (int k = 0; k < kStep; ++k) {
        const int u = (G == 1) ? own[k / G] : __shfl_sync(0xffffffffu, own[k / G], gbase + k % G);
        ld_words<WL>(Fl + (size_t)(unsigned)u * W, f[k]);
      }
      bool open = false;
#pragma unroll
      for (int i = 0; i < WL; ++i) {
#pragma unroll
        for (int k = 0; k < kStep; ++k) acc[i] |= f[k][i];
        open |= (st.al[i] & ~(vv[i] | acc[i])) != 0;
      }
      const unsigned om = __ballot_sync(0xffffffffu, act && open);
      e += kStep;
      left -= kStep;
      const bool fin = act && (left <= 0 || !(om & gmask));
      if (__any_sync(0xffffffffu, fin)) {
        u64 g[WL];
#pragma unroll
        for (int i = 0; i < WL; ++i) g[i] = acc[i] & ~vv[i];
        bu_close<W>(p, st, fin, v, deg, vv, g, Fn, fbn, level);
        if (fin) act = false;
      }
    }
    // ---- vertices that take the whole warp
    for (int h = 0; h < nh; ++h) {
      const int at = kList - 1 - h;
      const int hv = lv[at];
      const unsigned hb = lb[at], hd = (unsigned)ld[at];
      u64 need[WL];
      ld_words<WL>(p.vis + (size_t)hv * W + gl * WL, vv);
      bool open = false;
#pragma unroll
      for (int i = 0; i < WL; ++i) {
        need[i] = st.al[i] & ~vv[i];
        acc[i] = 0ull;
        open |= need[i] != 0;
      }
      if (__any_sync(0xffffffffu, open)) warp_pull<W>(p, Fc, sparse, hb, (int)hd, need, acc);
      u64 g[WL];
#pragma unroll
      for (int i = 0; i < WL; ++i) g[i] = acc[i] & need[i];
      bu_close<W>(p, st, lane < G, hv, hd, vv, g, Fn, fbn, level);
    }
  }
}

// Zeroes frontier L-1's words and bitmap (its ring slot is the next level's
// output): over its queue when it has one, else over its bitmap.
template <int W>
__device__ void retire(const Params<W>& p, long long f, bool queued) {
  u64* F = p.F[f % 3];
  uint32_t* fb = p.fbm[f % 3];
  const long long gtid = blockIdx.x * (long long)kBlock + threadIdx.x, nth = (long long)gridDim.x * kBlock;
  if (queued) {
    const unsigned cnt = (unsigned)(ld_cg_u64(&p.ctl->q[f & 3]) & kCountMask);
    const int* ids = p.qids[f & 3];
    for (long long i = gtid; i < cnt; i += nth) {
      const int u = ids[i];
#pragma unroll
      for (int w = 0; w < W; ++w) F[(size_t)u * W + w] = 0ull;
      fb[u >> 5] = 0u;
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  for (long long w = gtid >> 5; w < p.nwords; w += nth >> 5) {
    const uint32_t bits = ld_cg_u32(fb + w);
    if (!bits) continue;
    // the W words of every vertex in order over the lanes
    for (int k = lane; k < 32 * W; k += 32)
      if ((bits >> (k / W)) & 1u) F[(size_t)w * 32 * W + k] = 0ull;
    __syncwarp();
    if (lane == 0) fb[w] = 0u;
  }
}

template <int W>
__global__ void __launch_bounds__(kBlock, 2) k_msbfs(Params<W> p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  constexpr int WL = Geo<W>::WL, G = Geo<W>::G;
  Ctl* ctl = p.ctl;
  const uint32_t nb = gridDim.x;
  const int lane = threadIdx.x & 31;
  const long long gtid = blockIdx.x * (long long)kBlock + threadIdx.x, nth = (long long)gridDim.x * kBlock;
  long long m_done_total = 0;  // thread 0 only
  uint32_t epoch = 0;
  long long L = 0;
  bool qv = true, qvp = true;  // frontier L, frontier L-1 have a queue
  if (p.resume) {
    L = ctl->r_level;
    m_done_total = ctl->r_done;
    qv = ctl->r_qv != 0;
    qvp = ctl->r_qvp != 0;
  }
  for (;; ++L) {
    const int s0 = (int)(L & 3), s1 = (int)((L + 1) & 3), s2 = (int)((L + 2) & 3);
    if (threadIdx.x < W) {
      sm.alive[threadIdx.x] = ld_cg_u64(&ctl->alive[s0][threadIdx.x]);
      sm.next_alive[threadIdx.x] = 0ull;
    }
    if (threadIdx.x == 0) {
      const u64 pk = ld_cg_u64(&ctl->q[s0]);
      const u64 bn = ld_cg_u64(&ctl->n_f[s0]), bm = ld_cg_u64(&ctl->m_f[s0]);
      const u64 dn = L > 0 ? ld_cg_u64(&ctl->m_done[(L - 1) & 3]) : 0ull;
      const u64 n_f = qv ? (pk & kCountMask) : bn, m_f = qv ? (pk >> 31) : bm;
      int d = -1;  // empty frontier: finished
      if (n_f > 0) {
        if (L + 1 >= p.level_cap) {
          d = -2;
          if (blockIdx.x == 0) {
            ctl->more = 1;
            ctl->r_level = L;
            ctl->r_done = m_done_total;
            ctl->r_qv = qv;
            ctl->r_qvp = qvp;
          }
        } else {
          m_done_total += (long long)dn;
          const long long m_u = p.m_active - m_done_total;
          if (p.force == 0 || !p.allow_bu)
            d = 0;
          else if (p.force == 1)
            d = 1;
          else
            d = ((double)m_f * (double)p.alpha > (double)(m_u + p.bu_fixed)) ? 1 : 0;
          sm.sparse = (double)m_f * 2.0 < (double)p.m_active;
          sm.few = m_u * 8 < p.m_active;
          if (L >= p.max_levels) {
            atomicCAS(&ctl->bar.err, 0, (int)XBFS_ERR_INTERNAL);
            d = -2;
          } else if (blockIdx.x == 0) {
            ctl->strat_count[d] += 1;
          }
        }
      }
      sm.decision = d;
      sm.cnt_m = pk;
    }
    __syncthreads();
    const int D = sm.decision;
    if (D < 0) break;
    const u64* Fc = p.F[L % 3];
    u64* Fn = p.F[(L + 1) % 3];
    uint32_t* fbn = p.fbm[(L + 1) % 3];
    // ring slots of level L+2 (last used at level L-2)
    if (blockIdx.x == 0 && threadIdx.x < 8) {
      ctl->alive[s2][threadIdx.x] = 0ull;
      if (threadIdx.x == 0) {
        ctl->q[s2] = 0ull;
        ctl->n_f[s2] = 0ull;
        ctl->m_f[s2] = 0ull;
        ctl->m_done[s2] = 0ull;
        ctl->tick[s2] = 0u;
      }
    }
    if (L > 0) retire(p, L - 1, qvp);
    // The top plane of level 2^k is zeroed before any bit of it is set: planes
    // 1 and 2, which nearly every traversal reaches, during the level before;
    // the others when their level is sure to exist, behind a barrier of its own.
    const bool late = L >= 7;
    if (late ? ((L + 1) & L) == 0 : (L == 0 || L == 2)) {
      ulonglong2* z = reinterpret_cast<ulonglong2*>(plane(p, 31 - __clz((int)(late ? L + 1 : L + 2))));
      for (long long i = gtid; i < p.ps / 2; i += nth) z[i] = make_ulonglong2(0ull, 0ull);
      if (late && !grid_sync(&ctl->bar, nb, epoch, p.timeout_ns)) return;
    }
    const int level = (int)(L + 1);
    bool next_q;
    if (D == 0) {
      if (!qv) {
        // frontier L came from a bottom-up level: its bitmap becomes a queue
        const uint32_t* fb = p.fbm[L % 3];
        for (long long w = gtid >> 5; w < p.nwords; w += nth >> 5) {
          const uint32_t bits = ld_cg_u32(fb + w);
          if (!bits) continue;
          const bool have = (bits >> lane) & 1u;
          const int v = (int)(w * 32) + lane;
          long long deg = 0;
          unsigned b0 = 0;
          if (have) {
            const long long x = ld_nc_i64(p.beg + v);
            deg = ld_nc_i64(p.beg + v + 1) - x;
            b0 = (unsigned)x;
          }
          warp_enqueue(p, s0, have, v, deg, b0);
        }
        if (!grid_sync(&ctl->bar, nb, epoch, p.timeout_ns)) return;
        if (threadIdx.x == 0) sm.cnt_m = ld_cg_u64(&ctl->q[s0]);
        __syncthreads();
        qv = true;
      }
      long long m_done = 0;
      ms_td<W>(p, sm, s0, s1, Fc, Fn, fbn, level, m_done);
      if (W == 1) {
        m_done = warp_sum(m_done);
        if (lane == 0 && m_done) atomicAdd(&ctl->m_done[s0], (u64)m_done);
      }
      __syncthreads();
      next_q = true;
    } else {
      Bu<W> st;
      st.n_f = st.m_f = st.m_done = 0;
#pragma unroll
      for (int i = 0; i < WL; ++i) {
        st.al[i] = sm.alive[(lane % G) * WL + i];
        st.ga[i] = 0ull;
      }
      // frontiers that hold under half of the edges: most neighbours have no
      // frontier bits, and their bitmap word is 1/16 of a W = 8 read (level 1
      // of 512 sources on R-MAT scale 22: 1.84 -> 1.42 ms)
      const uint32_t* sparse = sm.sparse ? p.fbm[L % 3] : nullptr;
      const unsigned nt = ctl->n_tasks;
      // words per ticket: at least eight tickets per warp (balance) while many
      // edges are left to search, one ticket per warp (few atomics and
      // dependent loads) when only words without work or with little of it are
      const long long warps = (long long)nb * kWarps;
      const bool few = sm.few;
      long long per = few ? (p.nwords + warps - 1) / warps : p.nwords / (warps * 8);
      per = per < 1 ? 1 : (few ? (per > 32 ? 32 : per) : (per > kTicketWords ? kTicketWords : per));
      const unsigned tb = few ? 32 : 4;
      const unsigned tt = (nt + tb - 1) / tb;
      const long long total = tt + (p.nwords + per - 1) / per;
      for (;;) {
        unsigned t = 0;
        if (lane == 0) t = atomicAdd(&ctl->tick[s0], 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        if ((long long)t >= total) break;
        if (t < tt) {
          bu_chunks<W>(p, st, Fc, sparse, Fn, fbn, level, t * tb, min(nt, (t + 1) * tb));
        } else {
          const long long w0 = (long long)(t - tt) * per;
          bu_words<W>(p, sm, st, Fc, sparse, Fn, fbn, level, w0, (int)(p.nwords - w0 < per ? p.nwords - w0 : per));
        }
      }
#pragma unroll
      for (int i = 0; i < WL; ++i) {
#pragma unroll
        for (int o = G; o < 32; o <<= 1) st.ga[i] |= __shfl_xor_sync(0xffffffffu, st.ga[i], o);
        if (lane < G && st.ga[i]) atomicOr(&sm.next_alive[lane * WL + i], st.ga[i]);
      }
      long long x[3] = {st.n_f, st.m_f, st.m_done};
      block_sum_n<kBlock, 3, long long>(x, sm.red);
      if (threadIdx.x == 0) {
        if (x[0]) atomicAdd(&ctl->n_f[s1], (u64)x[0]);
        if (x[1]) atomicAdd(&ctl->m_f[s1], (u64)x[1]);
        if (x[2]) atomicAdd(&ctl->m_done[s0], (u64)x[2]);
      }
      next_q = false;
    }
    if (threadIdx.x < W && sm.next_alive[threadIdx.x])
      atomicOr(&ctl->alive[s1][threadIdx.x], sm.next_alive[threadIdx.x]);
    if (!grid_sync(&ctl->bar, nb, epoch, p.timeout_ns)) return;
    qvp = qv;
    qv = next_q;
  }
  if (sm.decision == -1) {
    // the last frontier's words and bitmap go back to zero for the next call
    if (L > 0) retire(p, L - 1, qvp);
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->depth = (int)L;
  }
}

// Start state: visited words and plane 0 zero, done = isolated vertices (or
// nothing on a directed CSR), and the chunks of the longest lists.
template <int W>
__global__ void k_ms_init(Params<W> p) {
  const long long gtid = blockIdx.x * (long long)blockDim.x + threadIdx.x, nth = (long long)gridDim.x * blockDim.x;
  ulonglong2* a = reinterpret_cast<ulonglong2*>(p.vis);
  ulonglong2* b = reinterpret_cast<ulonglong2*>(p.lo);
  for (long long i = gtid; i < p.ps / 2; i += nth) a[i] = b[i] = make_ulonglong2(0ull, 0ull);
  for (long long i = gtid; i < p.nwords; i += nth) p.done[i] = p.symmetric ? p.iso[i] : 0u;
  if (!p.have_mega) return;
  for (long long v = gtid; v < p.V; v += nth) {
    const long long d = p.beg[v + 1] - p.beg[v];
    if (d <= kMega) continue;
    const unsigned nch = (unsigned)((d + kMega - 1) >> kMegaLog);
    const unsigned i = atomicAdd(&p.ctl->n_mega, 1u), t = atomicAdd(&p.ctl->n_tasks, nch);
    p.mega_v[i] = (int)v;
    for (unsigned c = 0; c < nch; ++c) p.tasks[t + c] = make_uint2(i, c);
  }
}

// Seeds source s (bit s) at its vertex; sources that share a vertex share its
// queue entry (the first to set the vertex's frontier bit appends it).
template <int W>
__global__ void k_ms_seed(Params<W> p, Seeds sd) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  bool have = false;
  int v = 0;
  long long deg = 0;
  unsigned b0 = 0;
  if (s < sd.n) {
    v = sd.v[s];
    const int w = s >> 6;
    const u64 bit = 1ull << (s & 63);
    atomicOr(p.vis + (size_t)v * W + w, bit);
    const long long x = p.beg[v];
    deg = p.beg[v + 1] - x;
    b0 = (unsigned)x;
    if (deg > 0) {
      atomicOr(p.F[0] + (size_t)v * W + w, bit);
      atomicOr(&p.ctl->alive[0][w], bit);
      have = !((atomicOr(p.fbm[0] + (v >> 5), 1u << (v & 31)) >> (v & 31)) & 1u);
    }
  }
  warp_enqueue(p, 0, have, v, deg, b0);
}

// 4 bits to 4 bytes (0 or 1 each).
__device__ __forceinline__ uint32_t spread4(uint32_t x) { return (x * 0x00204081u) & 0x01010101u; }
// Byte j of x, sign-extended.
template <int J>
__device__ __forceinline__ int sbyte(uint32_t x) {
  int r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(x), "n"(J | (J | 8) << 4 | (J | 8) << 8 | (J | 8) << 12));
  return r;
}

// Level rows of 32 vertices (one per lane) and the 64 sources of one word:
// out[s * stride + v]. P planes, levels below 128 (P <= 7): four sources'
// levels are assembled in the bytes of one register, 0xff where the source
// did not reach the vertex.
template <int P>
__device__ __forceinline__ void expand_word(const u64* pl, size_t pstride, u64 vis, int n, int* out, size_t stride,
                                            bool in) {
  u64 x[P];
#pragma unroll
  for (int k = 0; k < P; ++k) x[k] = in ? *(pl + k * pstride) : 0ull;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t nv = (uint32_t)(~vis >> (32 * h));
    uint32_t y[P];
#pragma unroll
    for (int k = 0; k < P; ++k) y[k] = (uint32_t)(x[k] >> (32 * h));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int s = 32 * h + 4 * j;
      if (s >= n) return;
      uint32_t a = spread4((nv >> (4 * j)) & 15u) * 255u;
#pragma unroll
      for (int k = 0; k < P; ++k) a |= spread4((y[k] >> (4 * j)) & 15u) << k;
      if (in) {
        int* o = out + (size_t)s * stride;
        __stcs(o, sbyte<0>(a));
        if (s + 1 < n) __stcs(o + stride, sbyte<1>(a));
        if (s + 2 < n) __stcs(o + 2 * stride, sbyte<2>(a));
        if (s + 3 < n) __stcs(o + 3 * stride, sbyte<3>(a));
      }
    }
  }
}

// Visited words and level planes -> per-source int32 rows, coalesced over
// the vertices, and the degree sum of all reached (vertex, source) pairs.
// Does nothing while the traversal is unfinished. Bound by the row writes (512
// rows of R-MAT scale 22: 8.6 GB written, 1.1 GB read), and those by how many
// rows are written side by side: one CTA of 512 threads per SM that keeps to
// one row takes 1.6 ms, four CTAs of 256 free-running threads 1.9, eight 2.6.
//
// The largest level is depth - 1 where every reached vertex has an edge, as on
// a symmetric CSR. On a directed one the last frontier may reach only vertices
// without out-edges, which get level `depth` and form no frontier of their own;
// that level was processed, so the plane of its top bit has been zeroed.
__global__ void __launch_bounds__(kExpand, 1)
    k_ms_expand(const u64* vis, const u64* lo, const u64* hi, int W, size_t ps, long long V, const long long* beg, int n,
                int* out, size_t stride, int symmetric, Ctl* ctl) {
  __shared__ long long red[kExpand / 32 + 1];
  const int depth = ctl->depth;
  if (depth == 0 && (ctl->more || ctl->bar.err)) return;
  const int top = symmetric ? depth - 1 : depth;  // no level is above it
  const int P = top > 1 ? 32 - __clz(top) : 1;
  const long long v = blockIdx.x * (long long)kExpand + threadIdx.x;
  const bool in = v < V;
  long long reached = 0;
  const int wn = (n + 63) / 64;
  for (int w = 0; w < wn; ++w) {
    __syncthreads();  // keeps the CTA on the same rows: 2 KB runs per row
    const size_t idx = (size_t)v * W + w;
    const u64 x = in ? vis[idx] : 0ull;
    reached += __popcll(x);
    int* o = out + (size_t)w * 64 * stride + v;
    const int nn = min(64, n - w * 64);
    switch (P) {
      case 1: expand_word<1>(lo + idx, ps, x, nn, o, stride, in); break;
      case 2: expand_word<2>(lo + idx, ps, x, nn, o, stride, in); break;
      case 3: expand_word<3>(lo + idx, ps, x, nn, o, stride, in); break;
      case 4: expand_word<4>(lo + idx, ps, x, nn, o, stride, in); break;
      case 5: expand_word<5>(lo + idx, ps, x, nn, o, stride, in); break;
      case 6: expand_word<6>(lo + idx, ps, x, nn, o, stride, in); break;
      case 7: expand_word<7>(lo + idx, ps, x, nn, o, stride, in); break;
      default:
        if (in)
          for (int s = 0; s < nn; ++s) {
            int lv = -1;
            if ((x >> s) & 1ull) {
              lv = 0;
              for (int k = 0; k < P; ++k) {
                const u64 y = k < kLoPlanes ? lo[k * ps + idx] : hi[(k - kLoPlanes) * ps + idx];
                lv |= (int)((y >> s) & 1ull) << k;
              }
            }
            o[(size_t)s * stride] = lv;
          }
    }
  }
  const long long sum = block_sum<kExpand, long long>(in ? reached * (beg[v + 1] - beg[v]) : 0, red);
  if (threadIdx.x == 0 && sum) atomicAdd(&ctl->msum, (u64)sum);
}

}  // namespace ms

// ---------------------------------------------------------------------------
// Host driver
// ---------------------------------------------------------------------------
// Two allocations hold a traversal's buffers, the upper level planes excepted: an
// allocation and its release take 0.3 ms and more each, whatever their size, and a
// program that loads one graph after another pays both for every graph (R-MAT
// scale 18, 64 sources: 5.7 -> 1.1 ms for the first call, 5.7 -> 1.9 to
// free the graph, with 25 allocations and with two). What has to be zero when a
// traversal starts lies in one of its own, so that graphs and words per vertex of
// other sizes find zeros wherever their buffers are in it. (With both in one
// allocation 512 sources on R-MAT scale 21 took 3.334 ms, not 3.316.)
struct MsWorkspace {
  int device = 0;
  DevBuf zero, rest, hi;
  bool clean = false;  // `zero` is all zero (what a finished traversal leaves)
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  ~MsWorkspace() {
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
  }
};

// Idle workspaces. A call takes one (or makes a new one) and gives it back
// when its stream is through, so calls of several threads, graphs and streams
// never share one; at most kMsIdle stay allocated per device while graphs
// exist, none after the last graph handle is freed.
constexpr size_t kMsIdle = 2;
static std::mutex g_ms_mu;
static std::vector<std::unique_ptr<MsWorkspace>>& ms_idle() {
  static auto* v = new std::vector<std::unique_ptr<MsWorkspace>>();  // outlives the CUDA context: never destroyed
  return *v;
}
static int g_ms_graphs = 0;

void ms_graph_created() {
  std::lock_guard<std::mutex> lk(g_ms_mu);
  ++g_ms_graphs;
}

void ms_graph_freed() {
  std::vector<std::unique_ptr<MsWorkspace>> drop;
  {
    std::lock_guard<std::mutex> lk(g_ms_mu);
    if (--g_ms_graphs == 0) drop.swap(ms_idle());
  }
  for (auto& w : drop) {
    DeviceGuard dg(w->device);
    w.reset();
  }
}

namespace {
struct MsLease {
  std::unique_ptr<MsWorkspace> w;
  cudaStream_t s;
  MsLease(int device, cudaStream_t stream) : s(stream) {
    {
      std::lock_guard<std::mutex> lk(g_ms_mu);
      auto& idle = ms_idle();
      for (size_t i = idle.size(); i-- > 0;)
        if (idle[i]->device == device) {
          w = std::move(idle[i]);
          idle.erase(idle.begin() + (ptrdiff_t)i);
          break;
        }
    }
    if (!w) {
      w.reset(new MsWorkspace());
      w->device = device;
    }
  }
  ~MsLease() {
    if (cudaStreamSynchronize(s) != cudaSuccess) return;  // a faulted context: nothing to keep
    std::lock_guard<std::mutex> lk(g_ms_mu);
    auto& idle = ms_idle();
    size_t have = 0;
    for (auto& x : idle) have += x->device == w->device;
    if (have < kMsIdle && g_ms_graphs > 0) idle.push_back(std::move(w));
  }
};
}  // namespace

template <int W>
static xbfs_status run_pass(Graph* g, const int32_t* srcs, int n, int* d_out, size_t out_stride, float alpha,
                            int force, cudaStream_t s, int* depth, int* strat, unsigned long long* msum,
                            MsWorkspace& w) {
  const long long V = g->V;
  const long long nwords = (V + 31) / 32;
  const size_t ps = ((size_t)V * W + 1) & ~(size_t)1;
  const size_t words = ps * 8;  // one word set per vertex, in bytes
  const size_t bm = (size_t)(nwords + 64) * 4;
  const bool bu = g->symmetric;
  const size_t n_mega = bu ? (size_t)g->cnt_deg_gt[ms::kMegaLog] : 0;
  const size_t n_tasks = n_mega ? n_mega + ((size_t)g->E >> ms::kMegaLog) : 0;
  xbfs_status st;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t o = at;
    at += (bytes + 255) & ~(size_t)255;
    return o;
  };
  // the buffers that a finished traversal leaves all zero
  const size_t rows = words + 64;  // and one zero row past the last vertex
  size_t o_F[3], o_fbm[3], o_q[4][3];
  for (auto& o : o_F) o = take(rows);
  for (auto& o : o_fbm) o = take(bm);
  const size_t o_mega_n = take(n_mega * 4), o_mega_acc = take(n_mega * W * 8);
  const size_t nz = at;
  at = 0;
  const size_t o_vis = take(words), o_lo = take(words * ms::kLoPlanes), o_done = take(bm),
               o_ctl = take(sizeof(ms::Ctl)), o_mega_v = take(n_mega * 4), o_tasks = take(n_tasks * 8);
  for (auto& q : o_q)
    for (auto& o : q) o = take((size_t)V * 4 + 4);
  // a new allocation is not clean, wherever it lies: cudaMalloc may give it the
  // place of the one just freed
  if (nz > w.zero.bytes) w.clean = false;
  if ((st = w.zero.ensure(nz)) || (st = w.rest.ensure(at))) return st;
  char* const zero = w.zero.as<char>();
  char* const rest = w.rest.as<char>();
  if (!w.clean) XBFS_CUDA_TRY(cudaMemsetAsync(zero, 0, w.zero.bytes, s));
  w.clean = false;  // until this traversal has finished
  ms::Params<W> p;
  memset(&p, 0, sizeof(p));
  p.beg = g->beg.as<long long>();
  p.csr = g->csr.as<int>();
  p.V = V;
  p.E = g->E;
  p.vis = reinterpret_cast<ms::u64*>(rest + o_vis);
  for (int i = 0; i < 3; ++i) {
    p.F[i] = reinterpret_cast<ms::u64*>(zero + o_F[i]);
    p.fbm[i] = reinterpret_cast<uint32_t*>(zero + o_fbm[i]);
  }
  p.ps = (long long)ps;
  p.lo = reinterpret_cast<ms::u64*>(rest + o_lo);
  p.done = reinterpret_cast<uint32_t*>(rest + o_done);
  for (int i = 0; i < 4; ++i) {
    p.qids[i] = reinterpret_cast<int*>(rest + o_q[i][0]);
    p.qeb[i] = reinterpret_cast<unsigned*>(rest + o_q[i][1]);
    p.qbg[i] = reinterpret_cast<unsigned*>(rest + o_q[i][2]);
  }
  p.mega_v = reinterpret_cast<int*>(rest + o_mega_v);
  p.tasks = reinterpret_cast<uint2*>(rest + o_tasks);
  p.mega_n = reinterpret_cast<unsigned*>(zero + o_mega_n);
  p.mega_acc = reinterpret_cast<ms::u64*>(zero + o_mega_acc);
  p.ctl = reinterpret_cast<ms::Ctl*>(rest + o_ctl);
  p.nwords = nwords;
  p.m_active = g->E;
  // The single-source default (0.1) means "use the batched default". An edge
  // of a top-down level (64 bytes of visited words, up to eight atomics)
  // costs what 11 edges of a bottom-up level cost at W = 8 and 7 at W = 1
  // (R-MAT scale 22, 512 sources: 161 against 14 ps; scale 18, 64 sources: 50
  // against 6.7 ps), and a bottom-up level reads V/32 words and offsets
  // whatever the frontier.
  p.alpha = alpha > 0.5f ? alpha : 12.0f;
  p.bu_fixed = alpha > 0.5f ? 0 : V / 4;
  p.allow_bu = bu ? 1 : 0;
  p.force = force;
  p.symmetric = bu ? 1 : 0;
  p.have_mega = n_mega ? 1 : 0;
  p.level_cap = 255;
  p.timeout_ns = 20ull * 1000 * 1000 * 1000;
  p.max_levels = V + 2;
  p.iso = g->iso.as<uint32_t>();
  ms::Seeds sd;
  sd.n = n;
  memcpy(sd.v, srcs, sizeof(int) * (size_t)n);
  const void* kfn = (const void*)ms::k_msbfs<W>;
  const size_t smem = sizeof(ms::Smem);
  XBFS_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int nsm = 0, per_sm = 0;
  XBFS_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, g->device));
  XBFS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, ms::kBlock, smem));
  if (per_sm < 1) return set_error(XBFS_ERR_INTERNAL, "batched kernel cannot be resident");
  XBFS_CUDA_TRY(cudaMemsetAsync(p.ctl, 0, sizeof(ms::Ctl), s));
  ms::k_ms_init<W><<<(unsigned)std::min<long long>((V * W / 2 + 255) / 256 + 1, nsm * 8), 256, 0, s>>>(p);
  ms::k_ms_seed<W><<<(n + 127) / 128, 128, 0, s>>>(p, sd);
  XBFS_CUDA_TRY(cudaGetLastError());
  ms::Ctl hc;
  for (;;) {
    void* args[] = {&p};
    XBFS_CUDA_TRY(cudaLaunchCooperativeKernel(kfn, dim3(nsm * per_sm), dim3(ms::kBlock), args, smem, s));
    ms::k_ms_expand<<<(unsigned)((V + ms::kExpand - 1) / ms::kExpand), ms::kExpand, 0, s>>>(
        p.vis, p.lo, p.hi, W, p.ps, V, p.beg, n, d_out, out_stride, p.symmetric, p.ctl);
    XBFS_CUDA_TRY(cudaGetLastError());
    XBFS_CUDA_TRY(cudaMemcpyAsync(&hc, p.ctl, sizeof(hc), cudaMemcpyDeviceToHost, s));
    XBFS_CUDA_TRY(cudaStreamSynchronize(s));
    if (hc.bar.err)
      return set_error((xbfs_status)hc.bar.err, "batched traversal kernel reported %s", xbfs_strerror(hc.bar.err));
    if (!hc.more) break;
    if (p.hi) return set_error(XBFS_ERR_LEVEL_OVERFLOW, "batched traversal kernel reported %s",
                               xbfs_strerror(XBFS_ERR_LEVEL_OVERFLOW));
    // deeper than the low eight planes hold: allocate the others, carry on
    if ((st = w.hi.ensure(words * (ms::kMaxPlanes - ms::kLoPlanes)))) return st;
    p.hi = w.hi.as<ms::u64>();
    p.level_cap = 65535;
    p.resume = 1;
    XBFS_CUDA_TRY(cudaMemsetAsync(p.ctl, 0, sizeof(GridBarrier), s));
    XBFS_CUDA_TRY(cudaMemsetAsync(&p.ctl->more, 0, sizeof(int), s));
  }
  w.clean = true;
  *depth = std::max(*depth, hc.depth);
  strat[0] += hc.strat_count[0];
  strat[1] += hc.strat_count[1];
  *msum += hc.msum;
  return XBFS_OK;
}

xbfs_status bfs_batch(Graph* g, const int32_t* srcs, int32_t n, int32_t* levels, const xbfs_opts* uo,
                      xbfs_stats* stats, int words_per_vertex) {
  const auto t_start = std::chrono::steady_clock::now();
  if (!g || !srcs || !levels || n <= 0) return set_error(XBFS_ERR_INVALID_ARG, "bad arguments");
  for (int i = 0; i < n; ++i)
    if (srcs[i] < 0 || srcs[i] >= g->V) return set_error(XBFS_ERR_INVALID_ARG, "source %d out of range", srcs[i]);
  if (g->E >= (1ll << 32)) return set_error(XBFS_ERR_UNSUPPORTED, "batched path needs E < 2^32");
  xbfs_opts o;
  xbfs_opts_init(&o);
  if (uo) {
    if (uo->struct_size != (int32_t)sizeof(xbfs_opts)) return set_error(XBFS_ERR_INVALID_ARG, "bad opts struct_size");
    o = *uo;
  }
  int force = -1;
  if (o.policy == XBFS_POLICY_FORCED && o.forced && o.n_forced > 0) force = (o.forced[0] == XBFS_BU) ? 1 : 0;
  int W = words_per_vertex;
  if (W <= 0) W = n > 256 ? 8 : (n > 128 ? 4 : (n > 64 ? 2 : 1));
  if (W != 1 && W != 2 && W != 4 && W != 8) return set_error(XBFS_ERR_INVALID_ARG, "words per vertex must be 1, 2, 4 or 8");
  DeviceGuard dg(g->device);
  cudaStream_t s = o.stream ? (cudaStream_t)o.stream : g->stream;
  MsLease lease(g->device, s);
  MsWorkspace& w = *lease.w;
  const bool dev_out = is_device_pointer(levels);
  const int per_pass = 64 * W;
  DevBuf tmp_out;
  xbfs_status st;
  int* d_out = levels;
  if (!dev_out) {
    if ((st = tmp_out.ensure((size_t)std::min(n, per_pass) * g->V * 4))) return st;
    d_out = tmp_out.as<int>();
  }
  if (!w.e0) XBFS_CUDA_TRY(cudaEventCreate(&w.e0));
  if (!w.e1) XBFS_CUDA_TRY(cudaEventCreate(&w.e1));
  unsigned long long msum = 0;
  float total_ms = 0;
  int depth = 0, strat[2] = {0, 0};
  for (int s0 = 0; s0 < n; s0 += per_pass) {
    const int cnt = std::min(per_pass, n - s0);
    int* out = dev_out ? levels + (size_t)s0 * g->V : d_out;
    XBFS_CUDA_TRY(cudaEventRecord(w.e0, s));
    switch (W) {
      case 1: st = run_pass<1>(g, srcs + s0, cnt, out, g->V, o.alpha, force, s, &depth, strat, &msum, w); break;
      case 2: st = run_pass<2>(g, srcs + s0, cnt, out, g->V, o.alpha, force, s, &depth, strat, &msum, w); break;
      case 4: st = run_pass<4>(g, srcs + s0, cnt, out, g->V, o.alpha, force, s, &depth, strat, &msum, w); break;
      default: st = run_pass<8>(g, srcs + s0, cnt, out, g->V, o.alpha, force, s, &depth, strat, &msum, w); break;
    }
    if (st) return st;
    XBFS_CUDA_TRY(cudaEventRecord(w.e1, s));
    XBFS_CUDA_TRY(cudaEventSynchronize(w.e1));
    float ms = 0;
    cudaEventElapsedTime(&ms, w.e0, w.e1);
    total_ms += ms;
    if (!dev_out)
      XBFS_CUDA_TRY(cudaMemcpyAsync(levels + (size_t)s0 * g->V, d_out, (size_t)cnt * g->V * 4, cudaMemcpyDeviceToHost, s));
  }
  XBFS_CUDA_TRY(cudaStreamSynchronize(s));
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    stats->struct_size = (int32_t)sizeof(xbfs_stats);
    stats->depth = depth;
    stats->edges_mc = (int64_t)(msum / 2);
    stats->device_ms = total_ms;
    stats->kernel_ms = total_ms;
    stats->n_td_queue = strat[0];
    stats->n_bu = strat[1];
    stats->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
  }
  return XBFS_OK;
}

}  // namespace xbfs

using namespace xbfs;

extern "C" {

xbfs_status xbfs_bfs_batch(xbfs_graph* g, const int32_t* srcs, int32_t n, int32_t* levels, const xbfs_opts* opts,
                           xbfs_stats* stats) {
  return bfs_batch((Graph*)g, srcs, n, levels, opts, stats, 0);
}

xbfs_status xbfs_bfs_batch_w(xbfs_graph* g, const int32_t* srcs, int32_t n, int32_t* levels, const xbfs_opts* opts,
                             xbfs_stats* stats, int32_t words_per_vertex) {
  return bfs_batch((Graph*)g, srcs, n, levels, opts, stats, words_per_vertex);
}

}  // extern "C"
