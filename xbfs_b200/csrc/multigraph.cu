// Multi-graph BFS: many graphs of uneven size, one source each, in one
// persistent launch, replayed from a CUDA graph.
//
// No counterpart in the reference (one graph per process). B200 design:
//  * All graphs live in one arena (offsets per graph); a work list sorted by
//    edge count (largest first) is consumed through an atomic ticket, so the
//    big graphs start first and the small ones fill the gaps
//    (longest-processing-time order).
//  * Graphs of more than kBig vertices and edges are taken by teams of 8 to
//    64 CTAs: bitmaps in global memory (L2), levels separated by a barrier of the
//    team, the frontier copied to every CTA's shared memory for bottom-up
//    probes, vertices of long lists shared by the whole team. When no such
//    graph is left, the CTAs of a team go on singly.
//  * Each other graph is owned by one CTA for its whole traversal: visited /
//    current / next frontier bitmaps sit in shared memory (3 x 32 KB), so every
//    status probe is a shared-memory access and levels are separated by
//    __syncthreads.
//  * Each level picks top-down or bottom-up from its own counts. Top-down
//    expands frontier vertices of degree <= `thread_max` one per lane and
//    heavier ones warp-cooperatively; bottom-up gives each lane one unvisited
//    vertex and stops at the first parent.
//  * The CTA shape (threads per CTA), the thread/warp degree threshold and the
//    direction threshold are picked by a small autotuner (xbfs_multi_tune);
//    before that, teams and single CTAs have thresholds of their own.
#include <string.h>

#include <algorithm>
#include <chrono>
#include <memory>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "internal.hpp"

namespace xbfs {

namespace mg {

// CTAs per team (at least, at most), and the vertices plus edges above which a
// graph is a team's. Teams are as large as lets all big graphs run side by
// side: 16 graphs (up to R-MAT scale 18) take 0.55 ms in teams of 8 and 0.36 in
// teams of 16, 96 graphs 0.86 and 1.07.
constexpr int kTeamMin = 8, kTeamMax = 64;
constexpr long long kBig = 1 << 17;
constexpr int kHeavy = 1024;  // a team shares the edges of vertices above this degree
constexpr unsigned long long kTimeoutNs = 10ull * 1000 * 1000 * 1000;

// One team's state. Counters are rings by level: a level reads its own slot,
// adds to the next one and clears the one after that.
struct Team {
  GridBarrier bar;
  int graph;                    // ticket drawn for the team
  unsigned heavy[4];            // length of the list of long vertices
  unsigned long long n[4], m[4];  // frontier vertices, degree sum
};

struct Thresholds {
  int thread_max;  // top-down: degree <= thread_max expanded by one lane
  float alpha;     // bottom-up when m_f * alpha > m_u
  bool operator==(const Thresholds& o) const { return thread_max == o.thread_max && alpha == o.alpha; }
};

struct Desc {
  long long b_off;   // offset of the graph's V+1 local offsets in the beg arena
  long long e_off;   // offset of its neighbours in the csr arena
  long long v_off;   // offset of its levels in the output arena
  int V;
  int src;
  long long E;
};

struct Params {
  const long long* beg;   // local offsets, per graph
  const int* csr;         // local vertex ids
  const Desc* desc;
  const int* order;       // graph indices, largest first
  int n;
  int* levels;            // concatenated outputs
  unsigned* ticket;
  int n_big;              // the first n_big graphs of `order` are the teams'
  int team;               // CTAs per team
  Team* teams;
  uint32_t* bits;         // per team: visited and three frontier bitmaps of team_words words
  long long team_words;
  int* heavy;             // per team: list of long vertices, heavy_cap entries
  long long heavy_cap;
  int* err;               // status of the launch
  int smem_words;         // words per bitmap available in shared memory
  Thresholds single, by_team;  // of graphs owned by one CTA, and by a team
  unsigned long long* edges;  // per graph: sum of degrees of reached vertices
};

template <int BLOCK>
__device__ __forceinline__ long long block_sum_ll(long long v, long long* red) {
  return block_sum<BLOCK, long long>(v, red);
}

// One claimed edge of a team's top-down level.
__device__ __forceinline__ void team_claim(uint32_t* vis, uint32_t* nxt, const long long* beg, int* lv, int v, int level,
                                           long long& n, long long& m) {
  const uint32_t bit = 1u << (v & 31);
  if (ld_cg_u32(vis + (v >> 5)) & bit) return;
  if (atomicOr(vis + (v >> 5), bit) & bit) return;
  red_or_u32(nxt + (v >> 5), bit);
  lv[v] = level;
  n += 1;
  m += __ldg(beg + v + 1) - __ldg(beg + v);
}

// Four edges of a lane, their targets read together.
__device__ __forceinline__ void team_claim4(const int* csr, long long e, long long step, long long e1, uint32_t* vis,
                                            uint32_t* nxt, const long long* beg, int* lv, int level, long long& n,
                                            long long& m) {
  int v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = e + k * step < e1 ? __ldg(csr + e + k * step) : -1;
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = v[k] >= 0 ? ld_cg_u32(vis + (v[k] >> 5)) : ~0u;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (v[k] >= 0 && !((w[k] >> (v[k] & 31)) & 1u)) team_claim(vis, nxt, beg, lv, v[k], level, n, m);
}

// One graph by a team of p.team CTAs (rank: this CTA's place in it). False:
// the time limit of a barrier ran out.
template <int BLOCK>
__device__ bool team_bfs(const Params& p, Team* team, uint32_t* bits, int* heavy, int rank, uint32_t& epoch, int gi,
                         uint32_t* sbits, long long* red, int* s_decision, long long* s_mu) {
  constexpr int NW = BLOCK / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const Desc d = p.desc[p.order[gi]];
  const long long* beg = p.beg + d.b_off;
  const int* csr = p.csr + d.e_off;
  int* lv = p.levels + d.v_off;
  const int nw = (d.V + 31) / 32;
  uint32_t* vis = bits;
  uint32_t* fr[3] = {bits + p.team_words, bits + 2 * p.team_words, bits + 3 * p.team_words};
  const int src = d.src;
  // CTA ranks take words in turn, a warp's worth of words each (all of them
  // see dense and sparse parts of the vertex range)
  const int T = p.team;
  const int gw = wid * T + rank;  // this warp among the team's
  const int GW = NW * T;
  for (int w = rank * BLOCK + threadIdx.x; w < nw; w += T * BLOCK) {
    const uint32_t own = (w == (src >> 5)) ? 1u << (src & 31) : 0u;
    vis[w] = own | ((w == nw - 1 && (d.V & 31)) ? ~((1u << (d.V & 31)) - 1u) : 0u);
    fr[0][w] = own;
    fr[1][w] = 0u;
    fr[2][w] = 0u;
  }
  if (rank == 0 && threadIdx.x == 0) {
    lv[src] = 0;
    team->n[0] = 1ull;
    team->m[0] = (unsigned long long)(beg[src + 1] - beg[src]);
    for (int k = 1; k < 4; ++k) team->n[k] = team->m[k] = 0ull;
    for (int k = 0; k < 4; ++k) team->heavy[k] = 0u;
  }
  if (threadIdx.x == 0) *s_mu = d.E;
  if (!grid_sync(&team->bar, (uint32_t)p.team, epoch, kTimeoutNs)) return false;
  unsigned long long reached = 0;  // thread 0 of rank 0
  for (int L = 0;; ++L) {
    if (threadIdx.x == 0) {
      const long long n_f = (long long)ld_cg_u64(&team->n[L & 3]), m_f = (long long)ld_cg_u64(&team->m[L & 3]);
      *s_mu -= m_f;
      reached += (unsigned long long)m_f;
      *s_decision = n_f == 0 ? -1 : ((double)m_f * (double)p.by_team.alpha > (double)*s_mu ? 1 : 0);
      if (rank == 0) {
        team->n[(L + 2) & 3] = team->m[(L + 2) & 3] = 0ull;
        team->heavy[(L + 2) & 3] = 0u;
      }
    }
    __syncthreads();
    const int dec = *s_decision;
    if (dec < 0) break;
    const uint32_t* cur = fr[L % 3];
    uint32_t* nxt = fr[(L + 1) % 3];
    uint32_t* old = fr[(L + 2) % 3];
    long long my_n = 0, my_m = 0;
    // frontier L-1's bitmap becomes frontier L+2's
    for (int w = rank * BLOCK + threadIdx.x; w < nw; w += T * BLOCK) old[w] = 0u;
    if (dec == 1) {
      // ---- bottom-up over the frontier's bitmap in shared memory
      const bool staged = nw <= 3 * p.smem_words;
      if (staged) {
        for (int w = threadIdx.x; w < nw; w += BLOCK) sbits[w] = ld_cg_u32(cur + w);
        __syncthreads();
      }
      const uint32_t* f = staged ? sbits : cur;
      for (int w = gw; w < nw; w += GW) {
        const uint32_t un = ~ld_cg_u32(vis + w);
        if (!un) continue;
        const int v = w * 32 + lane;
        bool found = false, more = false;
        long long e0 = 0, e1 = 0;
        if ((un >> lane) & 1u) {
          e0 = __ldg(beg + v);
          e1 = __ldg(beg + v + 1);
          const long long d0 = e1 - e0;
          // up to eight neighbours by the lane itself, four at a time
          for (long long e = e0; e < e1 && e < e0 + 8 && !found; e += 4) {
            int u[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) u[k] = e + k < e1 ? __ldg(csr + e + k) : -1;
#pragma unroll
            for (int k = 0; k < 4; ++k) found = found || (u[k] >= 0 && ((f[u[k] >> 5] >> (u[k] & 31)) & 1u));
          }
          more = !found && d0 > 8;
          e0 += 8;
        }
        // the rest of the longer lists by the whole warp, one after another
        unsigned rest = __ballot_sync(0xffffffffu, more);
        while (rest) {
          const int hl = __ffs(rest) - 1;
          rest &= rest - 1;
          const long long h1 = __shfl_sync(0xffffffffu, e1, hl);
          for (long long e = __shfl_sync(0xffffffffu, e0, hl); e < h1; e += 64) {
            bool hit = false;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const long long x = e + k * 32 + lane;
              const int u = x < h1 ? __ldg(csr + x) : -1;
              hit = hit || (u >= 0 && ((f[u >> 5] >> (u & 31)) & 1u));
            }
            if (__any_sync(0xffffffffu, hit)) {
              if (lane == hl) found = true;
              break;
            }
          }
        }
        if (found) {
          lv[v] = L + 1;
          my_n += 1;
          my_m += __ldg(beg + v + 1) - __ldg(beg + v);
        }
        const unsigned got = __ballot_sync(0xffffffffu, found);
        if (lane == 0 && got) {
          nxt[w] = got;
          vis[w] = ~un | got;
        }
      }
      __syncthreads();
    } else {
      // ---- top-down
      unsigned* hc = &team->heavy[L & 3];
      for (int w = gw; w < nw; w += GW) {
        const uint32_t mine_bits = ld_cg_u32(cur + w);
        if (!mine_bits) continue;
        const int u = w * 32 + lane;
        const bool mine = (mine_bits >> lane) & 1u;
        long long e0 = 0, e1 = 0;
        if (mine) {
          e0 = __ldg(beg + u);
          e1 = __ldg(beg + u + 1);
        }
        const long long deg = e1 - e0;
        if (mine && deg <= p.by_team.thread_max)
          for (long long e = e0; e < e1; e += 4) team_claim4(csr, e, 1, e1, vis, nxt, beg, lv, L + 1, my_n, my_m);
        if (mine && deg > p.by_team.thread_max && deg > kHeavy) {
          const unsigned at = atomicAdd(hc, 1u);
          heavy[at] = u;
        }
        unsigned mid = __ballot_sync(0xffffffffu, mine && deg > p.by_team.thread_max && deg <= kHeavy);
        while (mid) {
          const int hl = __ffs(mid) - 1;
          mid &= mid - 1;
          const long long h0 = __shfl_sync(0xffffffffu, e0, hl), h1 = __shfl_sync(0xffffffffu, e1, hl);
          for (long long e = h0 + lane; e < h1; e += 128)
            team_claim4(csr, e, 32, h1, vis, nxt, beg, lv, L + 1, my_n, my_m);
        }
      }
      if (!grid_sync(&team->bar, (uint32_t)p.team, epoch, kTimeoutNs)) return false;
      const unsigned nh = ld_cg_u32(hc);
      for (unsigned h = 0; h < nh; ++h) {
        const int u = (int)ld_cg_u32(reinterpret_cast<const uint32_t*>(heavy + h));
        const long long h0 = __ldg(beg + u), h1 = __ldg(beg + u + 1);
        const long long step = (long long)T * BLOCK;
        for (long long e = h0 + rank * BLOCK + threadIdx.x; e < h1; e += 4 * step)
          team_claim4(csr, e, step, h1, vis, nxt, beg, lv, L + 1, my_n, my_m);
      }
    }
    long long x[2] = {my_n, my_m};
    block_sum_n<BLOCK, 2, long long>(x, red);
    if (threadIdx.x == 0 && x[0]) {
      atomicAdd(&team->n[(L + 1) & 3], (unsigned long long)x[0]);
      atomicAdd(&team->m[(L + 1) & 3], (unsigned long long)x[1]);
    }
    if (!grid_sync(&team->bar, (uint32_t)p.team, epoch, kTimeoutNs)) return false;
  }
  if (rank == 0 && threadIdx.x == 0) p.edges[p.order[gi]] = reached;
  __syncthreads();
  return true;
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_multi(Params p) {
  extern __shared__ __align__(16) uint32_t sbits[];
  __shared__ long long red[2 * (BLOCK / 32) + 1];
  __shared__ int s_g;
  __shared__ long long s_mu;
  __shared__ unsigned long long s_nf, s_mf;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr int NW = BLOCK / 32;
  // ---- the teams' graphs: the team's first CTA draws the tickets
  if (p.n_big > 0) {
    const int t = blockIdx.x / p.team, rank = blockIdx.x % p.team;
    Team* team = p.teams + t;
    uint32_t epoch = 0;
    bool ok = true;
    for (;;) {
      if (rank == 0 && threadIdx.x == 0) team->graph = (int)atomicAdd(p.ticket + 1, 1u);
      ok = grid_sync(&team->bar, (uint32_t)p.team, epoch, kTimeoutNs);
      if (!ok) break;
      if (threadIdx.x == 0) s_g = ld_acquire_i32(&team->graph);
      __syncthreads();
      const int gi = s_g;
      if (gi >= p.n_big) break;
      ok = team_bfs<BLOCK>(p, team, p.bits + (size_t)t * 4 * p.team_words, p.heavy + (size_t)t * p.heavy_cap, rank,
                           epoch, gi, sbits, red, &s_g, &s_mu);
      if (!ok) break;
    }
    if (!ok) {
      if (threadIdx.x == 0) atomicCAS(p.err, 0, (int)XBFS_ERR_DEVICE_TIMEOUT);
      return;
    }
    __syncthreads();
  }
  for (;;) {
    if (threadIdx.x == 0) s_g = p.n_big + (int)atomicAdd(p.ticket, 1u);
    __syncthreads();
    const int gi = s_g;
    if (gi >= p.n) break;
    const Desc d = p.desc[p.order[gi]];
    const int V = d.V;
    const long long* beg = p.beg + d.b_off;
    const int* csr = p.csr + d.e_off;
    int* lv = p.levels + d.v_off;
    const int nw = (V + 31) / 32;
    // volatile: a word that another thread changes by an atomic is read anew
    volatile uint32_t* vis = sbits;
    volatile uint32_t* cur = sbits + p.smem_words;
    volatile uint32_t* nxt = sbits + 2 * p.smem_words;
    for (int w = threadIdx.x; w < nw; w += BLOCK) {
      // bits past V count as visited so they are never searched
      const uint32_t tail = (w == nw - 1 && (V & 31)) ? ~((1u << (V & 31)) - 1u) : 0u;
      vis[w] = tail;
      cur[w] = 0u;
      nxt[w] = 0u;
    }
    __syncthreads();
    const int src = d.src;
    long long m_u = d.E;
    unsigned long long reached_deg = 0;
    if (threadIdx.x == 0) {
      vis[src >> 5] |= 1u << (src & 31);
      cur[src >> 5] |= 1u << (src & 31);
      lv[src] = 0;
      const long long dg = beg[src + 1] - beg[src];
      s_nf = 1;
      s_mf = (unsigned long long)dg;
    }
    __syncthreads();
    long long n_f = (long long)s_nf, m_f = (long long)s_mf;
    reached_deg = (unsigned long long)m_f;
    m_u -= m_f;
    int L = 0;
    while (n_f > 0) {
      const bool bu = (double)m_f * (double)p.single.alpha > (double)m_u;
      long long my_n = 0, my_m = 0;
      if (!bu) {
        // top-down: warps take frontier words; light vertices one per lane,
        // heavy ones warp-cooperatively
        for (int w = wid; w < nw; w += NW) {
          const uint32_t bits = cur[w];
          if (!bits) continue;
          const int u_l = w * 32 + lane;
          const bool mine = (bits >> lane) & 1u;
          long long e0 = 0, e1 = 0;
          if (mine) {
            e0 = __ldg(beg + u_l);
            e1 = __ldg(beg + u_l + 1);
          }
          const bool light = mine && (e1 - e0) <= p.single.thread_max;
          if (light) {
            for (long long e = e0; e < e1; ++e) {
              const int v = __ldg(csr + e);
              const uint32_t bit = 1u << (v & 31);
              if (vis[v >> 5] & bit) continue;
              if (atomicOr((uint32_t*)&vis[v >> 5], bit) & bit) continue;
              atomicOr((uint32_t*)&nxt[v >> 5], bit);
              lv[v] = L + 1;
              my_n += 1;
              my_m += __ldg(beg + v + 1) - __ldg(beg + v);
            }
          }
          unsigned heavy = __ballot_sync(0xffffffffu, mine && !light);
          while (heavy) {
            const int hl = __ffs(heavy) - 1;
            heavy &= heavy - 1;
            const long long h0 = __shfl_sync(0xffffffffu, e0, hl), h1 = __shfl_sync(0xffffffffu, e1, hl);
            for (long long e = h0 + lane; e < h1; e += 32) {
              const int v = __ldg(csr + e);
              const uint32_t bit = 1u << (v & 31);
              if (vis[v >> 5] & bit) continue;
              if (atomicOr((uint32_t*)&vis[v >> 5], bit) & bit) continue;
              atomicOr((uint32_t*)&nxt[v >> 5], bit);
              lv[v] = L + 1;
              my_n += 1;
              my_m += __ldg(beg + v + 1) - __ldg(beg + v);
            }
          }
        }
      } else {
        // bottom-up: lanes own unvisited vertices of a word
        for (int w = wid; w < nw; w += NW) {
          const uint32_t un = ~vis[w];
          if (!un) continue;
          const int v = w * 32 + lane;
          if ((un >> lane) & 1u) {
            const long long e0 = __ldg(beg + v), e1 = __ldg(beg + v + 1);
            for (long long e = e0; e < e1; ++e) {
              const int u = __ldg(csr + e);
              if ((cur[u >> 5] >> (u & 31)) & 1u) {
                lv[v] = L + 1;
                atomicOr((uint32_t*)&nxt[w], 1u << lane);
                my_n += 1;
                my_m += e1 - e0;
                break;
              }
            }
          }
        }
        __syncthreads();
        // newly found vertices become visited only after the sweep, so every
        // probe above saw the level-L frontier only
        for (int w = threadIdx.x; w < nw; w += BLOCK) vis[w] |= nxt[w];
      }
      const long long tn = block_sum_ll<BLOCK>(my_n, red);
      const long long tm = block_sum_ll<BLOCK>(my_m, red);
      // next frontier becomes current
      for (int w = threadIdx.x; w < nw; w += BLOCK) {
        cur[w] = nxt[w];
        nxt[w] = 0u;
      }
      __syncthreads();
      n_f = tn;
      m_f = tm;
      m_u -= tm;
      reached_deg += (unsigned long long)tm;
      ++L;
    }
    if (threadIdx.x == 0) p.edges[p.order[gi]] = reached_deg;
    __syncthreads();
  }
}

}  // namespace mg

struct MultiGraph {
  int device = 0;
  int n = 0;
  long long total_V = 0, total_E = 0;
  int n_big = 0;                 // graphs for teams, first in `horder`
  int max_teams = 0;             // teams the buffers are laid out for
  long long team_words = 0, heavy_cap = 0;
  size_t ctl_teams = 0;          // offset of the teams in ctl
  DevBuf beg, csr, desc, order, ctl, bits, heavy, srcs_dev, levels_tmp;
  std::vector<mg::Desc> hdesc;
  std::vector<int> horder;
  PinnedBuf srcs_pin, ctl_pin;
  cudaStream_t stream = nullptr;
  // tuned configuration
  int block = 512;
  // Before tuning. Teams: with 8 and 14 a set of 96 graphs takes 0.86 ms, with 32
  // and 4 1.40. One CTA: 30 graphs of up to 2^12 vertices take 218 us with 8 and
  // 14, 171 with 32 and 4 and 155 with 8 and 4; 128 of them 267, 243 and 221; 12
  // uniform random ones of 14,000 vertices 353, 320 and 289; 12 grids of 100 x 90
  // 995, 855 and 883. A configuration that was tuned or set is both's.
  mg::Thresholds single = {8, 4.f}, by_team = {8, 14.f};
  // captured replay
  cudaGraphExec_t exec = nullptr;
  int* exec_levels = nullptr;
  int exec_block = 0;
  mg::Thresholds exec_single = {0, 0.f}, exec_by_team = {0, 0.f};
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  ~MultiGraph() {
    DeviceGuard dg(device);
    if (exec) cudaGraphExecDestroy(exec);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (stream) cudaStreamDestroy(stream);
  }
};

// 3 x 32 KB: a single CTA's bitmaps of up to 262,144 vertices (larger graphs
// are the teams', as kBig is below that).
constexpr int kSmemWords = 8192;
static_assert(mg::kBig <= 32ll * kSmemWords, "graphs too large for shared memory must be the teams'");
// Control buffer, cleared before every launch: two tickets (single CTAs,
// teams) and the launch status; from kCtlEdges the graphs' edge counts; then
// the teams. What lies before the teams is copied to the host after it.
constexpr size_t kCtlEdges = 64;

static xbfs_status enqueue_multi(MultiGraph* m, int* d_levels, int block, const mg::Thresholds& single,
                                 const mg::Thresholds& by_team) {
  cudaStream_t s = m->stream;
  XBFS_CUDA_TRY(cudaMemsetAsync(d_levels, 0xff, (size_t)m->total_V * 4, s));
  XBFS_CUDA_TRY(cudaMemsetAsync(m->ctl.p, 0, m->ctl.bytes, s));
  // the per-graph sources are patched into the descriptors on the device
  mg::Params p;
  p.beg = m->beg.as<long long>();
  p.csr = m->csr.as<int>();
  p.desc = m->desc.as<mg::Desc>();
  p.order = m->order.as<int>();
  p.n = m->n;
  p.levels = d_levels;
  p.ticket = m->ctl.as<unsigned>();
  p.err = m->ctl.as<int>() + 2;
  p.teams = reinterpret_cast<mg::Team*>(m->ctl.as<char>() + m->ctl_teams);
  p.n_big = m->n_big;
  p.team = 1;
  p.bits = m->bits.as<uint32_t>();
  p.team_words = m->team_words;
  p.heavy = m->heavy.as<int>();
  p.heavy_cap = m->heavy_cap;
  p.smem_words = kSmemWords;
  p.single = single;
  p.by_team = by_team;
  p.edges = reinterpret_cast<unsigned long long*>(m->ctl.as<char>() + kCtlEdges);
  const size_t smem = (size_t)3 * p.smem_words * 4;
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, m->device);
  const void* kfn;
  switch (block) {
    case 256: kfn = (const void*)mg::k_multi<256>; break;
    case 1024: kfn = (const void*)mg::k_multi<1024>; break;
    default: kfn = (const void*)mg::k_multi<512>; block = 512; break;
  }
  XBFS_CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  XBFS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, block, smem));
  if (per_sm < 1) return set_error(XBFS_ERR_INTERNAL, "multi-graph kernel cannot be resident");
  void* args[] = {&p};
  if (m->n_big > 0) {
    // whole teams, all resident (their CTAs wait for one another); no more
    // teams than can have work
    const int slots = nsm * per_sm;
    p.team = mg::kTeamMin;
    while (p.team < mg::kTeamMax && 2 * p.team * m->n_big <= slots) p.team *= 2;
    const int single = (m->n - m->n_big + p.team - 1) / p.team;
    const int teams = std::min({slots / p.team, m->n_big + single, m->max_teams});
    if (teams < 1) return set_error(XBFS_ERR_INTERNAL, "multi-graph kernel cannot be resident");
    XBFS_CUDA_TRY(cudaLaunchCooperativeKernel(kfn, dim3(teams * p.team), dim3(block), args, smem, s));
  } else {
    XBFS_CUDA_TRY(cudaLaunchKernel(kfn, dim3(std::min(nsm * per_sm, m->n)), dim3(block), args, smem, s));
  }
  return XBFS_OK;
}

__global__ void k_mg_set_sources(mg::Desc* desc, const int* srcs, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) desc[i].src = srcs[i];
}

// One call: copy sources, patch descriptors, reset outputs, run. Captured into
// a CUDA graph on first use and replayed while the output pointer and the
// configuration stay the same.
static xbfs_status run_multi(MultiGraph* m, int* d_levels, int block, const mg::Thresholds& single,
                             const mg::Thresholds& by_team, float* ms_out) {
  cudaStream_t s = m->stream;
  const bool reuse = m->exec && m->exec_levels == d_levels && m->exec_block == block &&
                     m->exec_single == single && m->exec_by_team == by_team;
  if (!reuse) {
    if (m->exec) {
      cudaGraphExecDestroy(m->exec);
      m->exec = nullptr;
    }
    cudaGraph_t graph;
    XBFS_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    xbfs_status st = XBFS_OK;
    {
      cudaError_t e = cudaMemcpyAsync(m->srcs_dev.p, m->srcs_pin.p, sizeof(int) * m->n, cudaMemcpyHostToDevice, s);
      if (e == cudaSuccess) {
        k_mg_set_sources<<<(m->n + 255) / 256, 256, 0, s>>>(m->desc.as<mg::Desc>(), m->srcs_dev.as<int>(), m->n);
        e = cudaGetLastError();
      }
      if (e != cudaSuccess) st = set_error(XBFS_ERR_CUDA, "capture: %s", cudaGetErrorString(e));
      if (!st) st = enqueue_multi(m, d_levels, block, single, by_team);
      if (!st) {
        e = cudaMemcpyAsync(m->ctl_pin.p, m->ctl.p, m->ctl_teams, cudaMemcpyDeviceToHost, s);
        if (e != cudaSuccess) st = set_error(XBFS_ERR_CUDA, "capture: %s", cudaGetErrorString(e));
      }
    }
    cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (st) {
      if (ce == cudaSuccess) cudaGraphDestroy(graph);
      return st;
    }
    XBFS_CUDA_TRY(ce);
    cudaError_t ie = cudaGraphInstantiate(&m->exec, graph, 0);
    cudaGraphDestroy(graph);
    XBFS_CUDA_TRY(ie);
    m->exec_levels = d_levels;
    m->exec_block = block;
    m->exec_single = single;
    m->exec_by_team = by_team;
  }
  XBFS_CUDA_TRY(cudaEventRecord(m->e0, s));
  XBFS_CUDA_TRY(cudaGraphLaunch(m->exec, s));
  XBFS_CUDA_TRY(cudaEventRecord(m->e1, s));
  XBFS_CUDA_TRY(cudaEventSynchronize(m->e1));
  float ms = 0;
  XBFS_CUDA_TRY(cudaEventElapsedTime(&ms, m->e0, m->e1));
  if (ms_out) *ms_out = ms;
  const int err = m->ctl_pin.as<int>()[2];
  if (err) return set_error((xbfs_status)err, "multi-graph kernel reported %s", xbfs_strerror(err));
  return XBFS_OK;
}

}  // namespace xbfs

using namespace xbfs;

extern "C" {

xbfs_status xbfs_multi_create(xbfs_graph* const* graphs, int32_t n, int32_t device, xbfs_multi** out) {
  if (!graphs || n <= 0 || !out) return set_error(XBFS_ERR_INVALID_ARG, "bad arguments");
  *out = nullptr;
  std::unique_ptr<MultiGraph> m(new MultiGraph());
  m->device = device;
  m->n = n;
  DeviceGuard dg(device);
  m->hdesc.resize(n);
  long long vb = 0, bb = 0, eb = 0;
  for (int i = 0; i < n; ++i) {
    const Graph* g = (const Graph*)graphs[i];
    if (!g) return set_error(XBFS_ERR_INVALID_ARG, "graph %d is NULL", i);
    if (g->device != device) return set_error(XBFS_ERR_INVALID_ARG, "graph %d lives on device %d", i, g->device);
    if (!g->symmetric) return set_error(XBFS_ERR_UNSUPPORTED, "graph %d is not symmetric", i);
    if (g->V > INT32_MAX - 64) return set_error(XBFS_ERR_UNSUPPORTED, "graph %d too large", i);
    m->hdesc[i] = mg::Desc{bb, eb, vb, (int)g->V, 0, g->E};
    vb += g->V;
    bb += g->V + 1;
    eb += g->E;
  }
  m->total_V = vb;
  m->total_E = eb;
  xbfs_status st;
  if ((st = m->beg.ensure((size_t)bb * 8)) || (st = m->csr.ensure((size_t)eb * 4 + 64)) ||
      (st = m->desc.ensure(sizeof(mg::Desc) * n)) || (st = m->order.ensure(sizeof(int) * n)) ||
      (st = m->srcs_dev.ensure(4 * (size_t)n)) ||
      (st = m->srcs_pin.ensure(4 * (size_t)n)))
    return st;
  XBFS_CUDA_TRY(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
  XBFS_CUDA_TRY(cudaEventCreate(&m->e0));
  XBFS_CUDA_TRY(cudaEventCreate(&m->e1));
  for (int i = 0; i < n; ++i) {
    const Graph* g = (const Graph*)graphs[i];
    XBFS_CUDA_TRY(cudaMemcpyAsync(m->beg.as<long long>() + m->hdesc[i].b_off, g->beg.p, (size_t)(g->V + 1) * 8,
                                  cudaMemcpyDeviceToDevice, m->stream));
    if (g->E > 0)
      XBFS_CUDA_TRY(cudaMemcpyAsync(m->csr.as<int>() + m->hdesc[i].e_off, g->csr.p, (size_t)g->E * 4,
                                    cudaMemcpyDeviceToDevice, m->stream));
  }
  m->horder.resize(n);
  std::iota(m->horder.begin(), m->horder.end(), 0);
  std::stable_sort(m->horder.begin(), m->horder.end(), [&](int a, int b) {
    return m->hdesc[a].E + m->hdesc[a].V > m->hdesc[b].E + m->hdesc[b].V;
  });
  XBFS_CUDA_TRY(cudaMemcpyAsync(m->desc.p, m->hdesc.data(), sizeof(mg::Desc) * n, cudaMemcpyHostToDevice, m->stream));
  XBFS_CUDA_TRY(cudaMemcpyAsync(m->order.p, m->horder.data(), sizeof(int) * n, cudaMemcpyHostToDevice, m->stream));
  // the teams' bitmaps and lists, for as many teams as a launch may have
  long long big_v = 0, big_long = 0;
  for (int i = 0; i < n; ++i) {
    const mg::Desc& d = m->hdesc[i];
    if (d.E + d.V <= mg::kBig) continue;
    ++m->n_big;
    big_v = std::max<long long>(big_v, d.V);
    big_long = std::max<long long>(big_long, ((const Graph*)graphs[i])->cnt_deg_gt[10]);
  }
  if (m->n_big > 0) {
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
    m->max_teams = std::max(1, nsm * 2 / mg::kTeamMin);  // shared memory admits two CTAs per SM
    m->team_words = (big_v + 31) / 32;
    m->heavy_cap = big_long + 1;
    if ((st = m->bits.ensure((size_t)m->max_teams * 4 * (size_t)m->team_words * 4)) ||
        (st = m->heavy.ensure((size_t)m->max_teams * (size_t)m->heavy_cap * 4)))
      return st;
  }
  m->ctl_teams = (kCtlEdges + 8 * (size_t)n + 63) & ~(size_t)63;
  if ((st = m->ctl.ensure(m->ctl_teams + sizeof(mg::Team) * (size_t)m->max_teams)) ||
      (st = m->ctl_pin.ensure(m->ctl_teams)))
    return st;
  XBFS_CUDA_TRY(cudaStreamSynchronize(m->stream));
  *out = (xbfs_multi*)m.release();
  return XBFS_OK;
}

xbfs_status xbfs_multi_info(const xbfs_multi* mh, int64_t* total_V, int64_t* total_E, int64_t* level_offsets) {
  const MultiGraph* m = (const MultiGraph*)mh;
  if (!m) return set_error(XBFS_ERR_INVALID_ARG, "NULL handle");
  if (total_V) *total_V = m->total_V;
  if (total_E) *total_E = m->total_E;
  if (level_offsets)
    for (int i = 0; i < m->n; ++i) level_offsets[i] = m->hdesc[i].v_off;
  return XBFS_OK;
}

xbfs_status xbfs_multi_bfs(xbfs_multi* mh, const int32_t* srcs, int32_t* levels, const xbfs_opts* opts,
                           xbfs_stats* stats) {
  MultiGraph* m = (MultiGraph*)mh;
  if (!m || !srcs || !levels) return set_error(XBFS_ERR_INVALID_ARG, "NULL argument");
  (void)opts;
  for (int i = 0; i < m->n; ++i)
    if (srcs[i] < 0 || srcs[i] >= m->hdesc[i].V) return set_error(XBFS_ERR_INVALID_ARG, "source of graph %d out of range", i);
  DeviceGuard dg(m->device);
  const auto t0 = std::chrono::steady_clock::now();
  memcpy(m->srcs_pin.p, srcs, sizeof(int) * m->n);
  const bool dev = is_device_pointer(levels);
  int* d_levels = levels;
  xbfs_status st;
  if (!dev) {
    if ((st = m->levels_tmp.ensure((size_t)m->total_V * 4))) return st;
    d_levels = m->levels_tmp.as<int>();
  }
  float ms = 0;
  if ((st = run_multi(m, d_levels, m->block, m->single, m->by_team, &ms))) return st;
  if (!dev) XBFS_CUDA_TRY(cudaMemcpy(levels, d_levels, (size_t)m->total_V * 4, cudaMemcpyDeviceToHost));
  if (stats) {
    const unsigned long long* e = reinterpret_cast<unsigned long long*>(m->ctl_pin.as<char>() + kCtlEdges);
    memset(stats, 0, sizeof(*stats));
    stats->struct_size = (int32_t)sizeof(xbfs_stats);
    unsigned long long tot = 0;
    for (int i = 0; i < m->n; ++i) tot += e[i] / 2;
    stats->edges_mc = (int64_t)tot;
    stats->device_ms = ms;
    stats->kernel_ms = ms;
    stats->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  }
  return XBFS_OK;
}

// Autotuner: times every (threads per CTA, thread/warp degree threshold,
// direction threshold) candidate on the caller's sources and keeps the
// fastest. Returns the chosen configuration, of the two kinds of graph the one of
// single CTAs where they differ.
xbfs_status xbfs_multi_tune(xbfs_multi* mh, const int32_t* srcs, int32_t reps, int32_t* block_out,
                            int32_t* thread_max_out, float* alpha_out, float* best_ms_out) {
  MultiGraph* m = (MultiGraph*)mh;
  if (!m || !srcs) return set_error(XBFS_ERR_INVALID_ARG, "NULL argument");
  DeviceGuard dg(m->device);
  memcpy(m->srcs_pin.p, srcs, sizeof(int) * m->n);
  xbfs_status st;
  if ((st = m->levels_tmp.ensure((size_t)m->total_V * 4))) return st;
  const int blocks[] = {256, 512, 1024};
  const int tms[] = {8, 32, 128};
  const float alphas[] = {2.f, 4.f, 14.f};
  float best = 1e30f;
  int bb = m->block;
  mg::Thresholds bs = m->single, bt = m->by_team;
  if (reps < 1) reps = 1;
  auto time_one = [&](int b, const mg::Thresholds& single, const mg::Thresholds& by_team) -> xbfs_status {
    float tot = 0;
    for (int r = 0; r < reps + 1; ++r) {
      float ms = 0;
      if (xbfs_status e = run_multi(m, m->levels_tmp.as<int>(), b, single, by_team, &ms)) return e;
      if (r > 0) tot += ms;  // first run builds the graph
    }
    tot /= reps;
    if (tot < best) {
      best = tot;
      bb = b;
      bs = single;
      bt = by_team;
    }
    return XBFS_OK;
  };
  // the configuration that is there, whose two kinds of graph may differ, then
  // every common one
  if ((st = time_one(m->block, m->single, m->by_team))) return st;
  for (int b : blocks)
    for (int t : tms)
      for (float a : alphas)
        if ((st = time_one(b, {t, a}, {t, a}))) return st;
  m->block = bb;
  m->single = bs;
  m->by_team = bt;
  if (block_out) *block_out = bb;
  if (thread_max_out) *thread_max_out = bs.thread_max;
  if (alpha_out) *alpha_out = bs.alpha;
  if (best_ms_out) *best_ms_out = best;
  return XBFS_OK;
}

xbfs_status xbfs_multi_set_config(xbfs_multi* mh, int32_t block, int32_t thread_max, float alpha) {
  MultiGraph* m = (MultiGraph*)mh;
  if (!m) return set_error(XBFS_ERR_INVALID_ARG, "NULL handle");
  if (block != 256 && block != 512 && block != 1024) return set_error(XBFS_ERR_INVALID_ARG, "block must be 256/512/1024");
  if (thread_max < 0 || !(alpha > 0)) return set_error(XBFS_ERR_INVALID_ARG, "bad threshold");
  m->block = block;
  m->single = m->by_team = {thread_max, alpha};
  return XBFS_OK;
}

void xbfs_multi_free(xbfs_multi* mh) { delete (MultiGraph*)mh; }

}  // extern "C"
