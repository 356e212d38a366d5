// narrow.cuh -- a traversal with a small frontier, run by ONE thread-block
// cluster (up to 16 CTAs): BFS (every edge counts 1) and SSSP (uint32 weights).
//
// A level of a few thousand edges costs a whole-GPU persistent kernel 9-14 us
// of grid barriers and dependent loads whatever its size.  Here a step's cost
// is one chain of loads inside one CTA, and what is small is kept on chip:
//   * Work entries {v, begin, end, d} -- up to kPiece out-edges of v, reached
//     at distance d -- sit in shared memory.  Vertex v has a home CTA
//     (contiguous ranges of ids); a vertex improved by its home goes to that
//     CTA's next list, one improved elsewhere to its home's inbox through
//     distributed shared memory.
//   * A CTA runs up to kRounds rounds over what its own rounds produce, with
//     block barriers only, before the cluster barrier that makes the inboxes
//     readable: graphs whose ids follow their geometry (grids, road networks,
//     chains) cross the cluster barrier once per kRounds levels.
//   * Distances are lowered by atomicMin in L2 (the one L2 round trip that a
//     round waits for besides its adjacency loads); an entry whose d is no
//     longer v's distance is skipped.  Rounds of different CTAs may run at
//     different depths, so a vertex can be expanded again when a shorter path
//     arrives later; distances below the threshold T bound how far ahead a
//     CTA can get.  Whatever the schedule, the fixpoint -- the shortest
//     distances -- is the same.
//   * Distances of T and above wait in a far list per CTA (global memory);
//     when no CTA has near work, T advances to the smallest far distance plus
//     Delta (one cluster barrier), so all distances below the old T are final.
// A full list never loses work: its overflow goes to the near or far bitmap.
// The next step relaxes what is in the near bitmap where it stands, all of it
// (the far bitmap waits for the split).  Queued again instead, a vertex of
// several entries might get no further than its first ones every time (one of
// more than 2,097,152 out-edges, or several smaller ones, fill all lists), and a
// frontier wider than the lists would take many steps, each at another depth:
// BFS along a path of 24 vertices into a random graph of 4 M vertices, degree
// 16, 49.8 ms with queueing, 10.1 without.
//
// Which barrier a thread goes to next depends on words that other warps and
// other CTAs write; narrow_steps.h keeps them so that all threads read the same.
//
// Bound by latency: a level of a path of 4,001 vertices takes 1.7 us in BFS and
// 1.8 in SSSP, of which the atomic's round trip is about a third and its quarter
// of a cluster barrier with the words of the step 0.2.  Measured for SSSP with an
// earlier form (a 1,021 x 1,531 grid / a 40 x 3,000 grid / RMAT-12, ms; the grid
// kernel 81 / 88 / 0.29): 512 threads 13.5 / 11.4 / 0.17, 768 threads 10.9 /
// 11.7 / 0.14, 1,024 threads 10.8 / 13.0 / 0.14.  1,024 are kept for the widest
// frontiers (BFS on a 4,096 x 4,096 grid: 32.2, 30.2, 25.4 ms; 25.9 now).  Rounds
// per step, at 512 threads: 2 14.2 / 14.8, 4 12.7 / 14.8, 8 13.6 / 18.5, 16 16.7 /
// 20.8.
#pragma once

#include <cooperative_groups.h>

#include "device_util.cuh"
#include "narrow_steps.h"

namespace grus {
namespace narrow {

namespace cg = cooperative_groups;

constexpr int kBlock = 1024;
constexpr int kWarps = kBlock / 32;
constexpr int kMaxCluster = 16;
constexpr uint32_t kCap = 2048;      // entries of one list
constexpr uint32_t kPiece = 64;      // edges per entry
// Spilled vertices: up to kWideEdges edges go to one CTA, those of more to the
// whole cluster, kWide of them in a step.
constexpr uint32_t kWideEdges = 1024, kWide = 32;
// (Shared has to stay within 131 KB: past it the SM's L1 loses another 32 KB,
// 4,096 x 4,096 grid 25.9 -> 26.6 ms.)
// SSSP: a step that relaxes this many spilled vertices is the grid's work; the
// traversal is handed back.  (A path of 24 vertices into a binary tree of 4 M, ids
// in level order / shuffled: grid kernel alone 1.75 / 1.44 ms, cluster 3.4 / 5.1,
// handed back 1.68 / 2.14.)
constexpr uint32_t kHandBack = 1u << 17;
// Low-degree graphs, few entries: 4 or 8 lanes per entry instead of a scan
// over the entries' degrees (a path's round 1.57 -> 1.04 us with 512 threads;
// entries of up to 64 edges would take 8 serial steps instead: RMAT-12 0.19
// -> 0.25 ms).  0: the scan always.
inline uint32_t lanes_per_entry(uint32_t max_degree) {
  return max_degree <= 4 ? 4u : (max_degree <= 16 ? 8u : 0u);
}
// Whether a graph and its distances (`edge` bytes per edge) are beyond what L2
// keeps: a wave over such a graph fetches the lines ahead of it (BFS on a
// 4,096 x 4,096 grid 31.3 -> 29.1 ms; grids inside L2 lose 5 %).
inline bool beyond_l2(uint64_t n, uint64_t m, uint32_t edge) {
  return 8 * n + edge * m > (96ull << 20);
}
constexpr int kIlp = 2;              // 32-edge steps whose loads are in flight together
constexpr uint32_t kFarCap = 4096;   // most far entries per CTA and buffer, SSSP
constexpr uint32_t kFarCapUnit = 1024;  // ... and BFS
constexpr uint32_t kInf = 4294967294u;
constexpr uint32_t kRing = 128;      // BFS: depth counts, by depth modulo kRing
constexpr uint32_t kUnitDelta = 32;  // BFS: levels per threshold step (<= kRing / 2)

// Far lists of one cluster (2 buffers per CTA) for a graph of n vertices;
// small graphs get short ones, so that a first call's allocation stays small,
// and so does BFS, whose far vertices are those past one threshold's levels.
__host__ __device__ inline uint32_t far_cap(uint64_t n, uint32_t most = kFarCap) {
  return n >= 8ull * most ? most : (n < 512 ? 64u : (uint32_t)(n / 8));
}
inline size_t far_bytes(uint64_t n, uint32_t most = kFarCap) {
  return (size_t)kMaxCluster * 2 * far_cap(n, most) * sizeof(uint2);
}

// Per-step record (SSSP) or per-level record (BFS), the layout of the
// persistent kernels' traces.
struct Trace {
  unsigned long long t_ns, edges;
  uint32_t count, tag;
};

struct View {
  const uint32_t *__restrict__ offs;
  const uint32_t *__restrict__ cols;
  const uint32_t *__restrict__ wts;  // unused by BFS
  uint32_t n, W, m;
  uint32_t *dist;
  uint32_t *near0, *near1;  // even and odd steps' near bitmaps, W words, all zero at the start
  uint32_t *farbm;   // W words, zero but for what farbm_used announces
  uint2 *far;        // far_bytes(n)
  uint32_t far_cap;
  uint32_t delta;
  bool adapt;        // SSSP: delta may grow while threshold steps do little
  uint32_t lanes;    // lanes_per_entry of the graph
  bool ahead;        // low degrees, and beyond_l2
  bool hand_back;    // SSSP: stop at a step of kHandBack spilled vertices
  uint32_t *err;
  uint64_t timeout_ns;  // a step that takes longer ends the traversal
  // null: none.  SSSP: record i is the i-th step's (from 1); BFS: record d
  // counts the vertices of depth d.  Records to be written start out zero.
  Trace *trace;
  uint32_t trace_cap;
  uint32_t tag;      // SSSP: threshold steps taken before
};

// Starts filling this SM's L1 with the line holding p (no wait).
__device__ __forceinline__ void prefetch_l1(const void *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

struct Shared {
  uint4 loc[2][kCap];
  uint4 inb[2][kCap];
  uint32_t cnt[3];                      // local list lengths, rotating by round
  uint32_t incnt[2], farcnt[2];
  AwayCounts away;                      // entries pushed to other CTAs
  // the last step in which this CTA pushed to an inbox, spilled to the near
  // bitmap, put bits in the far bitmap (0: never), ...
  uint32_t pushed, spilled, farbm;
  // ... and rank 0: what the cluster found, by step parity, the last step that
  // put bits in the far bitmap and the last that had far vertices (both read
  // where no CTA can be past the step that wrote them)
  StepWords found[2];
  // taking spilled vertices: entries claimed in the list, the place of the first
  // claim that found no room, each warp's next words, and how many entries of
  // the wide list this CTA has had
  uint32_t claimed, refused, cur[kWarps], had;
  // rank 0, by step parity: spilled vertices that all CTAs relax together
  uint4 wide[2][kWide];
  uint32_t nwide[2], nspilled[2];
  unsigned long long t_step;            // rank 0: when the last step ended
  uint32_t g_farbm, g_far;
  // this CTA's copies: far bitmap bits up to this step have been taken; the
  // last threshold step and its size
  uint32_t scanned, last_split, delta;
  uint32_t min_far;                     // smallest distance of this CTA's far vertices
  uint32_t red[kWarps];
  unsigned long long red64[kWarps];
  int ring[kRing];                      // BFS: labels given minus labels replaced, by depth
  int ring_sum[kRing];                  // rank 0: summed over the cluster
};

struct Result {
  uint32_t steps = 0, splits = 0;
  uint32_t last = 0;                    // BFS: largest depth (valid in rank 0)
  uint32_t visits = 0, nr = 0, mr = 0;  // this thread's share (m < 2^32 bounds the last two)
};

static_assert(sizeof(Shared) <= 131 * 1024, "with 1 KB of the system's, 132 KB");

template <bool kUnit>
struct Engine {
  const View &a;
  Shared *s;
  cg::cluster_group cl;
  uint32_t rank, C, lane, warp;
  uint32_t lane_shift;        // log2 of a.lanes
  uint32_t scale;             // home of v: umulhi(v, scale)
  uint32_t T, step;           // steps count from 1 (0 = never)
  uint32_t cq, lb, fb;        // read: cnt[cq], loc[lb], far buffer fb
  int round;                  // of the step, 0 before its first
  Result res;
  bool handed_back = false;

  __device__ __forceinline__ Engine(const View &view, Shared *sh)
      : a(view), s(sh), cl(cg::this_cluster()) {
    rank = cl.block_rank();
    C = cl.num_blocks();
    lane = lane_id();
    warp = threadIdx.x >> 5;
    lane_shift = a.lanes ? 31 - __clz(a.lanes) : 0;
    const unsigned long long q = ((unsigned long long)C << 32) / max(a.n, 1u);
    scale = q > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)q;
    T = 0;
    step = 1;
    cq = lb = fb = 0;
    round = 0;
    if (threadIdx.x < 3) s->cnt[threadIdx.x] = 0u;
    if (threadIdx.x < 2) s->incnt[threadIdx.x] = s->farcnt[threadIdx.x] = 0u;
    if (threadIdx.x < kRounds) s->away.n[0][threadIdx.x] = s->away.n[1][threadIdx.x] = 0u;
    if (threadIdx.x < kRing) s->ring[threadIdx.x] = s->ring_sum[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
      s->pushed = s->spilled = s->farbm = s->g_farbm = 0u;
      s->found[0] = s->found[1] = StepWords{0u, 0u, 0u, 0u};
      s->nwide[0] = s->nwide[1] = s->nspilled[0] = s->nspilled[1] = 0u;
      s->t_step = global_timer_ns();
      s->g_far = 0u;
      s->scanned = s->last_split = 0u;
      s->delta = a.delta;
    }
  }

  // Which inbox is read in this step; the other one is written.
  __device__ __forceinline__ uint32_t ip() const { return (step & 1u) ^ 1u; }
  __device__ __forceinline__ uint32_t home(uint32_t v) const { return __umulhi(v, scale); }

  // The near bitmap that this step's pushes spill to.
  __device__ __forceinline__ uint32_t *near_of(uint32_t st) const {
    return st & 1u ? a.near1 : a.near0;
  }

  __device__ __forceinline__ void spill(uint32_t v) {
    atomicOr(near_of(step) + (v >> 5), 1u << (v & 31u));
    s->spilled = step;
  }

  // Queues the vertices u (edges [b,e), distance d) of the lanes with `want`:
  // one entry at its home, or pieces of kPiece edges dealt over the cluster
  // (kBig; without it no vertex has more).  Called by whole warps.
  template <bool kBig>
  __device__ __forceinline__ void push(bool want, uint32_t u, uint32_t b, uint32_t e, uint32_t d) {
    want = want && e > b;
    const uint32_t nq = cq == 2 ? 0 : cq + 1;
    const uint32_t o = home(u);
    bool big = kBig && want && e - b > kPiece;
    if (big && *(volatile uint32_t *)&s->cnt[nq] >= kCap) {  // no pieces into full lists
      spill(u);
      want = big = false;
    }
    const bool here = want && !big && o == rank;
    if (here) {
      const uint32_t pos = atomicAdd(&s->cnt[nq], 1u);
      if (pos < kCap) s->loc[lb ^ 1u][pos] = make_uint4(u, b, e, d);
      else spill(u);
    }
    if (__all_sync(0xffffffffu, here == want)) return;
    const bool far_home = want && !big && o != rank;
    const uint32_t mr = __ballot_sync(0xffffffffu, far_home);
    if (far_home) {
      const uint32_t peers = __match_any_sync(mr, o);
      const int leader = __ffs(peers) - 1;
      Shared *r = cl.map_shared_rank(s, o);
      uint32_t base = 0;
      if ((int)lane == leader) {
        base = atomicAdd(&r->incnt[ip() ^ 1u], __popc(peers));
        atomicAdd(&away_in(s->away, step, round), __popc(peers));
      }
      base = __shfl_sync(peers, base, leader);
      const uint32_t pos = base + __popc(peers & ((1u << lane) - 1u));
      if (pos < kCap) r->inb[ip() ^ 1u][pos] = make_uint4(u, b, e, d);
      else spill(u);
      s->pushed = step;
    }
    __syncwarp();
    if (kBig && __any_sync(0xffffffffu, big)) push_pieces(big, u, b, e, d);
  }

  // ... the vertices with more than kPiece edges: one piece per lane at a time.
  __device__ __forceinline__ void push_pieces(bool big, uint32_t u, uint32_t b, uint32_t e, uint32_t d) {
    const uint32_t nq = cq == 2 ? 0 : cq + 1;
    const uint32_t np = big ? (e - b + kPiece - 1) / kPiece : 0u;
    uint32_t incl = np;
#pragma unroll
    for (int o2 = 1; o2 < 32; o2 <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o2);
      if ((int)lane >= o2) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (lane == 0) atomicAdd(&away_in(s->away, step, round), total - total / C);
    for (uint32_t k0 = 0; k0 < total; k0 += 32) {
      const uint32_t k = k0 + lane;
      int j = 0;
#pragma unroll
      for (int st = 16; st >= 1; st >>= 1) {
        const uint32_t pv = __shfl_sync(0xffffffffu, incl, j + st - 1);
        if (pv <= k) j += st;
      }
      const uint32_t pu = __shfl_sync(0xffffffffu, u, j), pb = __shfl_sync(0xffffffffu, b, j);
      const uint32_t pe = __shfl_sync(0xffffffffu, e, j), pd = __shfl_sync(0xffffffffu, d, j);
      const uint32_t at = k - __shfl_sync(0xffffffffu, incl - np, j);
      if (k < total) {
        const uint32_t t = (home(pu) + at) % C;
        const uint32_t xb = pb + at * kPiece;
        const uint4 en = make_uint4(pu, xb, min(pe, xb + kPiece), pd);
        if (t == rank) {
          const uint32_t pos = atomicAdd(&s->cnt[nq], 1u);
          if (pos < kCap) s->loc[lb ^ 1u][pos] = en;
          else spill(pu);
        } else {
          Shared *r = cl.map_shared_rank(s, t);
          const uint32_t pos = atomicAdd(&r->incnt[ip() ^ 1u], 1u);
          if (pos < kCap) r->inb[ip() ^ 1u][pos] = en;
          else spill(pu);
          s->pushed = step;
        }
      }
    }
  }

  // Puts (u, d) of the lanes with `want` on this CTA's far list `buf`.
  __device__ __forceinline__ void push_far(bool want, uint32_t u, uint32_t d, uint32_t buf) {
    const uint32_t m = __ballot_sync(0xffffffffu, want);
    if (!m) return;
    uint32_t base = 0;
    const int leader = __ffs(m) - 1;
    if ((int)lane == leader) base = atomicAdd(&s->farcnt[buf], __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (want) {
      const uint32_t pos = base + __popc(m & ((1u << lane) - 1u));
      if (pos < a.far_cap) {
        a.far[(size_t)(rank * 2 + buf) * a.far_cap + pos] = make_uint2(u, d);
      } else {
        atomicOr(a.farbm + (u >> 5), 1u << (u & 31u));
        s->farbm = step;
      }
    }
  }

  // Relaxes the entries of a warp's lanes (v, [beg,end), d; the lanes with
  // `has` are the first ones and their ranges are not empty): their edges are
  // laid end to end, one per lane.  A target's offsets are loaded beside the
  // atomic that lowers its distance, so pushing it waits for nothing more.
  // Called by whole warps.
  // A stale entry's edges are not relaxed, and a plain read comes before each
  // atomic: most edges into a dense part of the graph improve nothing, and
  // their atomics would queue up on its hubs (without either, RMAT-12 SSSP
  // 0.136 -> 0.167 ms).
  __device__ __forceinline__ void relax(uint4 en, bool has) {
    const uint32_t deg = has ? en.z - en.y : 0u;
    const uint32_t cur = has ? __ldcg(a.dist + en.x) : 0u;
    uint32_t incl = deg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)lane >= o) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31), excl = incl - deg;
    const bool fresh = cur == en.w;
    for (uint32_t k0 = 0; k0 < total; k0 += 32 * kIlp) {
      uint32_t u[kIlp], nd[kIlp], b[kIlp], e[kIlp], old[kIlp];
      bool act[kIlp];
#pragma unroll
      for (int i = 0; i < kIlp; ++i) {
        if (i && k0 + 32 * i >= total) {
          u[i] = nd[i] = 0u;
          act[i] = false;
          continue;
        }
        // edge k0 + 32 i + lane's entry: the entries that begin before this
        // step, and those that begin in it up to this lane
        const uint32_t k1 = k0 + 32 * i, k = k1 + lane;
        const uint32_t before = __popc(__ballot_sync(0xffffffffu, has && excl < k1));
        const uint32_t heads =
            __reduce_or_sync(0xffffffffu, has && excl >= k1 && excl < k1 + 32 ? 1u << (excl - k1) : 0u);
        const uint32_t j = before + __popc(heads & (0xFFFFFFFFu >> (31u - lane))) - 1u;
        const uint32_t ob = __shfl_sync(0xffffffffu, en.y, j);
        const uint32_t of = __shfl_sync(0xffffffffu, excl, j);
        const uint32_t od = __shfl_sync(0xffffffffu, en.w, j);
        act[i] = k < total;
        const uint32_t x = ob + (k - of);
        u[i] = act[i] ? __ldg(a.cols + x) : 0u;
        nd[i] = od + (kUnit ? 1u : (act[i] ? __ldg(a.wts + x) : 0u));
        act[i] = __shfl_sync(0xffffffffu, (int)fresh, j) && act[i];
      }
#pragma unroll
      for (int i = 0; i < kIlp; ++i) old[i] = act[i] ? __ldcg(a.dist + u[i]) : 0u;
#pragma unroll
      for (int i = 0; i < kIlp; ++i) {
        res.visits += act[i];
        act[i] = act[i] && nd[i] < old[i];
      }
#pragma unroll
      for (int i = 0; i < kIlp; ++i) {
        b[i] = act[i] ? __ldg(a.offs + u[i]) : 0u;
        e[i] = act[i] ? __ldg(a.offs + u[i] + 1) : 0u;
        old[i] = act[i] ? atomicMin(a.dist + u[i], nd[i]) : 0u;
      }
      // the edges of the targets that improve and stay on this SM: started
      // before the atomics' answers arrive
#pragma unroll
      for (int i = 0; i < kIlp; ++i)
        if (e[i] > b[i]) prefetch_edges(b[i]);
      // one copy of the code for both steps: the kernel's rounds are short
      // enough to feel the instruction cache
      static_assert(kIlp == 2, "two steps");
#pragma unroll 1
      for (int i = 0; i < kIlp && k0 + 32 * i < total; ++i) {
        const bool imp = i ? act[1] && nd[1] < old[1] : act[0] && nd[0] < old[0];
        settle<true>(imp, true, i ? u[1] : u[0], i ? nd[1] : nd[0], i ? old[1] : old[0],
                     i ? b[1] : b[0], i ? e[1] : e[0]);
      }
    }
  }

  // The 128-byte lines behind and before word i's, within the array.
  __device__ __forceinline__ void prefetch_near(const uint32_t *p, uint32_t i, uint32_t size) {
    if (i + 32u < size) prefetch_l2(p + i + 32);
    if (i >= 32u) prefetch_l2(p + i - 32);
  }

  __device__ __forceinline__ void prefetch_edges(uint32_t b) {
    prefetch_l1(a.cols + b);
    if (!kUnit) prefetch_l1(a.wts + b);
  }

  // The lanes with `imp` lowered vertex u (edges [b,e)) from `old` to nd; the
  // ones with `queue` too push it.  Called by whole warps.
  template <bool kBig>
  __device__ __forceinline__ void settle(bool imp, bool queue, uint32_t u, uint32_t nd,
                                         uint32_t old, uint32_t b, uint32_t e) {
    if (!__any_sync(0xffffffffu, imp)) return;
    if (imp) {
      if (old == kInf) {
        res.nr += 1;
        res.mr += e - b;
      }
      if (kUnit) count_depth(nd, old, e - b);
    }
    // a wave that reaches the start of a line goes on to the next one (or
    // back to the one before): fetch both from HBM some levels ahead
    if (imp && a.ahead) {
      if ((u & 31u) == 16u) {
        prefetch_near(a.offs, u, a.n);
        prefetch_near(a.dist, u, a.n);
      }
      if ((b & 31u) < e - b) {
        prefetch_near(a.cols, b, a.m);
        if (!kUnit) prefetch_near(a.wts, b, a.m);
      }
    }
    push<kBig>(imp && queue && nd < T, u, b, e, nd);
    push_far(imp && queue && nd >= T && e > b, u, nd, fb);
  }

  // Few entries: a.lanes lanes per entry, no scan, and nothing waits for the
  // check that an entry is still current.  A stale entry may lower a distance,
  // but does not push: the entry that made it stale relaxes the same edge with
  // a smaller candidate, before (then this one lowers nothing) or after (then
  // that one lowers and pushes).  Called by whole warps.
  __device__ __forceinline__ void relax_few(uint4 en, bool has) {
    const uint32_t cur = has ? __ldcg(a.dist + en.x) : 0u;
    for (uint32_t x = en.y + (lane & (a.lanes - 1)); __any_sync(0xffffffffu, has && x < en.z);
         x += a.lanes) {
      const bool act = has && x < en.z;
      const uint32_t u = act ? __ldg(a.cols + x) : 0u;
      const uint32_t nd = en.w + (kUnit ? 1u : (act ? __ldg(a.wts + x) : 0u));
      const uint32_t b = act ? __ldg(a.offs + u) : 0u, e = act ? __ldg(a.offs + u + 1) : 0u;
      const uint32_t old = act ? atomicMin(a.dist + u, nd) : 0u;
      if (e > b) prefetch_edges(b);
      res.visits += act;
      settle<false>(act && nd < old, cur == en.w, u, nd, old, b, e);
    }
  }

  // BFS: a vertex of degree `deg` got label nd in place of old.
  __device__ __forceinline__ void count_depth(uint32_t nd, uint32_t old, uint32_t deg) {
    atomicAdd(&s->ring[nd % kRing], 1);
    if (old != kInf) atomicAdd(&s->ring[old % kRing], -1);
    if (a.trace && nd < a.trace_cap) {
      atomicAdd(&a.trace[nd].count, 1u);
      atomicAdd(&a.trace[nd].edges, (unsigned long long)deg);
    }
    if (a.trace && old < a.trace_cap) {
      atomicAdd(&a.trace[old].count, 0xFFFFFFFFu);
      atomicAdd(&a.trace[old].edges, 0ull - deg);
    }
  }

  // The next entries of what the step before spilled, in place of this round's
  // list, which has been read: first the vertices in this CTA's share of the
  // near bitmap's words, then its share of the wide list.  Returns how many,
  // 0 when all are done.  Called by the whole block.
  __device__ __forceinline__ uint32_t next_spilled() {
    __syncthreads();
    if (threadIdx.x == 0) {
      s->claimed = 0u;
      s->refused = kCap;
    }
    __syncthreads();
    if (!s->had) {
      take_words();
      __syncthreads();
      if (s->claimed) {
        const uint32_t count = min(s->claimed, s->refused);
        if (!kUnit && a.hand_back && threadIdx.x == 0) {
          Shared *r = cl.map_shared_rank(s, 0);
          if (atomicAdd(&r->nspilled[step & 1u], count) + count >= kHandBack)
            *(volatile uint32_t *)&words_of(r->found, step).many = step;
        }
        return count;
      }
      cl.sync();  // the wide list is complete
    }
    return take_wide();
  }

  // A warp takes 32 words at a time and of those one after another, until the
  // list has no room for a word's entries.  The words are dealt to the CTAs by
  // 32: neighbouring ids are often of the same depth.
  __device__ __forceinline__ void take_words() {
    uint32_t *bm = near_of(step - 1);
    uint32_t w = s->cur[warp];
    bool room = true;
    for (; room && w < a.W; w += room ? 32 * kWarps * C : 0) {
      const uint32_t at = w + lane;
      const uint32_t word = at < a.W ? __ldcg(bm + at) : 0u;
      for (uint32_t left = __ballot_sync(0xffffffffu, word != 0u); left; left &= left - 1) {
        const int src = __ffs(left) - 1;
        const bool has = (__shfl_sync(0xffffffffu, word, src) >> lane) & 1u;
        const uint32_t v = (w + src) * 32 + lane;
        const uint32_t b = has ? __ldg(a.offs + v) : 0u, e = has ? __ldg(a.offs + v + 1) : 0u;
        const uint32_t d = has ? __ldcg(a.dist + v) : 0u;
        const bool wide = e - b > kWideEdges;
        uint32_t np = wide ? 0u : (e - b + kPiece - 1) / kPiece, incl = np;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
          if ((int)lane >= o) incl += t;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t pos = lane == 0 ? atomicAdd(&s->claimed, total) : 0u;
        pos = __shfl_sync(0xffffffffu, pos, 0);
        // once one claim finds no room none does, so the first one's place is
        // where the entries end
        if (pos + total > kCap) {
          if (lane == 0) atomicMin(&s->refused, pos);
          room = false;
          break;
        }
        pos += incl - np;
        for (uint32_t x = b; np; --np, x += kPiece)
          s->loc[lb][pos++] = make_uint4(v, x, min(e, x + kPiece), d);
        if (wide) {
          Shared *r = cl.map_shared_rank(s, 0);
          const uint32_t i = atomicAdd(&r->nwide[step & 1u], 1u);
          if (i < kWide) r->wide[step & 1u][i] = make_uint4(v, b, e, d);
          else spill(v);
        }
        if ((int)lane == src) __stcg(bm + at, 0u);
      }
    }
    if (lane == 0) s->cur[warp] = w;
  }

  // The wide list's entries are dealt to the CTAs one by one.
  __device__ __forceinline__ uint32_t take_wide() {
    const Shared *r = cl.map_shared_rank(s, 0);
    const uint4 *wide = r->wide[step & 1u];
    const uint32_t nw = min(r->nwide[step & 1u], kWide), had = s->had;
    uint32_t all = 0;
    for (uint32_t j = 0; j < nw; ++j) all += (wide[j].z - wide[j].y + kPiece - 1) / kPiece;
    const uint32_t mine = all > rank ? (all - rank + C - 1) / C : 0u;
    const uint32_t count = min(mine - had, kCap);
    for (uint32_t k = threadIdx.x; k < count; k += kBlock) {
      uint32_t i = (had + k) * C + rank, j = 0;
      uint4 en = wide[0];
      for (uint32_t np; i >= (np = (en.z - en.y + kPiece - 1) / kPiece); en = wide[++j]) i -= np;
      en.y += i * kPiece;
      en.z = min(en.z, en.y + kPiece);
      s->loc[lb][k] = en;
    }
    __syncthreads();
    if (threadIdx.x == 0) s->had = had + count;
    return count;
  }

  __device__ __forceinline__ uint32_t block_min(uint32_t x) {
    x = __reduce_min_sync(0xffffffffu, x);
    if (lane == 0) s->red[warp] = x;
    __syncthreads();
    uint32_t m = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) m = min(m, s->red[i]);
    return m;
  }

  // No CTA has near work: T advances past the smallest far distance and the
  // far vertices below it are pushed (this CTA's list and, if any CTA put
  // bits there, its share of the far bitmap).  False when nothing is far.
  __device__ __forceinline__ bool split() {
    const uint2 *cur = a.far + (size_t)(rank * 2 + fb) * a.far_cap;
    const uint32_t fc = min(s->farcnt[fb], a.far_cap);
    const Shared *r0 = cl.map_shared_rank(s, 0);
    const bool bm = *(const volatile uint32_t *)&r0->g_farbm > s->scanned;
    // stamped in the step that just ended (no CTA is past this split)
    if (!bm && *(const volatile uint32_t *)&r0->g_far < step - 1) return false;
    const uint32_t per = (a.W + C - 1) / C;
    const uint32_t w0 = min(a.W, rank * per), w1 = min(a.W, w0 + per);
    uint32_t m = 0xFFFFFFFFu;
    for (uint32_t i = threadIdx.x; i < fc; i += kBlock) {
      const uint2 f = __ldcg(cur + i);
      if (__ldcg(a.dist + f.x) == f.y) m = min(m, f.y);
    }
    if (bm) {
      for (uint32_t w = w0 + threadIdx.x; w < w1; w += kBlock)
        for (uint32_t bits = __ldcg(a.farbm + w); bits; bits &= bits - 1) {
          const uint32_t d = __ldcg(a.dist + w * 32 + (__ffs(bits) - 1));
          if (d >= T) m = min(m, d);  // below T: expanded as near since
        }
    }
    m = block_min(m);
    if (threadIdx.x == 0) s->min_far = m;
    cl.sync();
    const uint32_t gm = __reduce_min_sync(
        0xffffffffu, *(volatile uint32_t *)&cl.map_shared_rank(s, lane % C)->min_far);
    if (gm == 0xFFFFFFFFu) return false;
    if (kUnit) {
      // every depth below T is final; the labels of depth T stay counted
      if (threadIdx.x < kRing && threadIdx.x != T % kRing) s->ring[threadIdx.x] = 0;
      if (a.trace && rank == 0 && threadIdx.x == 0)
        for (uint32_t d = T; d > 0 && d < a.trace_cap && a.trace[d].t_ns == 0; --d)
          a.trace[d].t_ns = global_timer_ns();
    }
    const uint32_t Told = T;
    // weights far above delta: a threshold step should last a few steps
    uint32_t delta = s->delta;
    if (a.adapt && step - s->last_split <= 3 && delta < 1u << 30) delta *= 2;
    T = gm > 0xFFFFFFFFu - delta ? 0xFFFFFFFFu : gm + delta;
    const uint32_t lists = (fc + kBlock - 1) / kBlock;
    const uint32_t words = bm ? (w1 - w0 + kWarps - 1) / kWarps : 0u;
    for (uint32_t r = 0; r < lists + words; ++r) {
      uint32_t v = 0, d = 0;
      bool live = false;
      if (r < lists) {
        const uint32_t i = r * kBlock + threadIdx.x;
        if (i < fc) {
          const uint2 f = __ldcg(cur + i);
          v = f.x;
          d = f.y;
          live = __ldcg(a.dist + v) == d;
        }
      } else {
        const uint32_t w = w0 + (r - lists) * kWarps + warp;
        // other CTAs may be setting bits of far vertices they cannot list
        uint32_t bits = 0;
        if (lane == 0 && w < w1 && __ldcg(a.farbm + w)) bits = atomicExch(a.farbm + w, 0u);
        bits = __shfl_sync(0xffffffffu, bits, 0);
        if (!bits) continue;
        v = w * 32 + lane;
        if ((bits >> lane) & 1u) {
          d = __ldcg(a.dist + v);
          live = d >= Told;
        }
      }
      const uint32_t b = live ? __ldg(a.offs + v) : 0u, e = live ? __ldg(a.offs + v + 1) : 0u;
      push<true>(live && d < T, v, b, e, d);
      push_far(live && d >= T, v, d, fb ^ 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      s->farcnt[fb] = 0u;
      s->scanned = step - 1;
      s->last_split = step;
      s->delta = delta;
      s->cnt[cq == 0 ? 2 : cq - 1] = 0u;  // the list of the rounds to come
    }
    fb ^= 1u;
    __syncthreads();
    ++res.splits;
    return true;
  }

  // SSSP: what waits in the lists goes to the bitmaps: near vertices to those of
  // the step that ended, far ones to the far bitmap.
  __device__ __forceinline__ void give_back() {
    uint32_t *near = near_of(step - 1);
    const uint32_t nc = min(s->cnt[cq], kCap), ni = min(s->incnt[ip()], kCap);
    for (uint32_t i = threadIdx.x; i < nc + ni; i += kBlock) {
      const uint32_t v = (i < nc ? s->loc[lb][i] : s->inb[ip()][i - nc]).x;
      atomicOr(near + (v >> 5), 1u << (v & 31u));
    }
    const uint2 *far = a.far + (size_t)(rank * 2 + fb) * a.far_cap;
    const uint32_t nf = min(s->farcnt[fb], a.far_cap);
    for (uint32_t i = threadIdx.x; i < nf; i += kBlock) {
      const uint32_t v = __ldcg(far + i).x;
      atomicOr(a.farbm + (v >> 5), 1u << (v & 31u));
    }
  }

  // What the cluster found in a step.
  struct Found {
    bool work, spilled, late, many;
  };

  // After a round: the pushes made before the call become readable by their
  // readers.
  __device__ __forceinline__ Found end_step() {
    if (threadIdx.x == 0) {
      Shared *r = cl.map_shared_rank(s, 0);
      volatile StepWords *w = &words_of(r->found, step);
      if (s->cnt[cq] || s->pushed == step) w->work = step;
      if (s->spilled == step) w->spilled = step;
      if (s->farbm == step) *(volatile uint32_t *)&r->g_farbm = step;
      if (s->farcnt[fb]) *(volatile uint32_t *)&r->g_far = step;
    }
    // the counts that the next step starts from: the last to read them was the
    // step before this one
    if (threadIdx.x >= 32 && threadIdx.x < 32 + kRounds)
      away_in(s->away, step + 1, threadIdx.x - 32) = 0u;
    if (rank == 0 && threadIdx.x == 64) {
      s->nwide[(step + 1) & 1u] = s->nspilled[(step + 1) & 1u] = 0u;
      const unsigned long long t = global_timer_ns();
      if (t - s->t_step > a.timeout_ns) words_of(s->found, step).late = step;
      s->t_step = t;
    }
    cl.sync();
    const StepWords w = words_of(cl.map_shared_rank(s, 0)->found, step);  // one load
    const Found f{found(w.work, step), found(w.spilled, step), found(w.late, step),
                  !kUnit && found(w.many, step)};
    ++step;
    return f;
  }

  __device__ __forceinline__ void next_round() {
    __syncthreads();
    cq = cq == 2 ? 0 : cq + 1;
    lb ^= 1u;
  }

  // Runs the traversal to its end.  Before the call the caller has
  // synchronised the cluster after construction and then pushed the starting
  // entries (all below T).
  __device__ __forceinline__ void run() {
    next_round();
    while (true) {
      const Found f = end_step();
      if (f.late) {
        if (rank == 0 && threadIdx.x == 0) atomicOr(a.err, kErrTimeout);
        break;
      }
      if (f.many) {
        give_back();
        handed_back = true;
        break;
      }
      if (!f.work && !f.spilled) {
        if (!split()) break;
        next_round();
      }
      const uint32_t v0 = res.visits;
      uint32_t taken = 0;
#pragma unroll 1
      for (round = 0; round < kRounds; ++round) {
        uint32_t nc = min(s->cnt[cq], kCap);
        uint32_t total = nc + (round == 0 ? min(s->incnt[ip()], kCap) : 0u);
        const bool scan = round == 0 && f.spilled;
        if (total == 0 && !scan) break;
        // ids that jump between homes: most of this step's pushes wait in
        // other CTAs' inboxes, and further rounds over the rest only delay them
        if (!goes_on(s->away, step, round, nc)) break;
        // the list after next was read in the round before this one
        if (threadIdx.x == 0) {
          s->cnt[cq == 0 ? 2 : cq - 1] = 0u;
          s->had = 0u;
        }
        if (scan && lane == 0) s->cur[warp] = 32u * (warp * C + rank);
        // once over the lists, then over what the step before spilled
        while (true) {
          taken += total;
          if (a.lanes && total * a.lanes <= 2 * kBlock) {
            for (uint32_t base = threadIdx.x; base < total * a.lanes + lane; base += kBlock) {
              const uint32_t i = base >> lane_shift;
              const bool has = i < total;
              uint4 en = make_uint4(0u, 0u, 0u, 0u);
              if (has) en = i < nc ? s->loc[lb][i] : s->inb[ip()][i - nc];
              relax_few(en, has);
            }
          } else {
            const uint32_t epw = min(32u, (total + kWarps - 1) / kWarps);
            for (uint32_t base = warp * epw; base < total; base += kWarps * epw) {
              const uint32_t i = base + lane;
              const bool has = lane < epw && i < total;
              uint4 en = make_uint4(0u, 0u, 0u, 0u);
              if (has) en = i < nc ? s->loc[lb][i] : s->inb[ip()][i - nc];
              relax(en, has);
            }
          }
          if (__builtin_expect(!scan, 1)) break;  // away from the rounds' code
          nc = total = next_spilled();
          if (total == 0) break;
        }
        next_round();
        if (round == 0 && threadIdx.x == 0) s->incnt[ip()] = 0u;
      }
      round = 0;
      ++res.steps;
      if (!kUnit && a.trace && res.steps < a.trace_cap) {
        Trace *t = a.trace + res.steps;
        atomicAdd(&t->edges, (unsigned long long)(res.visits - v0));
        if (threadIdx.x == 0) {
          atomicAdd(&t->count, taken);
          if (rank == 0) {
            t->t_ns = global_timer_ns();
            t->tag = a.tag + res.splits;
          }
        }
      }
      if ((unsigned long long)step > 16ull * a.n + 1024ull) {
        if (rank == 0 && threadIdx.x == 0) atomicOr(a.err, kErrLevels);
        break;
      }
    }
    if (kUnit) {
      // the largest depth still held by a vertex, among the last threshold's
      __syncthreads();
      if (threadIdx.x < kRing && s->ring[threadIdx.x])
        atomicAdd(&cl.map_shared_rank(s, 0)->ring_sum[threadIdx.x], s->ring[threadIdx.x]);
      cl.sync();
      if (rank == 0 && threadIdx.x == 0) {
        uint32_t d = T;  // the labels of [T - Delta, T] are counted
        while (d > T - a.delta && s->ring_sum[d % kRing] <= 0) --d;
        res.last = d;
      }
    } else {
      cl.sync();  // no CTA leaves while another may still read its shared memory
    }
  }

  // Sum over the block of a per-thread count; valid in thread 0.
  __device__ __forceinline__ unsigned long long block_sum(unsigned long long x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    __syncthreads();
    if (lane == 0) s->red64[warp] = x;
    __syncthreads();
    unsigned long long t = 0;
    if (threadIdx.x == 0)
      for (int i = 0; i < kWarps; ++i) t += s->red64[i];
    return t;
  }
};

// Launches of a one-cluster kernel of kBlock threads a CTA: the largest cluster
// (16, 8, 4, 2 or 1 CTAs) the current device can co-schedule.  Sets the kernel's
// attributes on that device.
template <class Kernel>
int cluster_size(Kernel kern, size_t smem) {
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  for (int k = kMaxCluster; k > 1; k /= 2) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)k;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)k);
    cfg.blockDim = dim3(kBlock);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) == cudaSuccess && nc >= 1) return k;
    cudaGetLastError();
  }
  return 1;
}

template <class Kernel, class Args>
cudaError_t launch(Kernel kern, int cluster, size_t smem, const Args &a, cudaStream_t s) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)cluster;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cluster);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, a);
}

}  // namespace narrow
}  // namespace grus
