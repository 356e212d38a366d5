// pagerank.cu -- pull PageRank, FP32 ranks, fixed iteration count, one
// persistent launch.
//
//   r_0(v) = 1/n,  r_{t+1}(v) = (1-d)/n + d * sum_{u -> v} r_t(u) / outdeg(u)
//
// Dangling mass is not redistributed, as in the reference, which never pushes
// from out-degree-0 vertices (samples/pagerank/pr.cu:29-31,83).  The reference
// itself runs a delta-push variant (pr.cu:17-90) whose pull mode is broken
// (kernel_pull never calls job.prepare(), include/kernel.cuh:128-133); the
// drop-in headers keep that sample's semantics, this entry point computes the
// definition above.
//
// Layout: in-edges (CSC) from grus_graph_build_csc; a contribution array
// c(u) = r(u)/outdeg(u) double-buffered across iterations, so an iteration is
// one fused pass: gather c over in-edges, form r, write c_next (and r on the
// last iteration).  Every warp takes an equal share of the edges and vertices
// (an edge counts 1, a vertex kVertexCost), a contiguous range of the CSC that
// may begin and end inside a vertex's list, whatever the degrees are; the
// sums of a list that several warps share are added by the last of them to
// finish, in order, so one grid barrier separates the iterations.
//
// Bound by the gathers.  L2 serves random 4-byte reads at 285 G/s at most,
// whatever the array's size beyond a few MB, and far fewer where they meet on
// few lines (148 G/s over 128 KB, 40 over 4 KB); shared memory serves several
// times more.  So each SM keeps contributions in shared memory (kHot): all of
// them on a small graph, else those of the kHotCap vertices of largest
// out-degree, if they are the sources of a quarter of the edges.  For that the
// graph's column ids are relabelled once (plan, kept with the workspace) to the
// contributions' places: first the slots, then the other vertices with
// out-edges, so that what L2 has to hold shrinks too.  With less L1 beside
// them the gathers in flight no longer fit: RMAT-24 with 16,384 / 24,576 /
// 32,768 / 40,960 slots 15.8 / 15.6 / 16.4 / 21 ms.
//
// 20 iterations, ms, before (a warp per 32 vertices, segmented scans, all
// gathers from L2, two barriers an iteration) and now: RMAT-24 (263 M edges)
// 23.0, 14.8 (355 G gathers/s); RMAT-20 1.70, 1.05; RMAT-16 0.62, 0.235;
// uniform 3 M vertices of degree 16 (no plan) 5.33, 3.62 (265 G/s); 50,021 of
// degree 12 0.567, 0.165.  Of that for RMAT-24: equal shares 23.0 -> 20.7, the
// next batch's loads in flight during the sums -> 16.8, shorter chains between
// them -> 15.6, no L2 window -> 15.0, compact places -> 14.8.
#include <algorithm>
#include <cstring>
#include <vector>

#include "edge_batches.h"
#include "grus_internal.cuh"

namespace grus {

namespace {

constexpr int kBlock = 1024;        // 1 CTA/SM
constexpr int kBatch = 256;         // edges a warp gathers at once
constexpr uint32_t kLongRun = 64;   // edges of one vertex in a batch that the warp adds
constexpr uint32_t kCutMin = 64;    // lists below it are not shared by warps
constexpr uint32_t kVertexCost = 4;  // in edges
constexpr uint32_t kWarpCost = 128; // least work per warp before fewer CTAs are launched
constexpr uint32_t kHotCap = 24576; // slots beside contributions gathered from L2
constexpr uint32_t kHotAll = 48000; // vertices of a graph kept whole in shared memory
constexpr uint32_t kNone = 0xFFFFFFFFu;  // no source: every id is smaller

struct Args {
  const uint32_t *__restrict__ toffs;  // CSC offsets
  const uint32_t *__restrict__ tcols;  // CSC sources
  const uint32_t *__restrict__ offs;   // CSR offsets (out-degrees)
  uint32_t n, m;
  float base, damping;
  int iters;
  float *c[2];
  float *rank;
  // kHot: how many contributions shared memory holds; with a plan, that of
  // vertex v is c[slot[v]], else (slot null) c[v]
  uint32_t hot;
  const uint32_t *__restrict__ slot;
  // lists that several warps share: warp w's sum of its first one (head) and
  // of its last one (tail), and the arrivals of the warps sharing w's last one
  float *head, *tail;
  uint32_t *arrived;
  unsigned long long share;  // work per warp
  GridBarrier *bar;
  uint32_t *err;
  uint64_t timeout_ns;
};

// Compensated accumulator (Neumaier's variant of Kahan summation).
struct KSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float t = s + x;
    c += fabsf(s) >= fabsf(x) ? (s - t) + x : (x - t) + s;
    s = t;
  }
  __device__ __forceinline__ float value() const { return s + c; }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Where v's contribution goes; kNone: nowhere.
template <bool kHot>
__device__ __forceinline__ uint32_t place(const Args &a, uint32_t v) {
  return kHot && a.slot ? __ldg(a.slot + v) : v;
}

// Writes to place p the contribution of a vertex of out-degree d for rank r.
__device__ __forceinline__ void contribute(uint32_t p, uint32_t d, float r, float *cn) {
  if (p != kNone) cn[p] = d ? r / (float)d : 0.0f;  // one rounding
}

__device__ __forceinline__ uint32_t out_degree(const Args &a, uint32_t v) {
  return __ldg(a.offs + v + 1) - __ldg(a.offs + v);
}

__device__ __forceinline__ void finish(const Args &a, uint32_t v, uint32_t p, uint32_t d, float sum,
                                       float *cn, bool last) {
  const float r = a.base + a.damping * sum;
  contribute(p, d, r, cn);
  if (last) a.rank[v] = r;
}

// A source id, read once per iteration: no line of L1 is kept for it.
__device__ __forceinline__ uint32_t source_id(const uint32_t *p) {
  uint32_t v;
  asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

template <bool kHot>
__device__ __forceinline__ float fetch(const Args &a, const float *cs, const float *sc, uint32_t u) {
  return kHot && u < a.hot ? sc[u] : __ldcg(cs + u);
}

// The work before vertex r, and the vertex whose work contains unit c: the
// largest r with work_before(r) <= c (a 32-way search by the whole warp).
__device__ __forceinline__ unsigned long long work_before(const Args &a, uint32_t r) {
  return (unsigned long long)__ldg(a.toffs + r) + (unsigned long long)kVertexCost * r;
}

__device__ __forceinline__ uint32_t vertex_at(const Args &a, unsigned long long c) {
  uint32_t lo = 0, hi = a.n + 1;
  while (hi - lo > 1) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint32_t p = lo + lane_id() * step;
    const bool below = p < hi && p >= lo && work_before(a, min(p, a.n)) <= c;
    const uint32_t k = __popc(__ballot_sync(0xffffffffu, below));
    lo += (k - 1) * step;
    hi = min(hi, lo + step);
  }
  return lo;
}

// A warp's share: edges [e0, e1), vertices r0 .. r1 - 1 and, if its end cuts
// r1's list (cut1), part of r1; cut0: its start cuts r0's list.
struct Share {
  uint32_t r0, r1, e0, e1;
  bool cut0, cut1;
};

__device__ __forceinline__ void share_bound(const Args &a, unsigned long long c, uint32_t &r,
                                            uint32_t &e, bool &cut) {
  r = vertex_at(a, c);
  e = a.m;
  cut = false;
  if (r >= a.n) return;
  const uint32_t b = __ldg(a.toffs + r), end = __ldg(a.toffs + r + 1);
  // a short list is not cut: the next warp takes all of it
  e = end - b < kCutMin ? b
                        : (uint32_t)min((unsigned long long)end, c - (unsigned long long)kVertexCost * r);
  cut = e > b;
}

// The source ids of the batch from edge x on, of which `left` are in the range,
// and the contributions of the sources; 0 past the end.
__device__ __forceinline__ void load_ids(const Args &a, uint32_t x, int left,
                                         uint32_t (&u)[kBatch / 32]) {
  const uint32_t *p = a.tcols + x + lane_id();
#pragma unroll
  for (int j = 0; j < kBatch / 32; ++j)
    u[j] = (int)lane_id() + 32 * j < left ? source_id(p + 32 * j) : kNone;
}

template <bool kHot>
__device__ __forceinline__ void load_values(const Args &a, const float *cs, const float *sc,
                                            const uint32_t (&u)[kBatch / 32],
                                            float (&f)[kBatch / 32]) {
#pragma unroll
  for (int j = 0; j < kBatch / 32; ++j) f[j] = u[j] != kNone ? fetch<kHot>(a, cs, sc, u[j]) : 0.f;
}

// One warp's share of an iteration.  The edges are taken in batches of kBatch:
// all source ids, then all contributions of a batch are loaded (coalesced,
// kBatch / 32 gathers in flight per lane) and put side by side in `sv`, from
// where each lane adds the run of its vertex, four at a time, compensated; a
// run of kLongRun or more is added by the whole warp.  Nothing has to find an
// edge's owner: a search and a segmented scan over the lanes per 32 edges
// cost more instructions than the rest.  u: the source ids of the first batch.
template <bool kHot>
__device__ __forceinline__ void run_share(const Args &a, const Share &sh, const float *cs,
                                          const float *sc, float *sv, float *cn, bool last,
                                          uint32_t gwarp, uint32_t (&u)[kBatch / 32]) {
  const uint32_t lane = lane_id();
  const uint32_t rows = sh.r1 - sh.r0 + sh.cut1;  // vertices with work here
  uint32_t x = sh.e0, lim = sh.e0;                // the batch [x, lim) is in sv
  // in flight while a batch is summed: the contributions of the next one and
  // the source ids of the one after it
  float f[kBatch / 32];
  load_values<kHot>(a, cs, sc, u, f);
  load_ids(a, x + kBatch, edges_left(x, sh.e1) - kBatch, u);
  for (uint32_t w = 0; w < rows; w += 32) {
    const uint32_t v = sh.r0 + w + lane;
    const bool ok = w + lane < rows;
    const uint32_t beg = ok ? max(__ldg(a.toffs + v), sh.e0) : sh.e1;
    const uint32_t end = ok ? min(__ldg(a.toffs + v + 1), sh.e1) : sh.e1;
    const uint32_t p = ok ? place<kHot>(a, v) : kNone;
    const uint32_t od0 = ok ? __ldg(a.offs + v) : 0u, od1 = ok ? __ldg(a.offs + v + 1) : 0u;
    const uint32_t stop = __shfl_sync(0xffffffffu, end, min(31u, rows - 1 - w));
    KSum acc;
    while (true) {
      const uint32_t lo = max(beg, x), hi = min(end, lim);
      uint32_t len = hi > lo ? hi - lo : 0u;
      for (uint32_t lm = __ballot_sync(0xffffffffu, len >= kLongRun); lm; lm &= lm - 1) {
        const int l = __ffs(lm) - 1;
        const uint32_t at = __shfl_sync(0xffffffffu, lo, l) - x;
        const uint32_t n = __shfl_sync(0xffffffffu, len, l);
        KSum t;
        for (uint32_t k = lane; k < n; k += 64)
          t.add(sv[at + k] + (k + 32 < n ? sv[at + k + 32] : 0.f));
        const float sum = warp_sum(t.value());
        if ((int)lane == l) {
          acc.add(sum);
          len = 0u;
        }
      }
      const float *run = sv + (lo - x);
      for (uint32_t k = 0; k < len; k += 4) {
        const float f0 = run[k], f1 = k + 1 < len ? run[k + 1] : 0.f;
        const float f2 = k + 2 < len ? run[k + 2] : 0.f, f3 = k + 3 < len ? run[k + 3] : 0.f;
        acc.add((f0 + f1) + (f2 + f3));
      }
      if (stop <= lim) break;  // these 32 vertices are complete
      __syncwarp();
      x = lim;
      const int left = edges_left(x, sh.e1);
      lim = batch_end(x, left, kBatch);
#pragma unroll
      for (int j = 0; j < kBatch / 32; ++j) sv[lane + 32 * j] = f[j];
      load_values<kHot>(a, cs, sc, u, f);
      load_ids(a, x + 2 * kBatch, left - 2 * kBatch, u);
      __syncwarp();
    }
    if (ok) {
      const float sum = acc.value();
      if (sh.cut0 && v == sh.r0) a.head[gwarp] = sum;
      else if (sh.cut1 && v == sh.r1) a.tail[gwarp] = sum;
      else finish(a, v, p, od1 - od0, sum, cn, last);
    }
  }
}

// This warp has written its sums of lists that it shares with others: its
// first one (begun by warp f0, ended by l0) and its last one (ended by l1).
// Of the warps sharing a list the last one to say so adds their sums in order.
template <bool kHot>
__device__ __forceinline__ void arrive(const Args &a, const Share &sh, uint32_t gwarp, uint32_t f0,
                                       uint32_t l0, uint32_t l1, int it, float *cn, bool last) {
  const uint32_t lane = lane_id();
  const bool tail = sh.cut1 && !(sh.cut0 && sh.r0 == sh.r1);
  __syncwarp();
  bool all = false;  // lane 0: every sum of the first list is there; lane 1: of the last
  if (lane < 2 && (lane ? tail : sh.cut0)) {
    __threadfence();
    const uint32_t sharers = lane ? l1 - gwarp + 1 : l0 - f0 + 1;
    all = atomicAdd(a.arrived + (lane ? gwarp : f0), 1u) + 1u == sharers * (uint32_t)(it + 1);
    __threadfence();
  }
  const uint32_t complete = __ballot_sync(0xffffffffu, all);
  for (uint32_t which = 0; which < 2; ++which) {
    if (!((complete >> which) & 1u)) continue;
    const uint32_t f = which ? gwarp : f0, l = which ? l1 : l0;
    KSum k;
    for (uint32_t w = f + lane; w <= l; w += 32) k.add(__ldcg(w == f ? a.tail + w : a.head + w));
    const float sum = warp_sum(k.value());
    const uint32_t v = which ? sh.r1 : sh.r0;
    if (lane == 0) finish(a, v, place<kHot>(a, v), out_degree(a, v), sum, cn, last);
  }
}

template <bool kHot>
__global__ void __launch_bounds__(kBlock, 1) pr_persistent(Args a) {
  extern __shared__ __align__(16) float s_hot[];  // hot contributions, then batches
  float *sv = s_hot + (kHot ? (a.hot + 31) / 32 * 32 : 0u) + (threadIdx.x >> 5) * kBatch;
  const uint32_t gtid = blockIdx.x * kBlock + threadIdx.x;
  const uint32_t nthreads = gridDim.x * kBlock;
  const uint32_t gwarp = gtid >> 5;
  const float r0 = 1.0f / (float)a.n;
  for (uint32_t v = gtid; v < a.n; v += nthreads) 
    contribute(place<kHot>(a, v), out_degree(a, v), r0, a.c[0]);
  if (lane_id() == 0) a.arrived[gwarp] = 0u;
  Share sh;
  share_bound(a, gwarp * a.share, sh.r0, sh.e0, sh.cut0);
  share_bound(a, (gwarp + 1) * a.share, sh.r1, sh.e1, sh.cut1);
  // the warps sharing the first list and the last one
  uint32_t f0 = 0, l0 = 0, l1 = 0;
  if (sh.cut0) {
    f0 = (uint32_t)(work_before(a, sh.r0) / a.share);
    l0 = (uint32_t)((work_before(a, sh.r0 + 1) - 1) / a.share);
  }
  if (sh.cut1) l1 = (uint32_t)((work_before(a, sh.r1 + 1) - 1) / a.share);
  if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;

  uint32_t u[kBatch / 32];
  load_ids(a, sh.e0, edges_left(sh.e0, sh.e1), u);
  for (int it = 0; it < a.iters; ++it) {
    const float *cs = a.c[it & 1];
    float *cn = a.c[(it + 1) & 1];
    const bool last = it + 1 == a.iters;
    if (kHot) {
      const uint32_t quads = a.hot / 4;
      for (uint32_t i = threadIdx.x; i < quads; i += kBlock)
        reinterpret_cast<float4 *>(s_hot)[i] = __ldcg(reinterpret_cast<const float4 *>(cs) + i);
      for (uint32_t i = 4 * quads + threadIdx.x; i < a.hot; i += kBlock) s_hot[i] = __ldcg(cs + i);
      __syncthreads();
    }
    run_share<kHot>(a, sh, cs, s_hot, sv, cn, last, gwarp, u);
    load_ids(a, sh.e0, edges_left(sh.e0, sh.e1), u);  // of the next iteration, before the wait
    if (sh.cut0 || sh.cut1) arrive<kHot>(a, sh, gwarp, f0, l0, l1, it, cn, last);
    if (!last && !grid_sync(a.bar, a.err, a.timeout_ns)) return;
  }
}

// ---- plan: the vertices of largest out-degree and the relabelled columns ----
constexpr uint32_t kBins = 1u << 16;  // out-degrees, the last bin open-ended

__global__ void k_degree_bins(const uint32_t *__restrict__ offs, uint32_t n, uint32_t *bins) {
  __shared__ uint32_t s_low[256];  // most vertices have few edges
  s_low[threadIdx.x] = 0u;
  __syncthreads();
  for (uint32_t v = blockIdx.x * 256 + threadIdx.x; v < n; v += gridDim.x * 256) {
    const uint32_t d = min(offs[v + 1] - offs[v], kBins - 1);
    if (d < 256) atomicAdd(&s_low[d], 1u);
    else atomicAdd(bins + d, 1u);
  }
  __syncthreads();
  if (s_low[threadIdx.x]) atomicAdd(bins + threadIdx.x, s_low[threadIdx.x]);
}

struct PlanCtl {
  uint32_t above, at, rest;  // slots given to degrees > cut, = cut, and to the others
  uint32_t n_above, cut;
  uint32_t made;
};

// One CTA of 1024: the largest degree of which not all vertices get slots.
__global__ void __launch_bounds__(1024) k_plan_cut(const uint32_t *__restrict__ bins, PlanCtl *ctl) {
  constexpr uint32_t per = kBins / 1024;
  const uint32_t hi = kBins - threadIdx.x * per;  // bins [hi - per, hi), from the top down
  const uint4 *mine = reinterpret_cast<const uint4 *>(bins + hi - per);
  uint32_t count = 0, total = 0;
#pragma unroll
  for (uint32_t i = 0; i < per / 4; ++i) {
    const uint4 x = mine[i];
    count += x.x + x.y + x.z + x.w;
  }
  uint32_t above = block_exclusive_scan<1024>(count, &total);
  if (above > kHotCap || above + count <= kHotCap) return;  // (more vertices than slots: one thread stays)
  uint32_t d = hi - 1;
  for (; above + bins[d] <= kHotCap; --d) above += bins[d];
  ctl->n_above = above;
  ctl->cut = d;
  ctl->made = 1u;
}

// slot[v]: below kHotCap for the vertices of largest out-degree, from kHotCap
// on for the others with out-edges (those of a block side by side, in order),
// kNone for vertices without: nothing reads their contributions.
__global__ void k_plan_slots(const uint32_t *__restrict__ offs, uint32_t n, PlanCtl *ctl,
                             uint32_t *slot) {
  __shared__ uint32_t s_base;
  const uint32_t cut = ctl->cut, above = ctl->n_above;
  for (uint32_t v0 = blockIdx.x * 256; v0 < n; v0 += gridDim.x * 256) {
    const uint32_t v = v0 + threadIdx.x;
    const uint32_t d = v < n ? offs[v + 1] - offs[v] : 0u;
    uint32_t s = kNone;
    if (min(d, kBins - 1) > cut) s = atomicAdd(&ctl->above, 1u);
    else if (d && d == cut) s = above + atomicAdd(&ctl->at, 1u);
    const bool rest = d && s >= kHotCap;
    uint32_t total = 0;
    const uint32_t at = block_exclusive_scan<256>(rest, &total);
    if (threadIdx.x == 0) s_base = kHotCap + atomicAdd(&ctl->rest, total);
    __syncthreads();
    if (v < n) slot[v] = rest ? s_base + at : s;
    __syncthreads();
  }
}

__global__ void k_plan_cols(const uint32_t *__restrict__ tcols, uint64_t m,
                            const uint32_t *__restrict__ slot, uint32_t *__restrict__ out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = __ldcg(slot + __ldcs(tcols + i));
}

struct Workspace {
  float *c = nullptr;   // 2 * stride contributions
  uint64_t stride = 0;
  // plan (n > kHotAll): slots and relabelled columns behind the contributions
  bool planned = false;  // queued
  uint32_t *slot = nullptr, *cols = nullptr;
  float *rank = nullptr;
  uint32_t *shared = nullptr;  // per warp: head, tail, arrivals
  uint32_t warps = 0;
  char *ctrl = nullptr, *ctrl_host = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

// (the pinned mirror has one more word: not 0 once the plan is made)
constexpr size_t kOffBar = 0, kOffErr = 256, kCtrlBytes = 384, kOffPlanned = kCtrlBytes;
static_assert(kOffBar + sizeof(GridBarrier) <= kOffErr, "barrier layout");

void ws_free(void *p) {
  Workspace *w = (Workspace *)p;
  if (!w) return;
  cudaFree(w->c);
  cudaFree(w->rank);
  cudaFree(w->shared);
  cudaFree(w->ctrl);
  if (w->ctrl_host) cudaFreeHost(w->ctrl_host);
  if (w->ev0) cudaEventDestroy(w->ev0);
  if (w->ev1) cudaEventDestroy(w->ev1);
  delete w;
}

// Whether a graph beyond kHotAll vertices gets a plan: where the kHotCap vertices
// of largest out-degree are the sources of a quarter of the edges (by the
// graph's degree counts, the edges of the last range in proportion), from
// kPlanEdges on.  Not a managed graph, whose columns may not fit the device.
// Below kPlanEdges it gains nothing (20 iterations without / with it: RMAT-16 of 8
// edges a vertex 219 / 224 us, 60,021 vertices of degree 12 165 / 174; RMAT-16 of
// 16 258 / 239, of 24 307 / 268, RMAT-18 524 / 403) and costs the first call
// 110 us, most of it the larger allocation.
constexpr uint64_t kPlanEdges = 3ull << 18;
bool wants_plan(const grus_graph *g) {
  if (g->n <= kHotAll || g->m < kPlanEdges || g->mem_mode == GRUS_MEM_MANAGED) return false;
  double edges = 0.0;
  uint64_t left = kHotCap;
  for (int i = 31; i >= 0 && left; --i) {
    const uint64_t take = std::min<uint64_t>(left, g->deg_count[i]);
    if (take) edges += (double)g->deg_edges[i] * ((double)take / (double)g->deg_count[i]);
    left -= take;
  }
  return 4.0 * edges >= (double)g->m;
}

constexpr uint64_t kPlanSmall = 64ull << 20;

int ws_get(grus_graph *g, Workspace **out) {
  if (g->ws[kWsPr]) {
    *out = (Workspace *)g->ws[kWsPr];
    return GRUS_OK;
  }
  Workspace *w = new Workspace();
  const uint64_t n1 = std::max<uint64_t>(g->n, 1);
  w->warps = (uint32_t)std::max(device_sm_count(), 1) * (kBlock / 32);
  w->stride = (n1 + (n1 > kHotAll ? kHotCap : 0u) + 31) / 32 * 32;
  // the plan's part is kept as long as the graph: not more than a sixteenth of
  // the free memory, which is asked for where it is more than any GPU's small change
  const uint64_t slots = (n1 + 31) / 32 * 32, plan = wants_plan(g) ? (slots + g->m) * 4 : 0;
  size_t free_bytes = 0, all_bytes = 0;
  bool room = plan && (plan <= kPlanSmall || (cudaMemGetInfo(&free_bytes, &all_bytes) == cudaSuccess &&
                                              plan <= free_bytes / 16));
  cudaError_t e = cudaMalloc(&w->c, 2 * w->stride * 4 + (room ? plan : 0));
  if (e != cudaSuccess && room) {
    room = false;
    e = cudaMalloc(&w->c, 2 * w->stride * 4);
  }
  cudaGetLastError();
  if (e == cudaSuccess && room) {
    w->slot = (uint32_t *)(w->c + 2 * w->stride);
    w->cols = w->slot + slots;
  }
  if (e == cudaSuccess) e = cudaMalloc(&w->shared, (size_t)w->warps * 12);
  if (e == cudaSuccess) e = cudaMalloc(&w->ctrl, kCtrlBytes);
  if (e == cudaSuccess) e = clear_now(w->ctrl, kCtrlBytes);
  if (e == cudaSuccess) e = cudaMallocHost(&w->ctrl_host, kCtrlBytes + 8);
  if (e == cudaSuccess) std::memset(w->ctrl_host + kOffPlanned, 0, 8);
  if (e == cudaSuccess) e = cudaEventCreate(&w->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&w->ev1);
  if (e != cudaSuccess) {
    cudaGetLastError();
    ws_free(w);
    set_last_error(std::string("pagerank workspace: ") + cudaGetErrorString(e));
    return status_from_cuda(e);
  }
  g->ws[kWsPr] = w;
  g->ws_free[kWsPr] = ws_free;
  *out = w;
  return GRUS_OK;
}

// Queues the making of the plan: a few passes over the vertices and one over the
// columns (RMAT-24: 1.3 ms and 1.1 GB).  It belongs to the first
// call, like the workspace: later ones only queue their kernel, also under
// capture.  Nothing waits; a later call uses the plan once its mark has arrived
// in pinned memory.  Bins and counters stand in the contributions.
void make_plan(grus_graph *g, Workspace *w, cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return;  // left to a call outside the capture
  }
  const uint32_t n = (uint32_t)g->n;
  const int grid = std::max(device_sm_count(), 1) * 8;
  static_assert(2ull * (kHotAll + kHotCap) >= kBins + sizeof(PlanCtl) / 4, "they fit the contributions");
  uint32_t *bins = (uint32_t *)w->c;
  PlanCtl *ctl = (PlanCtl *)(bins + kBins);
  cudaError_t e = cudaMemsetAsync(bins, 0, kBins * 4 + sizeof(PlanCtl), s);
  if (e == cudaSuccess) {
    k_degree_bins<<<grid, 256, 0, s>>>(g->csr.offs, n, bins);
    k_plan_cut<<<1, 1024, 0, s>>>(bins, ctl);
    k_plan_slots<<<grid, 256, 0, s>>>(g->csr.offs, n, ctl, w->slot);
    k_plan_cols<<<grid, 256, 0, s>>>(g->csc.cols, g->m, w->slot, w->cols);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(w->ctrl_host + kOffPlanned, &ctl->made, 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) w->planned = true;
  else cudaGetLastError();
}

template <bool kHot>
int launch(Workspace *w, Args &a, cudaStream_t s) {
  static PerDevice<int> fits;
  constexpr size_t batches = (size_t)(kBlock / 32) * kBatch * 4;
  const size_t smem = batches + (kHot ? (size_t)(a.hot + 31) / 32 * 128 : 0);
  int occ = 0;
  const int rc = fits.get(current_device(), &occ, [](int &v) -> int {
    constexpr size_t most = batches + (kHot ? (size_t)std::max(kHotAll, kHotCap) * 4 : 0);
    GRUS_CUDA_TRY(cudaFuncSetAttribute(pr_persistent<kHot>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    GRUS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, pr_persistent<kHot>, kBlock, most));
    return GRUS_OK;
  });
  if (rc) return rc;
  // small graphs take fewer CTAs: the barrier of each iteration is cheaper
  const uint64_t work = (uint64_t)a.m + (uint64_t)kVertexCost * a.n;
  const int ctas = (int)std::min<uint64_t>(
      (uint64_t)device_sm_count(), std::max<uint64_t>(1, work / (kWarpCost * (kBlock / 32))));
  const uint64_t warps = (uint64_t)ctas * (kBlock / 32);
  a.share = std::max<uint64_t>(1, (work + warps - 1) / warps);
  void *args[] = {&a};
  // no L2 persisting window on the contributions: RMAT-24 15.4 ms with one,
  // 15.0 without
  return launch_persistent((const void *)pr_persistent<kHot>, args, kBlock, 1, occ, s, nullptr, 0,
                           smem, ctas);
}

}  // namespace
}  // namespace grus

using namespace grus;

extern "C" int grus_pagerank(grus_graph *g, float damping, int iters, float *rank,
                             grus_stats *stats, void *stream) {
  if (!g || !rank || iters < 0 || !(damping >= 0.f && damping <= 1.f)) return GRUS_EINVAL;
  if (g->n == 0) return GRUS_OK;
  cudaStream_t s = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lk(g->mu);
  int rc = build_csc_locked(g);
  if (rc) return rc;
  Workspace *w = nullptr;
  rc = ws_get(g, &w);
  if (rc) return rc;
  const bool dev_out = is_device_pointer(rank);
  if (!dev_out && !w->rank) GRUS_CUDA_TRY(cudaMalloc(&w->rank, g->n * 4));
  bool plan = w->planned && *(volatile uint32_t *)(w->ctrl_host + kOffPlanned);
  if (iters > 0 && w->slot && !w->planned) {
    make_plan(g, w, s);
    plan = w->planned;  // this call's kernel follows it on the stream
  }
  Args a;
  std::memset(&a, 0, sizeof(a));
  a.toffs = g->csc.offs;
  a.tcols = g->csc.cols;
  a.offs = g->csr.offs;
  a.n = (uint32_t)g->n;
  a.m = (uint32_t)g->m;
  a.base = (1.0f - damping) / (float)g->n;
  a.damping = damping;
  a.iters = iters;
  a.c[0] = w->c;
  a.c[1] = w->c + w->stride;
  const bool hot = g->n <= kHotAll || plan;
  if (g->n <= kHotAll) {
    a.hot = a.n;
  } else if (plan) {
    a.tcols = w->cols;
    a.hot = kHotCap;
    a.slot = w->slot;
  }
  a.rank = dev_out ? rank : w->rank;
  a.head = (float *)w->shared;
  a.tail = a.head + w->warps;
  a.arrived = w->shared + 2 * w->warps;
  a.bar = (GridBarrier *)(w->ctrl + kOffBar);
  a.err = (uint32_t *)(w->ctrl + kOffErr);
  a.timeout_ns = (uint64_t)tune_or(g->tuning.timeout_ms, 30000u) * 1000000ull;
  if (iters == 0) {
    // r_0 = 1/n
    std::vector<float> h(g->n, 1.0f / (float)g->n);
    GRUS_CUDA_TRY(cudaMemcpyAsync(rank, h.data(), g->n * 4, cudaMemcpyDefault, s));
    GRUS_CUDA_TRY(cudaStreamSynchronize(s));
    return GRUS_OK;
  }
  // barrier and error word: a timed-out launch leaves stale barrier state
  GRUS_CUDA_TRY(cudaMemsetAsync(w->ctrl + kOffBar, 0, kOffErr + 4 - kOffBar, s));
  if (stats) GRUS_CUDA_TRY(cudaEventRecord(w->ev0, s));
  rc = hot ? launch<true>(w, a, s) : launch<false>(w, a, s);
  if (rc) return rc;
  if (stats) GRUS_CUDA_TRY(cudaEventRecord(w->ev1, s));
  if (!dev_out) GRUS_CUDA_TRY(cudaMemcpyAsync(rank, w->rank, g->n * 4, cudaMemcpyDeviceToHost, s));
  if (!stats && dev_out) return GRUS_OK;
  GRUS_CUDA_TRY(cudaMemcpyAsync(w->ctrl_host, w->ctrl, kCtrlBytes, cudaMemcpyDeviceToHost, s));
  GRUS_CUDA_TRY(cudaStreamSynchronize(s));
  const uint32_t errbits = *(uint32_t *)(w->ctrl_host + kOffErr);
  if (errbits) {
    cudaMemsetAsync(w->ctrl, 0, kCtrlBytes, s);
    cudaStreamSynchronize(s);
    return status_from_device_error(errbits);
  }
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->levels = (uint32_t)iters;
    stats->kernel_launches = 1;
    stats->vertices_reached = g->n;
    stats->edges_reached = g->m * (uint64_t)iters;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, w->ev0, w->ev1);
    stats->device_ms = ms;
  }
  return GRUS_OK;
}

namespace grus {
CtrlView pr_ctrl(grus_graph *g) {
  CtrlView v;
  std::lock_guard<std::mutex> lk(g->mu);
  const Workspace *w = (const Workspace *)g->ws[kWsPr];
  if (w) {
    v.ctrl = w->ctrl;
    v.bytes = kCtrlBytes;
    v.err_off = kOffErr;
    v.bar_off = kOffBar;
  }
  return v;
}
}  // namespace grus
