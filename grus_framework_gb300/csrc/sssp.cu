// sssp.cu -- exact single-source shortest paths over uint32 weights as one
// persistent launch (near/far label correcting, a Delta-stepping variant:
// Meyer & Sanders 2003; GPU near-far piles: Davidson et al. 2014).
//
// Replaces the reference's SSSP_single_gpu loop (samples/sssp/sssp.cu:123-170)
// over kernel<...,Frontier<BDF>> whose updater relaxes with a NON-atomic
// read-modify-write (sssp.cu:51-60) and can keep a larger distance when two
// sources race.  Here every relaxation is atomicMin, so the result is the
// unique fixpoint -- Dijkstra's distances -- whatever the schedule.
//
// The near and far sets are bitmaps (one bit per vertex):
//   N[L & 1]  vertices to expand at level L (improved below the threshold T)
//   N[~L & 1] vertices improved below T during level L
//   F         vertices improved to a distance >= T (far)
// A level
//   1. compacts N[L & 1] into binned work lists (degree < huge: vertex queue;
//      degree >= huge: 1024-edge chunks), clearing the bitmap as it reads it,
//      with one queue reservation per CTA (block scan of the counts);
//   2. expands the lists with the degree-binned mappings of expand.cuh; a
//      relaxation that beats the distance it read lowers it with a
//      non-returning atomicMin and sets v's bit in N[~L & 1] (new distance < T)
//      or F -- also a reduction, so the relaxation path waits on no atomic.
// When a level finds nothing to expand, T advances by Delta (or jumps to the
// bucket of the smallest far distance) and F is scanned: vertices below the
// old T were expanded as near since and are dropped, vertices below the new T
// move to N[L & 1], the rest stay.  Every wait is a bounded grid barrier.
//
// A level costs the grid at least 13 us, so levels that stay small are handed
// to one thread-block cluster (sssp_narrow, narrow.cuh), which also runs small
// graphs from the start and may hand back.
#include <algorithm>
#include <cstring>

#include "expand.cuh"
#include "grus_internal.cuh"
#include "narrow.cuh"

namespace grus {
namespace {

constexpr int kBlock = 256;
constexpr uint32_t kDefHuge = 1024;
constexpr uint32_t kDefDelta = 640;
// Hand-over to the cluster kernel (sssp_narrow): kSteady levels in a row of at
// most kNarrowNf near vertices per cluster CTA, and no more than a plane's
// circle would have (4 s^2 at level s; a random graph's frontier grows past
// it), if the unreached and far vertices have at most 2^kSteadyBits out-edges;
// 2^kLongBits after 3 kSteady such levels of a graph without a vertex of more
// than kLongDegree out-edges (grids, road networks).
// The bounds cap what the cluster, a tenth of the chip, can be left with when
// a long thin stretch ends in a dense part: uniform graphs of 2-9 M edges that
// were handed over at 2^20 took 1.1-3.2 times the grid kernel's time.  Under the
// wider bound the cluster hands a frontier that gets too wide for it back
// (narrow::kHandBack) to a second launch of the persistent kernel.
constexpr uint32_t kNarrowNf = 128;
constexpr uint32_t kSteady = 8;
constexpr uint32_t kSteadyBits = 19, kLongBits = 26;
constexpr uint32_t kLongDegree = 8;
// Delta of the cluster kernel unless the caller set one: its levels are
// short, so more distance per threshold step pays (grid 1021 x 1531: Delta
// 640 11.8 ms, 1,280 11.1 ms, 2,560 12.6 ms).
constexpr uint32_t kNarrowDelta = 1280;
// Graphs whose whole traversal runs in the cluster kernel, one launch without
// grid barriers: up to 2^17 edges, or 2^19 when no vertex has more than 64
// out-edges.  Times against the grid kernel: RMAT-10 0.079 / 0.213 ms, RMAT-12
// (97 K edges) 0.167 / 0.279; RMAT-13 (204 K, hubs) 0.27-0.43 / 0.35-0.38;
// uniform degree 8, 160 K edges 0.224 / 0.440, 400 K edges 0.38 / 0.57.
constexpr uint64_t kWholeM = 1u << 17, kWholeMLow = 1u << 19;
constexpr uint32_t kWholeDegree = 64;

struct Slot {
  uint32_t qcount, ccount;
  unsigned long long visits;  // edge relaxations attempted in the level
  uint32_t taken;             // tiles of the queue that CTAs have taken
  uint32_t pad[3];
};

// Far-set control.  minfar is double-buffered by split parity so that the
// value every CTA reads at the start of split k (written during split k-1) is
// never the one being reset or reduced during split k.
struct FarCtl {
  uint32_t moved, remaining;  // of the current split
  uint32_t minfar[2];
};

struct Summary {
  uint32_t levels, splits, pad0, pad1;
  unsigned long long visits, nr, mr;
};

// Per-level record: end time, relaxations, frontier size (queue entries +
// hub chunks) and the number of threshold advances so far.
constexpr int kMaxTrace = 256;
struct LevelTrace {
  unsigned long long t_ns, visits;
  uint32_t frontier, splits;
};

// Hand-over from the persistent kernel to sssp_narrow, and back.
constexpr int kMaxTries = 4;
struct Handover {
  uint32_t flag;                     // 1: sssp_narrow continues the traversal, 2: the grid again
  uint32_t qcount;                   // vertices of the near set (Args::queue)
  uint32_t T, pad;                   // threshold; near[0] and near[1] are all zero
  // by attempt: out-edges of the vertices that are not below the threshold,
  // and the unreached vertices with their out-edges
  unsigned long long left[kMaxTries], mu[kMaxTries];
  uint32_t nu[kMaxTries];
};

struct Args {
  const uint32_t *__restrict__ offs;
  const uint32_t *__restrict__ cols;
  const uint32_t *__restrict__ wts;
  uint32_t n, W;
  uint64_t m;
  uint32_t src;
  uint32_t *dist;
  uint32_t *near[2];      // W words each
  uint32_t *farbm;        // W words
  uint32_t *queue;        // this level's vertex queue
  uint4 *chunks;          // this level's hub chunks
  uint32_t queue_cap, chunk_cap;
  Slot *slots;
  FarCtl *farctl;
  GridBarrier *bar;
  uint32_t *err;
  Summary *summary;
  LevelTrace *trace;
  uint32_t delta, huge;
  uint64_t timeout_ns;
  Handover *ho;
  uint32_t narrow_nf;     // near vertices sssp_narrow may be handed (0: never)
  uint32_t narrow_delta;
  bool narrow_adapt;      // no Delta set by the caller
  uint2 *far;             // its far lists
  bool whole;             // sssp_narrow runs the whole traversal
  bool hand_back;         // the grid may have to go on after sssp_narrow ...
  bool resume;            // ... and does in this launch, if flag is 2
  uint32_t max_deg;       // of the graph
  uint32_t lanes;         // narrow::lanes_per_entry
  bool ahead;             // narrow::View::ahead
};

struct Workspace {
  uint32_t W = 0;
  uint32_t *dist = nullptr;
  uint32_t *bitmaps = nullptr;  // 3 * Wp words: near[2], farbm
  size_t bitmap_bytes = 0;
  uint32_t *queues = nullptr;   // n
  uint4 *chunks = nullptr;
  uint32_t chunk_cap = 0;
  uint2 *far = nullptr;         // far lists of sssp_narrow, behind the bitmaps
  char *ctrl = nullptr, *ctrl_host = nullptr;
  LevelTrace *trace = nullptr, *trace_host = nullptr;
  int trace_levels = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

constexpr size_t kOffSlots = 0, kOffFar = 256, kOffHo = 288, kOffBar = 384, kOffErr = 640,
                 kOffSummary = 704, kCtrlBytes = 768;
static_assert(kOffBar % 128 == 0 && kOffBar + sizeof(GridBarrier) <= kOffErr, "barrier layout");
static_assert(4 * sizeof(Slot) <= kOffFar && sizeof(FarCtl) <= kOffHo - kOffFar &&
                  sizeof(Handover) <= kOffBar - kOffHo &&
                  sizeof(Summary) <= kCtrlBytes - kOffSummary,
              "control block layout");

void ws_free(void *p) {
  Workspace *w = (Workspace *)p;
  if (!w) return;
  cudaFree(w->dist);
  cudaFree(w->bitmaps);
  cudaFree(w->queues);
  cudaFree(w->chunks);
  cudaFree(w->ctrl);
  cudaFree(w->trace);
  if (w->ctrl_host) cudaFreeHost(w->ctrl_host);
  if (w->trace_host) cudaFreeHost(w->trace_host);
  if (w->ev0) cudaEventDestroy(w->ev0);
  if (w->ev1) cudaEventDestroy(w->ev1);
  delete w;
}

int ws_get(grus_graph *g, Workspace **out) {
  if (g->ws[kWsSssp]) {
    *out = (Workspace *)g->ws[kWsSssp];
    return GRUS_OK;
  }
  Workspace *w = new Workspace();
  w->W = (uint32_t)((g->n + 31) / 32);
  const uint64_t Wp = ((uint64_t)w->W + 31) / 32 * 32;
  w->bitmap_bytes = 3 * Wp * 4;
  // chunk lists sized for any chunking degree down to 256 (the autotuner and
  // callers may lower it after the workspace exists)
  const uint32_t huge = std::min(tune_or(g->tuning.huge_degree, kDefHuge), 256u);
  w->chunk_cap = (uint32_t)std::min<uint64_t>(g->m / kChunk + g->m / huge + 2, 0x7FFFFFFFull);
  const uint64_t n1 = std::max<uint64_t>(g->n, 1);
  // one allocation with the far lists: a first call pays for each
  cudaError_t e = cudaMalloc(&w->bitmaps, w->bitmap_bytes + narrow::far_bytes(g->n));
  if (e == cudaSuccess) w->far = (uint2 *)((char *)w->bitmaps + w->bitmap_bytes);
  if (e == cudaSuccess) e = cudaMalloc(&w->queues, n1 * 4);
  if (e == cudaSuccess) e = cudaMalloc(&w->chunks, (uint64_t)w->chunk_cap * sizeof(uint4));
  if (e == cudaSuccess) e = cudaMalloc(&w->ctrl, kCtrlBytes);
  if (e == cudaSuccess) e = clear_now(w->ctrl, kCtrlBytes);
  if (e == cudaSuccess) e = cudaMallocHost(&w->ctrl_host, kCtrlBytes);
  if (e == cudaSuccess) e = cudaMalloc(&w->trace, kMaxTrace * sizeof(LevelTrace));
  if (e == cudaSuccess) e = cudaMallocHost(&w->trace_host, kMaxTrace * sizeof(LevelTrace));
  if (e == cudaSuccess) e = cudaEventCreate(&w->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&w->ev1);
  if (e != cudaSuccess) {
    cudaGetLastError();
    ws_free(w);
    set_last_error(std::string("sssp workspace: ") + cudaGetErrorString(e));
    return status_from_cuda(e);
  }
  g->ws[kWsSssp] = w;
  g->ws_free[kWsSssp] = ws_free;
  *out = w;
  return GRUS_OK;
}

struct RelaxVisitor {
  const Args *a;
  uint32_t T;
  uint32_t *nnext;
  uint32_t visits;  // of this thread in this level

  using aux_t = uint32_t;

  __device__ __forceinline__ uint32_t aux(uint32_t v) const { return __ldcg(a->dist + v); }
  // A reduction lowers dist(v) and another marks v; neither is waited for.
  // If another thread lowered dist(v) further meanwhile, v is marked all the
  // same (a bit), costing at most one redundant expansion.
  __device__ __forceinline__ void edge(uint32_t, uint32_t du, uint32_t x) {
    ++visits;
    const uint32_t v = __ldg(a->cols + x);
    const uint32_t nd = du + __ldg(a->wts + x);
    if (nd >= __ldcg(a->dist + v)) return;
    atomicMin(a->dist + v, nd);
    atomicOr((nd < T ? nnext : a->farbm) + (v >> 5), 1u << (v & 31u));
  }
};

// Attempt to hand the traversal over at level L, whose near set is the queue
// of qc vertices: kHandedOver when done, else how many small levels in a row
// the next attempt needs.  Every thread of the grid calls it; out of line, as
// it runs a few times per traversal at most and must not cost the level loop
// registers.
constexpr uint32_t kHandedOver = 0xFFFFFFFFu, kNever = 0xFFFFFFFEu;
__device__ __noinline__ uint32_t try_hand_over(const Args &a, uint32_t run, uint32_t L, uint32_t T,
                                               uint32_t splits, uint32_t qc) {
  const uint32_t gtid = blockIdx.x * kBlock + threadIdx.x, nthreads = gridDim.x * kBlock;
  // one set of counters per attempt: the runs they need are 8, 24, 72, ...
  uint32_t k = 0;
  for (uint32_t need = run; need > kSteady; need /= 3) ++k;
  if (k >= kMaxTries) return kNever;
  unsigned long long mu = 0, nu = 0, left = 0;
  for (uint32_t v = gtid; v < a.n; v += nthreads) {
    const uint32_t d = __ldcg(a.dist + v);
    if (d < T) continue;
    const uint32_t deg = __ldg(a.offs + v + 1) - __ldg(a.offs + v);
    left += deg;
    if (d == kInfinit) {
      ++nu;
      mu += deg;
    }
  }
  const unsigned long long bmu = block_sum_u64<kBlock>(mu);
  const unsigned long long bnu = block_sum_u64<kBlock>(nu);
  const unsigned long long bleft = block_sum_u64<kBlock>(left);
  if (threadIdx.x == 0 && (bnu || bleft)) {
    atomicAdd(&a.ho->left[k], bleft);
    atomicAdd(&a.ho->mu[k], bmu);
    atomicAdd(&a.ho->nu[k], (uint32_t)bnu);
  }
  if (!grid_sync(a.bar, a.err, a.timeout_ns)) return kHandedOver;
  mu = __ldcg(&a.ho->mu[k]);
  const uint32_t bits = run >= 3 * kSteady && a.max_deg <= kLongDegree ? kLongBits : kSteadyBits;
  if (__ldcg(&a.ho->left[k]) > 1ull << bits) return 3 * run;
  if (gtid == 0) {
    a.ho->qcount = qc;
    a.ho->T = T;
    a.summary->levels = L;
    a.summary->splits = splits;
    a.summary->nr = a.n - __ldcg(&a.ho->nu[k]);
    a.summary->mr = a.m - mu;
    a.ho->flag = 1u;
  }
  return kHandedOver;
}

// kTaken: the CTAs take large levels' tiles in turn.  Dealt in advance, the last
// CTAs of a level with hubs finish 13-16 % after the mean (RMAT-22: 636 us
// against 548 in the widest); taking costs barriers and registers, which graphs
// with less work a level do not earn back (taken / dealt: RMAT-23 3,440 / 3,719
// us, RMAT-22 1,701 / 1,785, RMAT-21 with 95 M edges 1,391 / 1,526, with 64 M
// 1,348 / 1,325; uniform graph of 32 M edges 1,802 / 1,733, RMAT-18 481 / 473).
constexpr uint64_t kTakenM = 1ull << 26;
bool takes_tiles(const grus_graph *g) { return g->m >= kTakenM && g->max_deg >= kDefHuge; }

template <bool kTaken>
__global__ void __launch_bounds__(kBlock, 8) sssp_persistent(Args a) {
  // small levels in a row, and how many the next attempt to hand over needs
  // (in shared memory: the level loop has no register to spare at 8 CTAs/SM)
  __shared__ uint32_t s_small, s_need;
  if (threadIdx.x == 0) {
    s_small = 0u;
    s_need = a.narrow_nf ? kSteady : kNever;
  }
  const uint32_t gtid = blockIdx.x * kBlock + threadIdx.x;
  const uint32_t nthreads = gridDim.x * kBlock;
  if (a.resume && __ldcg(&a.ho->flag) != 2u) return;  // the same answer in every CTA
  // prologue: distances to INFINIT, bitmaps and control words to zero
  if (!a.resume) {
    for (uint32_t i = gtid; i < a.n; i += nthreads) a.dist[i] = kInfinit;
    for (uint32_t i = gtid; i < a.W; i += nthreads) {
      a.near[0][i] = 0u;
      a.near[1][i] = 0u;
      a.farbm[i] = 0u;
    }
    if (gtid < 4 * sizeof(Slot) / 4) ((uint32_t *)a.slots)[gtid] = 0u;
    if (gtid < sizeof(FarCtl) / 4) ((uint32_t *)a.farctl)[gtid] = 0u;
    if (gtid < sizeof(Handover) / 4) ((uint32_t *)a.ho)[gtid] = 0u;
    if (gtid == 0) {
      a.farctl->minfar[0] = 0xFFFFFFFFu;
      a.farctl->minfar[1] = 0xFFFFFFFFu;
    }
    if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
    if (gtid == 0) {
      a.dist[a.src] = 0;
      a.near[0][a.src >> 5] = 1u << (a.src & 31u);
    }
    if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
  }

  uint32_t L = 0, T = a.delta, splits = 0;
  if (a.resume) {
    L = __ldcg(&a.summary->levels);
    T = __ldcg(&a.ho->T);
    splits = __ldcg(&a.summary->splits);
  } else if (gtid == 0 && a.trace) a.trace[0] = LevelTrace{global_timer_ns(), 0ull, 1u, 0u};
  while (true) {
    Slot *sl = a.slots + (L & 3u);
    if (gtid < sizeof(Slot) / 4) ((uint32_t *)(a.slots + ((L + 2) & 3u)))[gtid] = 0u;
    uint32_t *ncur = a.near[L & 1u], *nnext = a.near[(L + 1) & 1u];
    bitmap_to_binned<kBlock>(ncur, a.W, a.offs, a.huge, a.queue, &sl->qcount, a.queue_cap,
                             a.chunks, &sl->ccount, a.chunk_cap, a.err, blockIdx.x, gridDim.x);
    if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
    const uint32_t qc = min(__ldcg(&sl->qcount), a.queue_cap);
    const uint32_t cc = min(__ldcg(&sl->ccount), a.chunk_cap);
    if (qc + cc == 0) {
      // nothing near: advance the threshold and split the far set into ncur
      const uint32_t Told = T;
      uint32_t Tnew = T + a.delta;
      const uint32_t mf = __ldcg(&a.farctl->minfar[splits & 1u]);
      if (mf != 0xFFFFFFFFu && mf >= Tnew) Tnew = (mf / a.delta + 1) * a.delta;
      uint32_t moved = 0, remaining = 0, local_min = 0xFFFFFFFFu;
      for (uint32_t w = gtid; w < a.W; w += nthreads) {
        const uint32_t fw = __ldcg(a.farbm + w);
        if (!fw) continue;
        uint32_t keep = 0, mv = 0;
        for (uint32_t bits = fw; bits; bits &= bits - 1) {
          const uint32_t b = __ffs(bits) - 1;
          const uint32_t d = __ldcg(a.dist + w * 32 + b);
          if (d < Told) continue;  // improved below T since: expanded as near
          if (d < Tnew) {
            mv |= 1u << b;
          } else {
            keep |= 1u << b;
            local_min = min(local_min, d);
          }
        }
        a.farbm[w] = keep;
        if (mv) ncur[w] = mv;  // ncur is all zero after its compaction
        moved += __popc(mv);
        remaining += keep != 0;
      }
      for (int o = 16; o > 0; o >>= 1) {
        local_min = min(local_min, __shfl_down_sync(0xffffffffu, local_min, o));
        moved += __shfl_down_sync(0xffffffffu, moved, o);
        remaining += __shfl_down_sync(0xffffffffu, remaining, o);
      }
      if (lane_id() == 0) {
        if (local_min != 0xFFFFFFFFu) atomicMin(&a.farctl->minfar[(splits + 1) & 1u], local_min);
        if (moved) atomicAdd(&a.farctl->moved, moved);
        if (remaining) atomicAdd(&a.farctl->remaining, remaining);
      }
      if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
      const uint32_t mv_all = __ldcg(&a.farctl->moved), rem_all = __ldcg(&a.farctl->remaining);
      if (gtid == 0) a.farctl->minfar[splits & 1u] = 0xFFFFFFFFu;  // read by all before the barrier
      T = Tnew;
      ++splits;
      // every CTA has read the counters before they are cleared; the next
      // split adds to them only after the next compaction's barrier
      if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
      if (gtid == 0) {
        a.farctl->moved = 0u;
        a.farctl->remaining = 0u;
      }
      if (mv_all == 0 && rem_all == 0) break;  // nothing near, nothing far: done
      continue;  // compact the moved vertices (or split again)
    }
    // levels that are small one after another: the cluster kernel takes over
    if (threadIdx.x == 0) {
      s_small = cc == 0 && qc <= a.narrow_nf && qc <= 4 * s_small * s_small + 64 ? s_small + 1 : 0u;
    }
    __syncthreads();
    if (s_small == s_need) {
      const uint32_t r = try_hand_over(a, s_small, L, T, splits, qc);
      if (r == kHandedOver) return;
      if (threadIdx.x == 0) s_need = r;
    }
    RelaxVisitor vis{&a, T, nnext, 0u};
    if constexpr (kTaken) expand_taken<kBlock>(a.offs, a.queue, qc, a.chunks, cc, vis, &sl->taken);
    else expand_binned<kBlock>(a.offs, a.queue, qc, a.chunks, cc, vis);
    // counted for a caller that asked for statistics only
    if (a.trace) {
      const unsigned long long bv = block_sum_u64<kBlock>(vis.visits);
      if (threadIdx.x == 0 && bv) atomicAdd(&sl->visits, bv);
    }
    if (!grid_sync(a.bar, a.err, a.timeout_ns)) return;
    ++L;
    if (gtid == 0 && a.trace) {
      const unsigned long long lv = __ldcg(&sl->visits);
      a.summary->visits += lv;
      if (L < (uint32_t)kMaxTrace)
        a.trace[L] = LevelTrace{global_timer_ns(), lv, qc + cc, splits};
    }
    if (L > 4u * a.n + 64u) {
      if (gtid == 0) atomicOr(a.err, kErrLevels);
      break;
    }
  }
  // epilogue, for a caller that asked for statistics: reached vertices and
  // their out-degree sum (m_r)
  if (a.trace) {
    unsigned long long nr = 0, mr = 0;
    for (uint32_t v = gtid; v < a.n; v += nthreads)
      if (__ldcg(a.dist + v) != kInfinit) {
        ++nr;
        mr += __ldg(a.offs + v + 1) - __ldg(a.offs + v);
      }
    const unsigned long long bnr = block_sum_u64<kBlock>(nr);
    const unsigned long long bmr = block_sum_u64<kBlock>(mr);
    if (threadIdx.x == 0) {
      atomicAdd(&a.summary->nr, bnr);
      atomicAdd(&a.summary->mr, bmr);
    }
  }
  if (gtid == 0) {
    a.summary->levels = L;
    a.summary->splits = splits;
  }
}

// One cluster: the rest of a traversal whose near set has become small
// (handed over by sssp_persistent; returns at once otherwise), or all of a
// traversal of a small graph.
__global__ void __launch_bounds__(narrow::kBlock) sssp_narrow(Args a) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (!a.whole && __ldcg(&a.ho->flag) != 1u) return;  // the same answer in every CTA
  narrow::View view;
  view.offs = a.offs;
  view.cols = a.cols;
  view.wts = a.wts;
  view.n = a.n;
  view.W = a.W;
  view.m = (uint32_t)a.m;
  view.dist = a.dist;
  view.farbm = a.farbm;
  view.far = a.far;
  view.far_cap = narrow::far_cap(a.n);
  view.delta = a.narrow_delta;
  view.adapt = a.narrow_adapt;
  view.lanes = a.lanes;
  view.ahead = a.ahead;
  view.hand_back = a.hand_back;
  view.err = a.err;
  view.timeout_ns = a.timeout_ns;
  const uint32_t L0 = a.whole ? 0u : __ldcg(&a.summary->levels);
  view.tag = a.whole ? 0u : __ldcg(&a.summary->splits);
  view.near0 = a.near[0];
  view.near1 = a.near[1];
  view.trace = a.trace && L0 < (uint32_t)kMaxTrace ? (narrow::Trace *)a.trace + L0 : nullptr;
  view.trace_cap = L0 < (uint32_t)kMaxTrace ? kMaxTrace - L0 : 0u;
  narrow::Engine<false> E(view, (narrow::Shared *)smem);
  const uint32_t tid = E.rank * narrow::kBlock + threadIdx.x, nt = E.C * narrow::kBlock;
  if (a.whole) {
    for (uint32_t i = tid; i < a.n; i += nt) a.dist[i] = i == a.src ? 0u : kInfinit;
    for (uint32_t i = tid; i < a.W; i += nt) {
      a.near[0][i] = a.near[1][i] = 0u;
      a.farbm[i] = 0u;
    }
    if (tid == 0) {
      *a.summary = Summary{0u, 0u, 0u, 0u, 0ull, 1ull,
                           (unsigned long long)(__ldg(a.offs + a.src + 1) - __ldg(a.offs + a.src))};
      *a.err = 0u;
    }
  } else if (tid == 0) {
    E.s->g_farbm = 1u;  // far vertices wait in the bitmap
  }
  if (view.trace) {
    for (uint32_t i = tid; i < view.trace_cap; i += nt)
      if (i || a.whole) view.trace[i] = narrow::Trace{i ? 0ull : global_timer_ns(), 0ull, 0u, 0u};
  }
  E.cl.sync();
  if (a.whole) {
    E.T = a.narrow_delta;
    if (E.rank == 0 && E.warp == 0)
      E.push<true>(E.lane == 0, a.src, __ldg(a.offs + a.src), __ldg(a.offs + a.src + 1), 0u);
  } else {
    E.T = __ldcg(&a.ho->T);
    const uint32_t qc = __ldcg(&a.ho->qcount);
    for (uint32_t base = tid & ~31u; base < qc; base += nt) {
      const uint32_t i = base + E.lane;
      const bool has = i < qc;
      const uint32_t v = has ? __ldcg(a.queue + i) : 0u;
      E.push<true>(has, v, has ? __ldg(a.offs + v) : 0u, has ? __ldg(a.offs + v + 1) : 0u,
             has ? __ldcg(a.dist + v) : 0u);
    }
  }
  E.run();
  if (E.handed_back) {
    // level L's near set is near[L & 1]; the last step's is near[(step - 1) & 1]
    uint32_t L = L0 + E.res.steps;
    L += (L ^ (E.step - 1)) & 1u;
    if (tid < 4 * sizeof(Slot) / 4) ((uint32_t *)a.slots)[tid] = 0u;
    if (tid == 0) {
      a.farctl->moved = a.farctl->remaining = 0u;
      a.farctl->minfar[0] = a.farctl->minfar[1] = 0xFFFFFFFFu;
      a.summary->levels = L;
      a.summary->splits = view.tag + E.res.splits;
      a.summary->nr = a.summary->mr = 0ull;  // counted at the end
      a.ho->T = E.T;
      a.ho->flag = 2u;
    }
  }
  if (!a.trace) return;
  const unsigned long long bv = E.block_sum(E.res.visits);
  if (threadIdx.x == 0) {
    atomicAdd(&a.summary->visits, bv);
    if (E.rank == 0 && !E.handed_back) {
      a.summary->levels = L0 + E.res.steps;
      a.summary->splits = view.tag + E.res.splits;
    }
  }
  if (E.handed_back) return;
  const unsigned long long bnr = E.block_sum(E.res.nr);
  const unsigned long long bmr = E.block_sum(E.res.mr);
  if (threadIdx.x == 0) {
    atomicAdd(&a.summary->nr, bnr);
    atomicAdd(&a.summary->mr, bmr);
  }
}

int narrow_cluster() {
  static PerDevice<int> sizes;
  int c = 1;
  sizes.get(current_device(), &c, [](int &v) {
    v = narrow::cluster_size(sssp_narrow, sizeof(narrow::Shared));
    return 0;
  });
  return c;
}

// CTAs an SM, 0 for all that fit (8).  Without hubs the levels are many and
// small, and fewer CTAs pass their barriers sooner (uniform graphs, 2 / 4 / 5 / 6
// / 8 CTAs: 1.2 M edges 472 / 479 / 494 / 511 / 538 us, 1.6 M 550 / 567 / 586 /
// 616 / 681, 6.4 M 853 / 754 / 753 / 783 / 839, 9 M 835 / 769 / 761 / 804 / 858;
// 32 M 3,144 / 2,103 / 1,922 / 1,839 / 1,782).  With hubs only the smallest gain
// (RMAT-13 382 -> 364, 131 K vertices and 5.4 M edges 464 -> 444; RMAT-19 needs 8).
int grid_ctas(const grus_graph *g) {
  if (g->tuning.ctas_per_sm) return (int)g->tuning.ctas_per_sm;
  if (g->mem_mode == GRUS_MEM_MANAGED) return 0;
  if (g->max_deg >= 64) return g->n <= 1u << 17 ? 6 : 0;
  return g->m <= 1u << 21 ? 2 : (g->m <= 5u << 22 ? 5 : 0);
}

bool runs_whole(const grus_graph *g) {
  return g->tuning.tail_cluster != 2 &&
         (g->m <= kWholeM || (g->m <= kWholeMLow && g->max_deg <= kWholeDegree));
}

}  // namespace

bool sssp_tail(const grus_graph *g) {
  return !runs_whole(g) && g->tuning.tail_cluster != 2;
}

// Whether the cluster may be left with more than it should finish.
static bool may_return(const grus_graph *g) { return g->max_deg <= kLongDegree; }

int sssp_kernels(const grus_graph *g, bool tail) { return tail ? (may_return(g) ? 3 : 2) : 1; }

bool sssp_lane_tail(const grus_graph *g) { return sssp_tail(g) && g->max_deg <= kWholeDegree; }

int sssp_run(grus_graph *g, uint32_t src, uint32_t *dist, grus_stats *stats, cudaStream_t s,
             bool tail) {
  if (!g || !dist) return GRUS_EINVAL;
  if (g->n == 0 || src >= g->n) {
    set_last_error("source vertex out of range");
    return GRUS_EINVAL;
  }
  if (!g->csr.wts) {
    set_last_error("sssp needs edge weights (load with need_weights or generate weighted)");
    return GRUS_EINVAL;
  }
  std::lock_guard<std::mutex> lk(g->mu);
  Workspace *w = nullptr;
  int rc = ws_get(g, &w);
  if (rc) return rc;
  const bool dev_out = is_device_pointer(dist);
  if (!dev_out && !w->dist) GRUS_CUDA_TRY(cudaMalloc(&w->dist, g->n * 4));
  const bool taken = takes_tiles(g);
  auto kern = taken ? sssp_persistent<true> : sssp_persistent<false>;
  static int occ_tab[2] = {-1, -1};
  int &occ = occ_tab[taken];
  if (occ < 0) GRUS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kBlock, 0));

  Args a;
  std::memset(&a, 0, sizeof(a));
  a.offs = g->csr.offs;
  a.cols = g->csr.cols;
  a.wts = g->csr.wts;
  a.n = (uint32_t)g->n;
  a.W = w->W;
  a.m = g->m;
  a.src = src;
  a.dist = dev_out ? dist : w->dist;
  const uint64_t Wp = ((uint64_t)w->W + 31) / 32 * 32;
  a.near[0] = w->bitmaps;
  a.near[1] = w->bitmaps + Wp;
  a.farbm = w->bitmaps + 2 * Wp;
  a.queue = w->queues;
  a.chunks = w->chunks;
  a.queue_cap = (uint32_t)g->n;
  a.chunk_cap = w->chunk_cap;
  a.slots = (Slot *)(w->ctrl + kOffSlots);
  a.farctl = (FarCtl *)(w->ctrl + kOffFar);
  a.bar = (GridBarrier *)(w->ctrl + kOffBar);
  a.err = (uint32_t *)(w->ctrl + kOffErr);
  a.summary = (Summary *)(w->ctrl + kOffSummary);
  a.trace = stats ? w->trace : nullptr;
  a.delta = std::max(1u, tune_or(g->tuning.sssp_delta, kDefDelta));
  a.huge = tune_or(g->tuning.huge_degree, kDefHuge);
  a.timeout_ns = (uint64_t)tune_or(g->tuning.timeout_ms, 30000u) * 1000000ull;

  a.ho = (Handover *)(w->ctrl + kOffHo);
  a.far = w->far;
  a.max_deg = g->max_deg;
  a.lanes = narrow::lanes_per_entry(g->max_deg);
  a.ahead = a.lanes && narrow::beyond_l2(g->n, g->m, 8);
  const int ncl = narrow_cluster();
  a.narrow_nf = tail ? kNarrowNf * (uint32_t)ncl : 0u;
  a.narrow_delta = std::max(1u, tune_or(g->tuning.sssp_delta, kNarrowDelta));
  a.narrow_adapt = g->tuning.sssp_delta == 0;
  a.whole = runs_whole(g);
  a.hand_back = tail && may_return(g);

  const bool sync = stats != nullptr || !dev_out;
  // barrier, error word and summary: a timed-out launch leaves stale barrier state
  if (!a.whole) GRUS_CUDA_TRY(cudaMemsetAsync(w->ctrl + kOffBar, 0, kCtrlBytes - kOffBar, s));
  if (stats) GRUS_CUDA_TRY(cudaEventRecord(w->ev0, s));
  void *args[] = {&a};
  // the L2 window on the distances, which every relaxation reads and lowers
  // with an atomic: RMAT-22 1.99 -> 1.80-1.83 ms against the window on the
  // near/far bitmaps (small and hot enough to stay in L2 without it)
  if (!a.whole) {
    rc = launch_persistent((const void *)kern, args, kBlock,
                           grid_ctas(g), occ, s, a.dist, (size_t)g->n * 4);
    if (rc) return rc;
  }
  if (a.whole || a.narrow_nf) GRUS_CUDA_TRY(narrow::launch(sssp_narrow, ncl, sizeof(narrow::Shared), a, s));
  if (a.hand_back) {
    a.resume = true;
    a.narrow_nf = 0u;
    rc = launch_persistent((const void *)kern, args, kBlock,
                           grid_ctas(g), occ, s, a.dist, (size_t)g->n * 4);
    if (rc) return rc;
  }
  if (stats) GRUS_CUDA_TRY(cudaEventRecord(w->ev1, s));
  if (!dev_out) GRUS_CUDA_TRY(cudaMemcpyAsync(dist, w->dist, g->n * 4, cudaMemcpyDeviceToHost, s));
  if (!sync) return GRUS_OK;
  GRUS_CUDA_TRY(cudaMemcpyAsync(w->ctrl_host, w->ctrl, kCtrlBytes, cudaMemcpyDeviceToHost, s));
  GRUS_CUDA_TRY(cudaStreamSynchronize(s));
  const uint32_t errbits = *(uint32_t *)(w->ctrl_host + kOffErr);
  if (errbits) {
    cudaMemsetAsync(w->ctrl, 0, kCtrlBytes, s);
    cudaStreamSynchronize(s);
    return status_from_device_error(errbits);
  }
  if (stats) {
    const Summary *sm = (const Summary *)(w->ctrl_host + kOffSummary);
    GRUS_CUDA_TRY(cudaMemcpy(w->trace_host, w->trace, kMaxTrace * sizeof(LevelTrace),
                             cudaMemcpyDeviceToHost));
    w->trace_levels = std::min<int>((int)sm->levels + 1, kMaxTrace);
    std::memset(stats, 0, sizeof(*stats));
    stats->levels = sm->levels;
    stats->direction_switches = sm->splits;  // threshold advances
    stats->kernel_launches = sssp_kernels(g, tail);
    stats->vertices_reached = sm->nr;
    stats->edges_reached = sm->mr;
    stats->edges_relaxed = sm->visits;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, w->ev0, w->ev1);
    stats->device_ms = ms;
  }
  return GRUS_OK;
}

}  // namespace grus

using namespace grus;

extern "C" int grus_sssp(grus_graph *g, uint32_t src, uint32_t *dist,
                         grus_stats *stats, void *stream) {
  return sssp_run(g, src, dist, stats, (cudaStream_t)stream, g && sssp_tail(g));
}

extern "C" int grus_sssp_trace(grus_graph *g, grus_level_trace *out, int max_levels) {
  if (!g || (!out && max_levels > 0) || max_levels < 0) return GRUS_EINVAL;
  std::lock_guard<std::mutex> lk(g->mu);
  const Workspace *w = (const Workspace *)g->ws[kWsSssp];
  if (!w || w->trace_levels < 2) return 0;
  const int levels = std::min(w->trace_levels - 1, max_levels);
  const uint64_t t0 = w->trace_host[0].t_ns;
  for (int i = 0; i < levels; ++i) {
    const LevelTrace &r = w->trace_host[i + 1];
    out[i].end_ns = r.t_ns - t0;
    out[i].edges = r.visits;
    out[i].vertices = r.frontier;
    out[i].pull = r.splits;
  }
  return levels;
}

namespace grus {
CtrlView sssp_ctrl(grus_graph *g) {
  CtrlView v;
  std::lock_guard<std::mutex> lk(g->mu);
  const Workspace *w = (const Workspace *)g->ws[kWsSssp];
  if (w) {
    v.ctrl = w->ctrl;
    v.bytes = kCtrlBytes;
    v.err_off = kOffErr;
    v.bar_off = kOffBar;
  }
  return v;
}
}  // namespace grus
