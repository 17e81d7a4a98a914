// preprocess.cu -- COO pairs -> degeneracy-ordered CSR, entirely on the GPU.
//
// Replaces the reference's single-threaded host pipeline:
//   Graph::LoadFromFile edge handling   src/graph.cc:64-152  (self-loops dropped,
//       u<v, sort+unique, dense relabel of present labels in ascending order)
//   Graph::SortByDegeneracy/ApplyOrder  src/graph.cc:281-306, 54-77
//   Graph::ConvertToCsr + LoadFromCpu   src/graph.cc:216-236, src/graph_gpu.cu:3-58
// Steps: pack (min,max) keys -> radix sort -> unique -> mark/scan dense ids ->
// the same edges by (max,min) by a second sort -> degrees and adjacency from
// the two sorted lists -> k-core peeling in synchronous rounds (one cooperative
// launch) -> both edge directions under the new ids, already ordered by column
// -> radix sort by row -> CSR -> root list (v0 < v1) by flag+scan.
//
// Every list that is built is a sorted one, so degrees are lengths of runs and
// places in a row are differences of positions: no counting or cursor atomics,
// which serialise on the hubs of a skewed graph (R-MAT 20: 3.9 of the build's
// 14.5 ms on a B200).
#include <algorithm>
#include <vector>

#include "barrier.h"
#include "common.cuh"
#include "engine.h"

namespace mce {

namespace {

constexpr uint64_t kInvalidKey = ~0ULL;

__global__ void k_pack_keys(const uint32_t *u, const uint32_t *v, uint64_t n, int bits, uint64_t *keys) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t a = u[i], b = v[i];
    if (a == b) {
      keys[i] = kInvalidKey;
      continue;
    }
    if (a > b) {
      uint32_t t = a;
      a = b;
      b = t;
    }
    keys[i] = ((uint64_t)a << bits) | b;
  }
}

__global__ void k_unique_flags(const uint64_t *keys, uint64_t n, uint32_t *flags) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t k = keys[i];
    flags[i] = (k != kInvalidKey && (i == 0 || keys[i - 1] != k)) ? 1u : 0u;
  }
}

__global__ void k_compact_keys(const uint64_t *keys, const uint32_t *flags, const uint32_t *pos, uint64_t n,
                               uint64_t *out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    if (flags[i]) out[pos[i]] = keys[i];
}

__global__ void k_mark_labels(const uint64_t *edges, uint64_t m, int bits, uint32_t *mark) {
  const uint64_t mask = (1ULL << bits) - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    mark[edges[i] >> bits] = 1;
    mark[edges[i] & mask] = 1;
  }
}

__global__ void k_labels_from_marks(const uint32_t *mark, const uint32_t *id, uint64_t nl, uint32_t *labels) {
  for (uint64_t l = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; l < nl; l += (uint64_t)gridDim.x * blockDim.x)
    if (mark[l]) labels[id[l]] = (uint32_t)l;
}

// edges (label pair) -> dense ids
__global__ void k_map_edges(uint64_t *edges, uint64_t m, int bits, const uint32_t *id, uint32_t *eu,
                            uint32_t *ev) {
  const uint64_t mask = (1ULL << bits) - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    eu[i] = id[edges[i] >> bits];
    ev[i] = id[edges[i] & mask];
  }
}

// the edges keyed by (larger id, smaller id)
__global__ void k_swap_keys(const uint32_t *eu, const uint32_t *ev, uint64_t m, int nb, uint64_t *keys) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x)
    keys[i] = ((uint64_t)ev[i] << nb) | eu[i];
}

// Where each vertex's run begins and ends in the edges by smaller id (eu: its
// larger neighbours) and by larger id (the keys' rows: its smaller ones);
// vertices without a run keep begin = end = 0.
__global__ void k_run_bounds(const uint32_t *eu, const uint64_t *by_v, uint64_t m, int nb, uint32_t *ub, uint32_t *ue,
                             uint32_t *lb, uint32_t *le) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t a = eu[i], b = (uint32_t)(by_v[i] >> nb);
    if (i == 0 || eu[i - 1] != a) ub[a] = (uint32_t)i;
    if (i == m - 1 || eu[i + 1] != a) ue[a] = (uint32_t)i + 1;
    if (i == 0 || (uint32_t)(by_v[i - 1] >> nb) != b) lb[b] = (uint32_t)i;
    if (i == m - 1 || (uint32_t)(by_v[i + 1] >> nb) != b) le[b] = (uint32_t)i + 1;
  }
}

__global__ void k_run_degrees(const uint32_t *ub, const uint32_t *ue, const uint32_t *lb, const uint32_t *le,
                              uint32_t n, uint32_t *deg) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    deg[v] = (ue[v] - ub[v]) + (le[v] - lb[v]);
}

// Row r of vertex v (rank[v], or v without ranks) starts at off[r]; its smaller
// neighbours come first.  The element at position i of a sorted edge list goes to i + (the list's base of
// v), modulo 2^32.
__global__ void k_run_bases(const uint32_t *off, const uint32_t *rank, const uint32_t *ub, const uint32_t *lb,
                            const uint32_t *le, uint32_t n, uint32_t *ubase, uint32_t *lbase) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint32_t o = off[rank ? rank[v] : v];
    lbase[v] = o - lb[v];
    ubase[v] = o + (le[v] - lb[v]) - ub[v];
  }
}

// The bases for rows that start at off_new[rank[v]] instead of off_old[v]: with
// them the runs' bounds, four words a vertex, need not be kept while peeling.
__global__ void k_move_bases(const uint32_t *off_old, const uint32_t *off_new, const uint32_t *rank, uint32_t n,
                             uint32_t *ubase, uint32_t *lbase) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint32_t by = off_new[rank[v]] - off_old[v];
    lbase[v] += by;
    ubase[v] += by;
  }
}

// symmetric adjacency for peeling
__global__ void k_fill_adj(const uint32_t *eu, const uint32_t *ev, const uint64_t *by_v, uint64_t m, int nb,
                           const uint32_t *ubase, const uint32_t *lbase, uint32_t *adj) {
  const uint64_t mask = (1ULL << nb) - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    adj[ubase[eu[i]] + (uint32_t)i] = ev[i];
    adj[lbase[by_v[i] >> nb] + (uint32_t)i] = (uint32_t)(by_v[i] & mask);
  }
}

__global__ void k_iota(uint32_t *a, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    a[i] = (uint32_t)i;
}

// ---- k-core peeling in synchronous rounds (one cooperative launch) ----
//
// Level k: the frontier F_0 = unremoved vertices of residual degree <= k; each
// round removes its whole frontier at once and decrements the neighbours, and
// every neighbour that drops to k joins the next round's frontier.  A vertex's
// position is (global round, vertex id): every later neighbour of x is either
// in x's round or in a later one, all of which were unremoved when x's
// residual degree fell to <= k, so x has at most k later neighbours -- a
// degeneracy order.  The rounds make the order deterministic, so root ids
// (edges of the ordered CSR) are stable from run to run; the reference's
// sequential queue (graph.cc:289-304) orders vertices inside a round
// differently, which changes neither the degeneracy nor the clique set.
// A skewed graph's core peels in hundreds of rounds with little work in most:
// the time is a round's chain of dependent L2 accesses and its barrier.  So
// counters are never reused (one per round and per level, cleared up front),
// which leaves one barrier a scan and one a round; the barrier is one counter
// that 148 blocks add to, with one fence a block; a frontier entry is the
// vertex's adjacency range, read when it is claimed; a warp keeps four
// neighbours in flight; and small rounds decrement a neighbour without asking
// first whether it is gone: a vertex removed at level k' <= k never has
// residual degree k + 1 again.
// Measured (B200): R-MAT 20 (192 levels, 622 rounds) 5.3 -> 4.1 ms, the core below
// included.
struct PeelCtl {
  uint32_t arrived;     // kBarrierStart + barrier arrivals so far
  uint32_t degeneracy;
  uint32_t rounds;
  uint32_t levels;
  uint32_t error;       // 1: level bound exceeded (cannot happen on a consistent CSR); 2: a barrier wait ran out
  // where the grid stopped, for the core kernel: nrem vertices left (0: none)
  // in list `list` (0: A, 1: B), level and round counts, next k
  uint32_t nrem, list, lev, r, k;
};
// The rest of a graph is peeled by one block once it fits that block's shared
// memory and is worth few enough neighbour visits.
constexpr uint32_t kCoreVertices = 16384, kCoreEntries = 3u << 20;
constexpr uint32_t kPeelThreads = 512;
// A barrier waits for the other blocks' share of a round, which is work that
// ends, so a caller's limit on idle polls does not cut it short: at least this
// many polls, most of a minute.
constexpr uint64_t kPeelSpinMin = 1ULL << 26;
// Frontiers from this size on ask first whether a neighbour is removed, which
// saves its atomic and costs a load before it.  Measured (B200), whole build, ms,
// for always, 256, 4096 and never: R-MAT 20 7.96, 7.88, 7.86, 7.82, Chung-Lu 10^6
// 5.14, 5.09, 5.10, 4.99: it matters little either way.
constexpr uint32_t kPeelAsk = 256;

// One barrier of the whole grid (all blocks are resident); false when the wait
// ran out.
__device__ __forceinline__ bool grid_barrier(PeelCtl *ctl, uint32_t *target, uint64_t spin_limit) {
  __shared__ uint32_t ok;
  *target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();  // the block's writes, ordered before this by the barrier above
    atomicAdd(&ctl->arrived, 1u);
    uint32_t seen = 0;
    uint64_t n = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&ctl->arrived) : "memory");
    } while (!barrier_reached(seen, *target) && ++n < spin_limit);
    ok = barrier_reached(seen, *target);
    if (!ok) atomicExch(&ctl->error, 2u);
  }
  __syncthreads();
  return ok != 0;
}

// fcnt[r]: vertices claimed into round r; rcnt[l], rmin[l], rsum[l]: survivors
// of level l's scan, their smallest residual degree and the sum of them.
__global__ void __launch_bounds__(kPeelThreads) k_peel_rounds(uint32_t n, const uint32_t *off, const uint32_t *adj,
                                                              int *deg, uint32_t *state, uint32_t *remA,
                                                              uint32_t *remB, uint2 *frA, uint2 *frB,
                                                              PeelCtl *ctl, uint32_t *fcnt, uint32_t *rcnt,
                                                              uint32_t *rmin, unsigned long long *rsum,
                                                              uint32_t max_levels,
                                                              uint64_t spin_limit) {
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t gwarp = tid >> 5, nwarps = nthreads >> 5;
  const bool leader = tid == 0;
  __shared__ uint32_t s_at[2][kPeelThreads / 32], s_min[kPeelThreads / 32];
  __shared__ unsigned long long s_sum[kPeelThreads / 32];
  uint32_t target = kBarrierStart;
  uint32_t k = 0, degen = 0, lev = 0, r = 0, removed = 0, nrem = n;
  uint32_t *rem_cur = remA, *rem_nxt = remB;
  while (removed < n) {
    if (lev > max_levels) {
      if (leader) atomicExch(&ctl->error, 1u);
      break;  // uniform: every thread sees the same lev
    }
    // the sum is from before the last level's rounds, so at least the true one
    if (lev && nrem <= kCoreVertices && __ldcg(&rsum[lev - 1]) <= kCoreEntries) {
      if (leader) {
        ctl->nrem = nrem;
        ctl->list = rem_cur == remB;
        ctl->lev = lev;
        ctl->r = r;
        ctl->k = k;
      }
      break;
    }
    uint2 *fr = (r & 1) ? frB : frA;
    // scan: claim residual degree <= k into F_r, keep the rest
    uint32_t local_min = 0xffffffffu;
    unsigned long long local_sum = 0;
    // block-uniform trip count; one atomic a block and list (every survivor is
    // appended at every level, and atomics on one counter serialise)
    for (uint64_t base = (uint64_t)blockIdx.x * kPeelThreads; base < nrem; base += nthreads) {
      const uint64_t i = base + threadIdx.x;
      uint32_t v = 0;
      int d = 0;
      bool claim = false, keep = false;
      if (i < nrem) {
        v = __ldcg(rem_cur + i);
        d = __ldcg(deg + v);
        if (!__ldcg(state + v)) {
          claim = d <= (int)k;
          keep = !claim;
        }
      }
      const uint32_t cm = __ballot_sync(kFull, claim), km = __ballot_sync(kFull, keep);
      if (lane == 0) {
        s_at[0][wid] = __popc(cm);
        s_at[1][wid] = __popc(km);
      }
      __syncthreads();
      if (wid < 2) {  // warp 0: claims, warp 1: survivors
        const uint32_t c = lane < kPeelThreads / 32 ? s_at[wid][lane] : 0;
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += y;
        }
        uint32_t at = 0;
        if (lane == 31 && incl) at = atomicAdd(wid ? &rcnt[lev] : &fcnt[r], incl);
        at = __shfl_sync(kFull, at, 31);
        if (lane < kPeelThreads / 32) s_at[wid][lane] = at + incl - c;
      }
      __syncthreads();
      if (claim) {
        state[v] = r + 1;
        fr[s_at[0][wid] + __popc(cm & lanemask_lt())] = make_uint2(off[v], off[v + 1]);
      } else if (keep) {
        rem_nxt[s_at[1][wid] + __popc(km & lanemask_lt())] = v;
        local_min = min(local_min, (uint32_t)d);
        local_sum += (uint32_t)d;
      }
      __syncthreads();
    }
    local_min = __reduce_min_sync(kFull, local_min);
    local_sum = warp_sum_u64(local_sum);
    if (lane == 0) {
      s_min[wid] = local_min;
      s_sum[wid] = local_sum;
    }
    __syncthreads();
    if (wid == 0) {
      local_min = __reduce_min_sync(kFull, lane < kPeelThreads / 32 ? s_min[lane] : 0xffffffffu);
      local_sum = warp_sum_u64(lane < kPeelThreads / 32 ? s_sum[lane] : 0);
      if (lane == 0 && local_min != 0xffffffffu) {
        atomicMin(&rmin[lev], local_min);
        atomicAdd(&rsum[lev], local_sum);
      }
    }
    if (!grid_barrier(ctl, &target, spin_limit)) return;
    uint32_t level_claims = 0;
    for (;;) {
      const uint32_t nf = __ldcg(&fcnt[r]);
      if (nf == 0) break;
      level_claims += nf;
      removed += nf;
      const uint2 *cur = (r & 1) ? frB : frA;
      uint2 *nxt = (r & 1) ? frA : frB;
      // Each frontier vertex's adjacency is shared by `per` warps (all the
      // grid's warps split evenly when the frontier is small: the dense
      // cores' hubs hold tens of thousands of neighbours each).
      const uint64_t per = nf < nwarps ? nwarps / nf : 1;
      for (uint64_t i = gwarp / per; i < nf; i += nwarps / per) {
        const uint2 range = __ldcg(cur + i);
        const uint32_t e1 = range.y;
        const uint32_t part = (uint32_t)(gwarp % per);
        const uint64_t step = 32ULL * per;
        for (uint64_t e = (uint64_t)range.x + 32ULL * part + lane; e < e1; e += 4 * step) {
          uint32_t u[4];
          bool open[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            open[j] = e + j * step < e1;
            u[j] = open[j] ? adj[e + j * step] : 0;
          }
          if (nf >= kPeelAsk) {
#pragma unroll
            for (int j = 0; j < 4; j++) open[j] = open[j] && !__ldcg(state + u[j]);
          }
          int was[4];
#pragma unroll
          for (int j = 0; j < 4; j++) was[j] = open[j] ? atomicSub(&deg[u[j]], 1) : 0;
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (open[j] && was[j] == (int)k + 1) {  // one decrement alone sees k + 1: it claims the vertex
              state[u[j]] = r + 2;
              const uint2 next = make_uint2(off[u[j]], off[u[j] + 1]);
              nxt[atomicAdd(&fcnt[r + 1], 1u)] = next;
            }
        }
      }
      if (!grid_barrier(ctl, &target, spin_limit)) return;
      r++;
    }
    // F_r is empty: round index r is skipped, so no vertex of the next level
    // shares a round number with this level's
    r++;
    nrem = __ldcg(&rcnt[lev]);
    const uint32_t least = __ldcg(&rmin[lev]);
    uint32_t *t = rem_cur;
    rem_cur = rem_nxt;
    rem_nxt = t;
    if (level_claims) {
      degen = k;
      k = k + 1;
    } else {
      if (least == 0xffffffffu) break;
      k = max(k + 1, least);
    }
    lev++;
    // The next scan needs no barrier of its own: the last one above came after
    // every decrement of this level, and the lists and counters the scan
    // writes are not read any more.
  }
  if (leader) {
    ctl->degeneracy = degen;
    ctl->rounds = r;
    ctl->levels = lev;
  }
}

// The vertices that are left: their numbers in the list, and their residual
// degrees, which are their numbers of neighbours left.  One of the list's
// vertices may have been claimed in the level's last rounds: degree 0 here.
__global__ void k_core_ids(const PeelCtl *ctl, const uint32_t *remA, const uint32_t *remB, const uint32_t *state,
                           const int *deg, uint32_t *id, uint32_t *cdeg) {
  const uint32_t *rem = ctl->list ? remB : remA;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < kCoreVertices; i += gridDim.x * blockDim.x) {
    uint32_t d = 0;
    if (i < ctl->nrem) {
      const uint32_t v = rem[i];
      id[v] = i;
      if (!state[v]) d = (uint32_t)deg[v];
    }
    cdeg[i] = d;
  }
}

// their adjacency among themselves (in any order), one block a vertex: a hub
// still has its whole list
__global__ void __launch_bounds__(256) k_core_fill(const PeelCtl *ctl, const uint32_t *remA, const uint32_t *remB,
                                                   const uint32_t *off, const uint32_t *adj, const uint32_t *state,
                                                   const uint32_t *id, const uint32_t *coff, uint16_t *cadj) {
  __shared__ uint32_t s_at;
  const uint32_t *rem = ctl->list ? remB : remA;
  const uint32_t lane = threadIdx.x & 31, nrem = ctl->nrem;
  for (uint32_t i = blockIdx.x; i < nrem; i += gridDim.x) {
    const uint32_t v = rem[i];
    if (state[v]) continue;
    if (threadIdx.x == 0) s_at = coff[i];
    __syncthreads();
    const uint32_t e1 = off[v + 1];
    for (uint64_t base = (uint64_t)off[v] + threadIdx.x - lane; base < e1; base += 4 * 256) {
      uint32_t u[4];
      bool left[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        left[j] = base + j * 256 + lane < e1;
        u[j] = left[j] ? adj[base + j * 256 + lane] : 0;
      }
#pragma unroll
      for (int j = 0; j < 4; j++) left[j] = left[j] && !state[u[j]];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t bal = __ballot_sync(kFull, left[j]);
        uint32_t at = 0;
        if (lane == 0 && bal) at = atomicAdd(&s_at, (uint32_t)__popc(bal));
        at = __shfl_sync(kFull, at, 0);
        if (left[j]) cadj[at + __popc(bal & lanemask_lt())] = (uint16_t)id[u[j]];
      }
    }
    __syncthreads();
  }
}

// The remaining rounds, in one block: residual degrees (negative once removed),
// list offsets and frontiers in shared memory, so that a round waits on one
// global load, the neighbours.  A round of the whole grid costs about 5 us,
// nearly all of it dependent L2 accesses and the barrier; here it costs 1 to
// 2 us.  Same rounds, so same order.
// Measured (B200), whole build: R-MAT 14 (all of it here) 1.65 -> 1.38 ms,
// R-MAT 17 3.1 -> 2.9 ms; 6 M entries instead of 3 M cost R-MAT 20 0.5 ms.
constexpr uint32_t kCoreThreads = 1024;
constexpr size_t kCoreSmem = (kCoreVertices + 4) * (2 * sizeof(int) + 2 * sizeof(uint16_t));

__global__ void __launch_bounds__(kCoreThreads) k_peel_core(PeelCtl *ctl, const uint32_t *remA, const uint32_t *remB,
                                                            uint32_t *state, const uint32_t *cdeg,
                                                            const uint32_t *coff, const uint16_t *cadj,
                                                            uint32_t *cround) {
  extern __shared__ int sdeg[];
  uint32_t *soff = (uint32_t *)(sdeg + kCoreVertices);  // n + 1
  uint16_t *fr[2] = {(uint16_t *)(soff + kCoreVertices + 4), (uint16_t *)(soff + kCoreVertices + 4) + kCoreVertices};
  __shared__ uint32_t cnt[3];  // frontier sizes, by round mod 3
  __shared__ uint32_t s_min;
  const uint32_t n = ctl->nrem;
  if (n == 0) return;
  const uint32_t *rem = ctl->list ? remB : remA;
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nwarps = kCoreThreads / 32;
  constexpr int kGone = -(1 << 30);
  uint32_t gone = 0;
  for (uint32_t i = tid; i < n; i += kCoreThreads) {
    const bool left = !state[rem[i]];
    sdeg[i] = left ? (int)cdeg[i] : kGone;
    cround[i] = 0;
    gone += !left;
  }
  for (uint32_t i = tid; i <= n; i += kCoreThreads) soff[i] = coff[i];
  if (tid < 3) cnt[tid] = 0;
  __syncthreads();
  if (gone) atomicAdd(&cnt[0], gone);
  __syncthreads();
  uint32_t left = n - cnt[0];
  uint32_t k = ctl->k, r = ctl->r, lev = ctl->lev, degen = ctl->degeneracy;
  __syncthreads();
  if (tid == 0) cnt[0] = 0;
  while (left) {
    if (tid == 0) s_min = 0xffffffffu;
    __syncthreads();
    // scan: claim residual degree <= k
    uint32_t least = 0xffffffffu;
    for (uint32_t base = tid - lane; base < n; base += kCoreThreads) {
      const uint32_t i = base + lane;
      const int d = i < n ? sdeg[i] : kGone;
      const bool claim = d >= 0 && d <= (int)k;
      if (d > (int)k) least = min(least, (uint32_t)d);
      const uint32_t bal = __ballot_sync(kFull, claim);
      uint32_t at = 0;
      if (lane == 0 && bal) at = atomicAdd(&cnt[r % 3], (uint32_t)__popc(bal));
      at = __shfl_sync(kFull, at, 0);
      if (claim) {
        sdeg[i] = kGone;
        cround[i] = r + 1;
        fr[r & 1][at + __popc(bal & lanemask_lt())] = (uint16_t)i;
      }
    }
    least = __reduce_min_sync(kFull, least);
    if (lane == 0 && least != 0xffffffffu) atomicMin(&s_min, least);
    __syncthreads();
    uint32_t claims = 0;
    for (;;) {
      const uint32_t nf = cnt[r % 3];
      if (nf == 0) break;
      claims += nf;
      left -= nf;
      if (tid == 0) cnt[(r + 2) % 3] = 0;  // last read in round r - 1
      const uint16_t *cur = fr[r & 1];
      uint16_t *nxt = fr[(r + 1) & 1];
      const uint32_t per = nf < nwarps ? nwarps / nf : 1;
      for (uint32_t i = wid / per; i < nf; i += nwarps / per) {
        const uint32_t x = cur[i], e1 = soff[x + 1], step = 32 * per;
        for (uint32_t e = soff[x] + 32 * (wid % per) + lane; e < e1; e += 4 * step) {
          uint32_t u[4];
#pragma unroll
          for (int j = 0; j < 4; j++) u[j] = e + j * step < e1 ? cadj[e + j * step] : 0xffffffffu;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (u[j] == 0xffffffffu || atomicSub(&sdeg[u[j]], 1) != (int)k + 1) continue;
            sdeg[u[j]] = kGone;
            cround[u[j]] = r + 2;
            nxt[atomicAdd(&cnt[(r + 1) % 3], 1u)] = (uint16_t)u[j];
          }
        }
      }
      __syncthreads();
      r++;
    }
    // as on the grid: an empty round separates the levels
    r++;
    if (claims) {
      degen = k;
      k++;
    } else {
      k = max(k + 1, s_min);
    }
    lev++;
    __syncthreads();
    if (tid < 3) cnt[tid] = 0;
  }
  __syncthreads();
  for (uint32_t i = tid; i < n; i += kCoreThreads)
    if (cround[i]) state[rem[i]] = cround[i];
  if (tid == 0) {
    ctl->degeneracy = degen;
    ctl->rounds = r;
    ctl->levels = lev;
  }
}

__global__ void k_round_keys(const uint32_t *state, uint32_t n, int nb, uint64_t *keys) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    keys[i] = ((uint64_t)(state[i] - 1) << nb) | i;
}

__global__ void k_order_from_round_keys(const uint64_t *keys, uint32_t n, uint64_t mask, uint32_t *order) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    order[i] = (uint32_t)(keys[i] & mask);
}

__global__ void k_rank_from_order(const uint32_t *order, uint32_t n, uint32_t *rank) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) rank[order[i]] = i;
}

__global__ void k_permute_degrees(const uint32_t *deg, const uint32_t *rank, uint32_t n, uint32_t *deg_new) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) deg_new[rank[i]] = deg[i];
}

// Both directions of every edge under the new ids, packed (row << nb) | col.
// Vertex v's edges are written with v as the column, in v's new row: the list
// comes out ordered by column, and a stable sort by row alone finishes it.
__global__ void k_relabel_keys(const uint32_t *eu, const uint32_t *ev, const uint64_t *by_v, uint64_t m,
                               const uint32_t *rank, const uint32_t *ubase, const uint32_t *lbase, int nb,
                               uint64_t *keys) {
  const uint64_t mask = (1ULL << nb) - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t u = eu[i], v = (uint32_t)(by_v[i] >> nb);
    keys[ubase[u] + (uint32_t)i] = ((uint64_t)rank[ev[i]] << nb) | rank[u];
    keys[lbase[v] + (uint32_t)i] = ((uint64_t)rank[by_v[i] & mask] << nb) | rank[v];
  }
}

__global__ void k_csr_cols(const uint64_t *keys, uint64_t m2, int nb, uint32_t *adj, uint32_t *upflag) {
  const uint64_t mask = (1ULL << nb) - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m2; i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t r = (uint32_t)(keys[i] >> nb), c = (uint32_t)(keys[i] & mask);
    adj[i] = c;
    upflag[i] = r < c ? 1u : 0u;
  }
}

__global__ void k_roots(const uint64_t *keys, uint64_t m2, int nb, const uint32_t *upflag, const uint32_t *pos,
                        uint32_t *root_v0, uint32_t *root_v1) {
  const uint64_t mask = (1ULL << nb) - 1;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m2; i += (uint64_t)gridDim.x * blockDim.x)
    if (upflag[i]) {
      root_v0[pos[i]] = (uint32_t)(keys[i] >> nb);
      root_v1[pos[i]] = (uint32_t)(keys[i] & mask);
    }
}

// first root of each vertex: the roots before its row
__global__ void k_root_off(const uint32_t *off, const uint32_t *pos, uint32_t n, uint32_t *root_off) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x)
    root_off[v] = pos[off[v]];
}

__global__ void k_permute_labels(const uint32_t *labels_old, const uint32_t *rank, uint32_t n, uint32_t *labels,
                                 uint64_t *h1, uint64_t *h2) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t l = labels_old[i];
    uint32_t r = rank ? rank[i] : i;
    labels[r] = l;
    h1[r] = mix64((uint64_t)l);
    h2[r] = mix64((uint64_t)l ^ kGolden);
  }
}

__global__ void k_degree_keys(const uint32_t *deg, uint32_t n, int desc, uint64_t *keys) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t d = desc ? ~deg[i] : deg[i];
    keys[i] = ((uint64_t)d << 32) | i;
  }
}

__global__ void k_order_from_keys(const uint64_t *keys, uint32_t n, uint32_t *order) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    order[i] = (uint32_t)keys[i];
}

int bits_for(uint64_t maxval) {
  int b = 1;
  while (b < 64 && (maxval >> b) != 0) b++;
  return b;
}

template <typename T>
struct DevBuf {
  T *p = nullptr;
  cudaStream_t st = nullptr;
  mce_status alloc(size_t n, cudaStream_t s) {
    st = s;
    if (cudaMallocAsync(&p, std::max<size_t>(n, 1) * sizeof(T), s) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
      return MCE_ERR_OUT_OF_MEMORY;
    }
    return MCE_OK;
  }
  void release() {
    if (p) cudaFreeAsync(p, st);
    p = nullptr;
  }
  ~DevBuf() { release(); }
};

template <typename T>
mce_status read_scalar(const T *d, T *h, cudaStream_t st) {
  MCE_CUDA_TRY(cudaMemcpyAsync(h, d, sizeof(T), cudaMemcpyDeviceToHost, st));
  MCE_CUDA_TRY(cudaStreamSynchronize(st));
  return MCE_OK;
}

// k-core peeling over an unsorted symmetric CSR; allocates and fills order[] (position -> vertex)
mce_status peel(uint32_t n, const uint32_t *off, const uint32_t *adj, const uint32_t *deg0, uint32_t max_degree,
                uint64_t entries, DevBuf<uint32_t> &order, uint32_t *degeneracy, uint64_t spin_limit, cudaStream_t st) {
  DevBuf<int> deg;
  DevBuf<uint32_t> state, remA, remB;
  DevBuf<uint2> frA, frB;
  DevBuf<PeelCtl> ctl;
  MCE_TRY(deg.alloc(n, st));
  MCE_TRY(state.alloc(n, st));
  MCE_TRY(remA.alloc(n, st));
  MCE_TRY(remB.alloc(n, st));
  MCE_TRY(frA.alloc(n, st));
  MCE_TRY(frB.alloc(n, st));
  MCE_TRY(ctl.alloc(1, st));
  MCE_CUDA_TRY(cudaMemcpyAsync(deg.p, deg0, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  MCE_CUDA_TRY(cudaMemsetAsync(state.p, 0, n * sizeof(uint32_t), st));
  k_iota<<<grid_for(n, 256), 256, 0, st>>>(remA.p, n); note_launch();
  // one counter a round (every round but the last of a level claims a vertex)
  // and two a level
  spin_limit = std::max(spin_limit, kPeelSpinMin);
  const uint64_t max_levels = (uint64_t)max_degree + 2, max_rounds = (uint64_t)n + max_levels + 4;
  const bool core_only = n <= kCoreVertices && entries <= kCoreEntries;
  DevBuf<uint32_t> counters;
  DevBuf<unsigned long long> sums;
  if (!core_only) {
    MCE_TRY(counters.alloc(max_rounds + 2 * (max_levels + 2), st));
    MCE_TRY(sums.alloc(max_levels + 2, st));
  }
  uint32_t *fcnt = counters.p, *rcnt = fcnt + max_rounds, *rmin = rcnt + max_levels + 2;
  unsigned long long *rsum = sums.p;
  // the control block goes through ordinary host memory: pinning it for each
  // build (and unpinning, which synchronises the device) would stall other
  // streams' work, e.g. concurrently served requests
  PeelCtl h{};
  h.arrived = kBarrierStart;
  PeelCtl *hc = &h;
  if (core_only) h.nrem = n;
  MCE_CUDA_TRY(cudaMemcpyAsync(ctl.p, hc, sizeof(PeelCtl), cudaMemcpyHostToDevice, st));
  if (!core_only) {
    MCE_CUDA_TRY(cudaMemsetAsync(fcnt, 0, (max_rounds + max_levels + 2) * sizeof(uint32_t), st));
    MCE_CUDA_TRY(cudaMemsetAsync(rmin, 0xff, (max_levels + 2) * sizeof(uint32_t), st));
    MCE_CUDA_TRY(cudaMemsetAsync(rsum, 0, (max_levels + 2) * sizeof(unsigned long long), st));
    int dev = 0, sms = 0, per_sm = 0;
    MCE_CUDA_TRY(cudaGetDevice(&dev));
    MCE_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MCE_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_peel_rounds, kPeelThreads, 0));
    if (per_sm < 1) return MCE_ERR_INTERNAL;
    // a cooperative launch: every block is resident, so the barrier is sound
    const uint32_t blocks = (uint32_t)sms;
    uint32_t nn = n, maxl = (uint32_t)max_levels;
    int *degp = deg.p;
    uint32_t *statep = state.p, *ra = remA.p, *rb = remB.p;
    uint2 *fa = frA.p, *fb = frB.p;
    PeelCtl *cp = ctl.p;
    void *args[] = {&nn, (void *)&off, (void *)&adj, &degp, &statep, &ra, &rb, &fa, &fb, &cp, &fcnt, &rcnt, &rmin, &rsum,
                    &maxl, &spin_limit};
    MCE_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_peel_rounds, dim3(blocks), dim3(kPeelThreads), args, 0, st));
    note_launch();
  }
  {
    DevBuf<uint32_t> core;  // residual degrees and offsets of the vertices left
    DevBuf<uint16_t> cadj;
    MCE_TRY(core.alloc(3 * kCoreVertices + 1, st));
    MCE_TRY(cadj.alloc(std::min<uint64_t>(entries, kCoreEntries), st));
    uint32_t *cdeg = core.p, *coff = cdeg + kCoreVertices, *cround = coff + kCoreVertices + 1;
    uint32_t *id = (uint32_t *)frA.p;
    k_core_ids<<<kCoreVertices / 256, 256, 0, st>>>(ctl.p, remA.p, remB.p, state.p, deg.p, id, cdeg); note_launch();
    MCE_TRY(scan_exclusive_u32(cdeg, coff, kCoreVertices, coff + kCoreVertices, st));
    k_core_fill<<<grid_for(std::min(n, kCoreVertices), 1, 148 * 8), 256, 0, st>>>(ctl.p, remA.p, remB.p, off, adj, state.p, id, coff, cadj.p); note_launch();
    MCE_CUDA_TRY(cudaFuncSetAttribute(k_peel_core, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoreSmem));
    k_peel_core<<<1, kCoreThreads, kCoreSmem, st>>>(ctl.p, remA.p, remB.p, state.p, cdeg, coff, cadj.p,
                                                      cround); note_launch();
    MCE_CUDA_TRY(cudaGetLastError());
  }
  MCE_CUDA_TRY(cudaMemcpyAsync(hc, ctl.p, sizeof(PeelCtl), cudaMemcpyDeviceToHost, st));
  MCE_CUDA_TRY(cudaStreamSynchronize(st));
  if (h.error) return h.error == 2 ? MCE_ERR_TIMEOUT : MCE_ERR_INTERNAL;
  *degeneracy = h.degeneracy;
  // order = vertices sorted by (round, id)
  const int nb = bits_for(n ? n - 1 : 0), rb_bits = bits_for(h.rounds);
  if (nb + rb_bits > 64) return MCE_ERR_TOO_LARGE;
  DevBuf<uint64_t> keys, tmp;
  MCE_TRY(keys.alloc(n, st));
  MCE_TRY(tmp.alloc(n, st));
  k_round_keys<<<grid_for(n, 256), 256, 0, st>>>(state.p, n, nb, keys.p); note_launch();
  // the keys are in vertex order already: a stable sort by round finishes them
  MCE_TRY(radix_sort_u64(keys.p, tmp.p, n, nb, nb + rb_bits, st));
  MCE_TRY(order.alloc(n, st));
  k_order_from_round_keys<<<grid_for(n, 256), 256, 0, st>>>(keys.p, n, (1ULL << nb) - 1, order.p); note_launch();
  MCE_CUDA_TRY(cudaGetLastError());
  return MCE_OK;
}

}  // namespace

namespace {

__global__ void k_pack_keys64(const uint32_t *u, const uint32_t *v, uint64_t n, uint64_t *keys) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t a = u[i], b = v[i];
    if (a == b) {
      keys[i] = kInvalidKey;  // (a < b) keys never reach all-ones
      continue;
    }
    if (a > b) {
      uint32_t t = a;
      a = b;
      b = t;
    }
    keys[i] = ((uint64_t)a << 32) | b;
  }
}

__global__ void k_endpoints(const uint64_t *edges, uint64_t m, uint64_t *ends) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    ends[2 * i] = edges[i] >> 32;
    ends[2 * i + 1] = edges[i] & 0xffffffffULL;
  }
}

__global__ void k_labels_from_sorted(const uint64_t *ends, const uint32_t *flag, const uint32_t *pos, uint64_t k,
                                     uint32_t *labels) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k; i += (uint64_t)gridDim.x * blockDim.x)
    if (flag[i]) labels[pos[i]] = (uint32_t)ends[i];
}

__device__ __forceinline__ uint32_t find_label(const uint32_t *labels, uint32_t n, uint32_t l) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (labels[mid] < l) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__global__ void k_map_edges_search(const uint64_t *edges, uint64_t m, const uint32_t *labels, uint32_t n,
                                   uint32_t *eu, uint32_t *ev) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    eu[i] = find_label(labels, n, (uint32_t)(edges[i] >> 32));
    ev[i] = find_label(labels, n, (uint32_t)(edges[i] & 0xffffffffULL));
  }
}

// present labels, ascending, by sorting the 2m endpoints; ids by binary search
mce_status build_sparse_labels(const uint32_t *u, const uint32_t *v, uint64_t np, int order_kind,
                               uint64_t spin_limit, cudaStream_t st, DeviceGraph *g) {
  if (np >= (1ULL << 32)) return MCE_ERR_TOO_LARGE;
  DevBuf<uint64_t> keys, tmp;
  MCE_TRY(keys.alloc(np, st));
  MCE_TRY(tmp.alloc(np, st));
  k_pack_keys64<<<grid_for(np, 256), 256, 0, st>>>(u, v, np, keys.p); note_launch();
  MCE_TRY(radix_sort_u64(keys.p, tmp.p, np, 0, 64, st));
  DevBuf<uint32_t> flags, pos;
  MCE_TRY(flags.alloc(np + 1, st));
  MCE_TRY(pos.alloc(np + 1, st));
  k_unique_flags<<<grid_for(np, 256), 256, 0, st>>>(keys.p, np, flags.p); note_launch();
  MCE_TRY(scan_exclusive_u32(flags.p, pos.p, np, pos.p + np, st));
  uint32_t m32 = 0;
  MCE_TRY(read_scalar(pos.p + np, &m32, st));
  const uint64_t m = m32;
  if (2 * m >= (1ULL << 32)) return MCE_ERR_TOO_LARGE;
  DevBuf<uint64_t> edges;
  MCE_TRY(edges.alloc(m, st));
  k_compact_keys<<<grid_for(np, 256), 256, 0, st>>>(keys.p, flags.p, pos.p, np, edges.p); note_launch();
  keys.release();
  tmp.release();
  flags.release();
  pos.release();
  const uint64_t k = 2 * m;
  DevBuf<uint64_t> ends, etmp;
  MCE_TRY(ends.alloc(k, st));
  MCE_TRY(etmp.alloc(k, st));
  k_endpoints<<<grid_for(m, 256), 256, 0, st>>>(edges.p, m, ends.p); note_launch();
  MCE_TRY(radix_sort_u64(ends.p, etmp.p, k, 0, 32, st));
  etmp.release();
  DevBuf<uint32_t> f2, p2;
  MCE_TRY(f2.alloc(k + 1, st));
  MCE_TRY(p2.alloc(k + 1, st));
  k_unique_flags<<<grid_for(k, 256), 256, 0, st>>>(ends.p, k, f2.p); note_launch();
  MCE_TRY(scan_exclusive_u32(f2.p, p2.p, k, p2.p + k, st));
  uint32_t n = 0;
  MCE_TRY(read_scalar(p2.p + k, &n, st));
  DevBuf<uint32_t> labels0, eu, ev;
  MCE_TRY(labels0.alloc(n, st));
  MCE_TRY(eu.alloc(m, st));
  MCE_TRY(ev.alloc(m, st));
  k_labels_from_sorted<<<grid_for(k, 256), 256, 0, st>>>(ends.p, f2.p, p2.p, k, labels0.p); note_launch();
  k_map_edges_search<<<grid_for(m, 256), 256, 0, st>>>(edges.p, m, labels0.p, n, eu.p, ev.p); note_launch();
  ends.release();
  f2.release();
  p2.release();
  edges.release();
  MCE_TRY(finish_graph(n, m, eu.p, ev.p, labels0.p, order_kind, spin_limit, st, g));
  return MCE_OK;
}

}  // namespace

mce_status build_from_pairs(const uint32_t *u, const uint32_t *v, uint64_t np, int order_kind,
                            uint64_t spin_limit, cudaStream_t st, DeviceGraph *g) {
  *g = DeviceGraph{};
  DevBuf<uint32_t> maxbuf;
  MCE_TRY(maxbuf.alloc(2, st));
  MCE_TRY(reduce_max_u32(u, np, maxbuf.p, st));
  MCE_TRY(reduce_max_u32(v, np, maxbuf.p + 1, st));
  uint32_t hm[2] = {0, 0};
  MCE_CUDA_TRY(cudaMemcpyAsync(hm, maxbuf.p, sizeof(hm), cudaMemcpyDeviceToHost, st));
  MCE_CUDA_TRY(cudaStreamSynchronize(st));
  const uint32_t maxlab = std::max(hm[0], hm[1]);
  // labels much sparser than the pair count (or near 2^32): sort-based relabel
  if (maxlab >= (1u << 30) || (uint64_t)maxlab > 8 * np + (1u << 20))
    return build_sparse_labels(u, v, np, order_kind, spin_limit, st, g);
  const int lb = bits_for(maxlab);
  if (2 * lb > 63) return MCE_ERR_TOO_LARGE;

  // 1) normalised (min,max) keys, sorted, unique
  DevBuf<uint64_t> keys, tmp;
  MCE_TRY(keys.alloc(np, st));
  MCE_TRY(tmp.alloc(np, st));
  k_pack_keys<<<grid_for(np, 256), 256, 0, st>>>(u, v, np, lb, keys.p); note_launch();
  MCE_TRY(radix_sort_u64(keys.p, tmp.p, np, 0, 2 * lb, st));
  DevBuf<uint32_t> flags, pos;
  MCE_TRY(flags.alloc(np + 1, st));
  MCE_TRY(pos.alloc(np + 1, st));
  k_unique_flags<<<grid_for(np, 256), 256, 0, st>>>(keys.p, np, flags.p); note_launch();
  MCE_TRY(scan_exclusive_u32(flags.p, pos.p, np, pos.p + np, st));
  uint32_t m32 = 0;
  MCE_TRY(read_scalar(pos.p + np, &m32, st));
  const uint64_t m = m32;
  if (np > 0xffffffffULL || 2 * m >= (1ULL << 32)) return MCE_ERR_TOO_LARGE;
  DevBuf<uint64_t> edges;
  MCE_TRY(edges.alloc(m, st));
  k_compact_keys<<<grid_for(np, 256), 256, 0, st>>>(keys.p, flags.p, pos.p, np, edges.p); note_launch();
  keys.release();
  tmp.release();
  flags.release();
  pos.release();

  // 2) dense ids of present labels, ascending (src/graph.cc:123-130)
  const uint64_t nl = (uint64_t)maxlab + 1;
  DevBuf<uint32_t> mark, id;
  MCE_TRY(mark.alloc(nl + 1, st));
  MCE_TRY(id.alloc(nl + 1, st));
  MCE_CUDA_TRY(cudaMemsetAsync(mark.p, 0, nl * sizeof(uint32_t), st));
  k_mark_labels<<<grid_for(m, 256), 256, 0, st>>>(edges.p, m, lb, mark.p); note_launch();
  MCE_TRY(scan_exclusive_u32(mark.p, id.p, nl, id.p + nl, st));
  uint32_t n = 0;
  MCE_TRY(read_scalar(id.p + nl, &n, st));
  DevBuf<uint32_t> labels0, eu, ev;
  MCE_TRY(labels0.alloc(n, st));
  MCE_TRY(eu.alloc(m, st));
  MCE_TRY(ev.alloc(m, st));
  k_labels_from_marks<<<grid_for(nl, 256), 256, 0, st>>>(mark.p, id.p, nl, labels0.p); note_launch();
  k_map_edges<<<grid_for(m, 256), 256, 0, st>>>(edges.p, m, lb, id.p, eu.p, ev.p); note_launch();
  mark.release();
  id.release();
  edges.release();
  MCE_TRY(finish_graph(n, m, eu.p, ev.p, labels0.p, order_kind, spin_limit, st, g));
  return MCE_OK;
}

// eu/ev: m edges eu < ev on dense ids, sorted by (eu, ev), without duplicates;
// labels0: original labels of the dense ids.
mce_status finish_graph(uint32_t n, uint64_t m, const uint32_t *eu, const uint32_t *ev, const uint32_t *labels0,
                        int order_kind, uint64_t spin_limit, cudaStream_t st, DeviceGraph *g) {
  *g = DeviceGraph{};
  g->n = n;
  g->m = m;
  g->stream = st;
  if (2 * m >= (1ULL << 32)) return MCE_ERR_TOO_LARGE;
  const int nb = bits_for(n ? n - 1 : 0);
  const uint64_t m2 = 2 * m;
  // the edges by larger id, and every vertex's runs in both lists
  DevBuf<uint64_t> by_v, tmp_v;
  MCE_TRY(by_v.alloc(m, st));
  MCE_TRY(tmp_v.alloc(m, st));
  k_swap_keys<<<grid_for(m, 256), 256, 0, st>>>(eu, ev, m, nb, by_v.p); note_launch();
  MCE_TRY(radix_sort_u64(by_v.p, tmp_v.p, m, nb, 2 * nb, st));
  tmp_v.release();
  DevBuf<uint32_t> runs, bases, deg;
  MCE_TRY(runs.alloc(4ULL * n, st));
  MCE_TRY(bases.alloc(2ULL * n, st));
  MCE_TRY(deg.alloc(n + 1, st));
  uint32_t *ub = runs.p, *ue = ub + n, *lb = ue + n, *le = lb + n, *ubase = bases.p, *lbase = ubase + n;
  MCE_CUDA_TRY(cudaMemsetAsync(runs.p, 0, 4ULL * n * sizeof(uint32_t), st));
  k_run_bounds<<<grid_for(m, 256), 256, 0, st>>>(eu, by_v.p, m, nb, ub, ue, lb, le); note_launch();
  k_run_degrees<<<grid_for(n, 256), 256, 0, st>>>(ub, ue, lb, le, n, deg.p); note_launch();
  DevBuf<uint32_t> maxd;
  MCE_TRY(maxd.alloc(1, st));
  MCE_TRY(reduce_max_u32(deg.p, n, maxd.p, st));
  MCE_TRY(read_scalar(maxd.p, &g->max_degree, st));

  // 3) vertex order
  DevBuf<uint32_t> order, rank, off0;  // off0: row starts under the old ids, degeneracy order only
  g->degeneracy = g->max_degree;  // Graph::LoadFromFile leaves degeneracy_ = max degree (graph.cc:149)
  if (order_kind == MCE_ORDER_DEGENERACY && n > 0) {
    DevBuf<uint32_t> adj0;
    MCE_TRY(off0.alloc(n + 1, st));
    MCE_TRY(adj0.alloc(m2, st));
    MCE_TRY(scan_exclusive_u32(deg.p, off0.p, n, off0.p + n, st));
    k_run_bases<<<grid_for(n, 256), 256, 0, st>>>(off0.p, nullptr, ub, lb, le, n, ubase, lbase); note_launch();
    runs.release();
    k_fill_adj<<<grid_for(m, 256), 256, 0, st>>>(eu, ev, by_v.p, m, nb, ubase, lbase, adj0.p); note_launch();
    MCE_TRY(peel(n, off0.p, adj0.p, deg.p, g->max_degree, m2, order, &g->degeneracy, spin_limit, st));
  } else if ((order_kind == MCE_ORDER_DEGREE_ASC || order_kind == MCE_ORDER_DEGREE_DESC) && n > 0) {
    DevBuf<uint64_t> dk, dt;
    MCE_TRY(dk.alloc(n, st));
    MCE_TRY(dt.alloc(n, st));
    k_degree_keys<<<grid_for(n, 256), 256, 0, st>>>(deg.p, n, order_kind == MCE_ORDER_DEGREE_DESC, dk.p); note_launch();
    MCE_TRY(radix_sort_u64(dk.p, dt.p, n, 0, 64, st));
    MCE_TRY(order.alloc(n, st));
    k_order_from_keys<<<grid_for(n, 256), 256, 0, st>>>(dk.p, n, order.p); note_launch();
  } else {
    MCE_TRY(order.alloc(n, st));
    k_iota<<<grid_for(n, 256), 256, 0, st>>>(order.p, n); note_launch();
  }
  MCE_TRY(rank.alloc(n, st));
  k_rank_from_order<<<grid_for(n, 256), 256, 0, st>>>(order.p, n, rank.p); note_launch();
  order.release();

  // 4) relabelled symmetric edge keys -> sorted CSR
  DevBuf<uint64_t> keys, tmp;
  MCE_TRY(keys.alloc(m2, st));
  MCE_TRY(tmp.alloc(m2, st));
  DevBuf<uint32_t> deg_new;
  MCE_TRY(deg_new.alloc(n + 1, st));
  k_permute_degrees<<<grid_for(n, 256), 256, 0, st>>>(deg.p, rank.p, n, deg_new.p); note_launch();
  MCE_CUDA_TRY(cudaMallocAsync(&g->off, (n + 1) * sizeof(uint32_t), st));
  MCE_TRY(scan_exclusive_u32(deg_new.p, g->off, n, g->off + n, st));
  if (off0.p) {
    k_move_bases<<<grid_for(n, 256), 256, 0, st>>>(off0.p, g->off, rank.p, n, ubase, lbase); note_launch();
  } else {
    k_run_bases<<<grid_for(n, 256), 256, 0, st>>>(g->off, rank.p, ub, lb, le, n, ubase, lbase); note_launch();
  }
  k_relabel_keys<<<grid_for(m, 256), 256, 0, st>>>(eu, ev, by_v.p, m, rank.p, ubase, lbase, nb, keys.p); note_launch();
  by_v.release();
  MCE_TRY(radix_sort_u64(keys.p, tmp.p, m2, nb, 2 * nb, st));
  tmp.release();
  MCE_CUDA_TRY(cudaMallocAsync(&g->adj, std::max<uint64_t>(m2, 1) * sizeof(uint32_t), st));
  DevBuf<uint32_t> upflag, uppos;
  MCE_TRY(upflag.alloc(m2 + 1, st));
  MCE_TRY(uppos.alloc(m2 + 1, st));
  k_csr_cols<<<grid_for(m2, 256), 256, 0, st>>>(keys.p, m2, nb, g->adj, upflag.p); note_launch();
  MCE_TRY(scan_exclusive_u32(upflag.p, uppos.p, m2, uppos.p + m2, st));
  MCE_CUDA_TRY(cudaMallocAsync(&g->root_v0, std::max<uint64_t>(m, 1) * sizeof(uint32_t), st));
  MCE_CUDA_TRY(cudaMallocAsync(&g->root_v1, std::max<uint64_t>(m, 1) * sizeof(uint32_t), st));
  k_roots<<<grid_for(m2, 256), 256, 0, st>>>(keys.p, m2, nb, upflag.p, uppos.p, g->root_v0, g->root_v1); note_launch();
  MCE_CUDA_TRY(cudaMallocAsync(&g->root_off, (n + 1) * sizeof(uint32_t), st));
  k_root_off<<<grid_for(n + 1, 256), 256, 0, st>>>(g->off, uppos.p, n, g->root_off); note_launch();
  keys.release();

  // 5) labels and their hashes under the new ids
  MCE_CUDA_TRY(cudaMallocAsync(&g->labels, std::max<uint32_t>(n, 1) * sizeof(uint32_t), st));
  MCE_CUDA_TRY(cudaMallocAsync(&g->h1, std::max<uint32_t>(n, 1) * sizeof(uint64_t), st));
  MCE_CUDA_TRY(cudaMallocAsync(&g->h2, std::max<uint32_t>(n, 1) * sizeof(uint64_t), st));
  k_permute_labels<<<grid_for(n, 256), 256, 0, st>>>(labels0, rank.p, n, g->labels, g->h1, g->h2); note_launch();
  MCE_CUDA_TRY(cudaGetLastError());
  MCE_CUDA_TRY(cudaStreamSynchronize(st));
  return MCE_OK;
}

// CSR given by the caller (rows sorted).  already_ordered: use ids as given.
mce_status build_from_csr(uint64_t n, const uint32_t *off_d, const uint32_t *adj_d, const uint32_t *labels_d,
                          int already_ordered, int order_kind, uint32_t degeneracy_hint, uint64_t spin_limit,
                          cudaStream_t st, DeviceGraph *g) {
  *g = DeviceGraph{};
  uint32_t m2 = 0;
  MCE_CUDA_TRY(cudaMemcpyAsync(&m2, off_d + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  MCE_CUDA_TRY(cudaStreamSynchronize(st));
  const uint64_t m = m2 / 2;
  // edges (r < c) from the CSR
  DevBuf<uint32_t> eu, ev, labels0;
  MCE_TRY(labels0.alloc(n, st));
  if (labels_d)
    MCE_CUDA_TRY(cudaMemcpyAsync(labels0.p, labels_d, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  else
    k_iota<<<grid_for(n, 256), 256, 0, st>>>(labels0.p, n); note_launch();
  MCE_TRY(csr_to_edges(n, off_d, adj_d, m, &eu.p, &ev.p, st));
  eu.st = ev.st = st;
  MCE_TRY(finish_graph((uint32_t)n, m, eu.p, ev.p, labels0.p,
                       already_ordered ? MCE_ORDER_UNCHANGED : order_kind, spin_limit, st, g));
  if (already_ordered && degeneracy_hint) g->degeneracy = degeneracy_hint;
  return MCE_OK;
}

namespace {
__global__ void k_upper_flags(const uint32_t *off, const uint32_t *adj, uint64_t n, uint32_t *flag) {
  // one warp per row
  const uint32_t lane = lane_id();
  for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n;
       r += ((uint64_t)gridDim.x * blockDim.x) >> 5)
    for (uint32_t e = off[r] + lane; e < off[r + 1]; e += 32) flag[e] = adj[e] > r ? 1u : 0u;
}
__global__ void k_upper_edges(const uint32_t *off, const uint32_t *adj, uint64_t n, const uint32_t *flag,
                              const uint32_t *pos, uint32_t *eu, uint32_t *ev) {
  const uint32_t lane = lane_id();
  for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n;
       r += ((uint64_t)gridDim.x * blockDim.x) >> 5)
    for (uint32_t e = off[r] + lane; e < off[r + 1]; e += 32)
      if (flag[e]) {
        eu[pos[e]] = (uint32_t)r;
        ev[pos[e]] = adj[e];
      }
}
}  // namespace

mce_status csr_to_edges(uint64_t n, const uint32_t *off, const uint32_t *adj, uint64_t m, uint32_t **eu,
                        uint32_t **ev, cudaStream_t st) {
  DevBuf<uint32_t> flag, pos;
  MCE_TRY(flag.alloc(2 * m + 1, st));
  MCE_TRY(pos.alloc(2 * m + 1, st));
  k_upper_flags<<<grid_for(n * 32, 256), 256, 0, st>>>(off, adj, n, flag.p); note_launch();
  MCE_TRY(scan_exclusive_u32(flag.p, pos.p, 2 * m, pos.p + 2 * m, st));
  uint32_t mu = 0;
  MCE_TRY(read_scalar(pos.p + 2 * m, &mu, st));
  if (mu != m) return MCE_ERR_FORMAT;  // not symmetric / has self-loops
  MCE_CUDA_TRY(cudaMallocAsync(eu, std::max<uint64_t>(m, 1) * sizeof(uint32_t), st));
  MCE_CUDA_TRY(cudaMallocAsync(ev, std::max<uint64_t>(m, 1) * sizeof(uint32_t), st));
  k_upper_edges<<<grid_for(n * 32, 256), 256, 0, st>>>(off, adj, n, flag.p, pos.p, *eu, *ev); note_launch();
  MCE_CUDA_TRY(cudaGetLastError());
  return MCE_OK;
}

void free_graph(DeviceGraph *g) {
  cudaStream_t st = g->stream;
  cudaFreeAsync(g->off, st);
  cudaFreeAsync(g->adj, st);
  cudaFreeAsync(g->labels, st);
  cudaFreeAsync(g->h1, st);
  cudaFreeAsync(g->h2, st);
  cudaFreeAsync(g->root_v0, st);
  cudaFreeAsync(g->root_v1, st);
  cudaFreeAsync(g->root_off, st);
  if (g->slot) cudaFreeAsync(g->slot, st);
  *g = DeviceGraph{};
}

}  // namespace mce
