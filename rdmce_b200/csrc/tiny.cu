// tiny.cu -- vertices with few later neighbours, 32 to a warp.
//
// The first pass of a range solve of a large graph.  A maximal clique belongs
// to its first vertex in the degeneracy order; a vertex with p later
// neighbours has at most 2^p - 1 sets of them to decide, and on a sparse graph
// most vertices have a handful.  A warp's time on one such vertex is dependent
// loads with a few lanes at work (50 to 75 thousand cycles on Chung-Lu 10^6,
// 32 warps an SM), so here a warp takes 32 vertices, one a lane: the pairs of
// later neighbours and the earlier neighbours of all of them are flattened
// over the lanes, and every lane then decides its own vertex on words of
// subsets.  The other vertices are listed for the enumeration kernel (enum.cu),
// which takes the last P.single_items vertices of the order itself.  A root
// range is its vertices' interval (range_vertices).
// Measured (B200): Chung-Lu 10^6 (mean degree 16) enumeration 7.3 -> 6.4 ms.
#include <algorithm>

#include "common.cuh"
#include "engine.h"

namespace mce {

namespace {

// Flattened work of a warp's lanes: lane l has cnt items, and item t of all of
// them is item t - first(l) of its lane.  next() gives this lane's item of the
// current window of 32: its owner lane and number there.
struct Flat {
  uint32_t *owner, *first;  // shared memory, 32 each: the o-th lane with items, its first item
  uint32_t cnt, mine, total, started;
  __device__ __forceinline__ Flat(uint32_t *smem, uint32_t n) : owner(smem), first(smem + 32), cnt(n), started(0) {
    const uint32_t lane = lane_id();
    uint32_t incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, d);
      if (lane >= (uint32_t)d) incl += y;
    }
    mine = incl - n;
    total = __shfl_sync(kFull, incl, 31);
    const uint32_t have = __ballot_sync(kFull, n != 0);
    __syncwarp();
    if (n) {
      const uint32_t o = __popc(have & lanemask_lt());
      owner[o] = lane;
      first[o] = mine;
    }
    __syncwarp();
  }
  __device__ __forceinline__ bool next(uint32_t t0, uint32_t *who, uint32_t *item) {
    const uint32_t lane = lane_id();
    const uint32_t heads = __reduce_or_sync(kFull, cnt && mine - t0 < 32 ? 1u << (mine - t0) : 0u);
    const uint32_t o = started + __popc(heads & (lanemask_lt() | (1u << lane))) - 1;
    started += __popc(heads);
    *who = owner[o];
    *item = t0 + lane - first[o];
    return t0 + lane < total;
  }
};

// A vertex is taken here with 1 to kTinyP later neighbours and up to
// kTinyDegree neighbours (its earlier ones are visited too).
// Measured (B200), ms, up to 5, 6 and 8 later neighbours: Chung-Lu 10^6 7.8,
// 7.5, 6.8, G(10^6, mean degree 6) 0.31, 0.30, 0.30.  Up to 64, 256 or 1024
// neighbours is the same on these; the bound keeps one lane's list from holding
// up the other 31.
constexpr uint32_t kTinyP = 8, kTinyDegree = 256, kTinyWarps = 8;
// An earlier neighbour's list is walked from its end for this many elements,
// then searched for the later neighbours not yet passed.  In a degeneracy order
// few of its neighbours come after v and the walk ends first; in the other
// orders a hub comes early and has nearly its whole list there.
// Measured (B200), enumeration: a hub of 200,000 neighbours with 1 and 7 later
// neighbours each (stored order) 60 and 237 ms walked to the end, 1.05 and 1.51
// here, 1.15 and 1.93 with 256 elements; searching from the first element on,
// G(10^6, mean degree 6) takes 0.33 ms instead of 0.30.
constexpr uint32_t kTinyWalk = 16;

// A set of later neighbours is a lane number (the first five) and a group (the
// others); the sets of one group are one 32-bit word.
struct TinyWarp {
  uint32_t dead[8][32];  // sets that earlier neighbours rule out, by group and lane
  uint32_t adj[32];      // bit j (j - 1) / 2 + i: later neighbours i < j are adjacent
  uint32_t flat[64];
};

// Decides this lane's vertex v, if p > 0: its list starts at b, x earlier
// neighbours first.  Adds the cliques' hashes to *chk and returns their
// numbers by size, byte k for size k + 2 (fewer than 256 a vertex).
__device__ uint64_t tiny_vertex(const DevGraph &g, TinyWarp *ts, uint32_t v, uint32_t b, uint32_t x, uint32_t p,
                                uint64_t *chk_out) {
  const uint32_t lane = lane_id();
  uint32_t *flat = ts->flat;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; k++) ts->dead[k][lane] = 0;
  ts->adj[lane] = 0;
  __syncwarp();
  const uint32_t first = b + x;  // later neighbours at adj[first .. first + p)
  {
    Flat f(flat, p * (p - (p != 0)) / 2);
    for (uint32_t t0 = 0; t0 < f.total; t0 += 32) {
      uint32_t o, t;
      const bool in = f.next(t0, &o, &t);
      const uint32_t base = __shfl_sync(kFull, first, o);
      if (in) {
        const uint32_t j = (uint32_t)((1.0f + sqrtf((float)(8 * t + 1))) * 0.5f), i = t - j * (j - 1) / 2;
        const uint32_t pi = __ldg(g.adj + base + i), pj = __ldg(g.adj + base + j);
        const uint32_t bi = g.off[pi], ni = g.off[pi + 1] - bi, bj = g.off[pj], nj = g.off[pj + 1] - bj;
        // in the shorter of the two lists
        if (ni <= nj ? contains_u32(g.adj + bi, ni, pj) : contains_u32(g.adj + bj, nj, pi))
          atomicOr(&ts->adj[o], 1u << t);
      }
    }
  }
  {
    Flat f(flat, p ? x : 0);
    for (uint32_t t0 = 0; t0 < f.total; t0 += 32) {
      uint32_t o, t;
      const bool in = f.next(t0, &o, &t);
      const uint32_t base = __shfl_sync(kFull, first, o), list = __shfl_sync(kFull, b, o),
                     n = __shfl_sync(kFull, p, o);
      if (in) {
        const uint32_t u = __ldg(g.adj + list + t);
        const uint32_t ub = g.off[u], ue = g.off[u + 1];
        // its list from the end, against the later neighbours from the last
        uint32_t m = 0, e = ue, k = n, c = __ldg(g.adj + base + n - 1);
        const uint32_t least = __ldg(g.adj + base);
        while (e > ub && k) {
          if (ue - e == kTinyWalk) {  // many neighbours after v: search them for the others
            for (uint32_t i = 0; i < k; i++)
              if (contains_u32(g.adj + ub, e - ub, __ldg(g.adj + base + i))) m |= 1u << i;
            break;
          }
          const uint32_t y = __ldg(g.adj + e - 1);
          if (y < least) break;
          while (k && c > y) {
            k--;
            if (k) c = __ldg(g.adj + base + k - 1);
          }
          if (k && c == y) m |= 1u << (k - 1);
          e--;
        }
        if (m) {
          uint32_t sub = 1;
#pragma unroll
          for (int i = 0; i < 5; i++)
            if ((m >> i) & 1) sub |= sub << (1 << i);
          const uint32_t mh = m >> 5;
          uint32_t gr = 0;
          do {  // the groups inside its high part
            atomicOr(&ts->dead[gr][o], sub);
            gr = (gr - mh) & mh;
          } while (gr);
        }
      }
    }
  }
  __syncwarp();
  // every lane decides its vertex
  constexpr uint32_t kWith[5] = {0xAAAAAAAAu, 0xCCCCCCCCu, 0xF0F0F0F0u, 0xFF00FF00u, 0xFFFF0000u};
  const uint32_t pairs = ts->adj[lane];
  uint32_t row[kTinyP], dead_in[kTinyP];
#pragma unroll
  for (int i = 0; i < (int)kTinyP; i++) {
    row[i] = 0;
#pragma unroll
    for (int j = 0; j < (int)kTinyP; j++) {
      if (j == i) continue;
      const int lo = j < i ? j : i, hi = j < i ? i : j;
      if ((pairs >> (hi * (hi - 1) / 2 + lo)) & 1) row[i] |= 1u << j;
    }
    uint32_t sub = 1;
#pragma unroll
    for (int k = 0; k < 5; k++)
      if ((row[i] >> k) & 1) sub |= sub << (1 << k);
    dead_in[i] = i < 5 ? sub | (kWith[i < 5 ? i : 0] & ~(sub << (1 << (i < 5 ? i : 0)))) : sub;
    row[i] >>= 5;  // the group part
  }
  const uint64_t s10 = p ? g.h1[v] : 0, s20 = p ? g.h2[v] : 0;
  uint64_t h1[5], h2[5];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const bool have = (uint32_t)i < p;
    const uint32_t w = have ? __ldg(g.adj + first + i) : 0;
    h1[i] = have ? g.h1[w] : 0;
    h2[i] = have ? g.h2[w] : 0;
  }
  const uint32_t high = p > 5 ? (1u << (p - 5)) - 1 : 0;
  const uint32_t all = p >= 5 ? 0xffffffffu : p ? (1u << (1u << p)) - 1 : 0u;
  uint64_t chk = 0, sizes = 0;  // byte k: cliques of size k + 2 (fewer than 256 a vertex)
#pragma unroll 1
  for (uint32_t gr = 0; __any_sync(kFull, gr <= high); gr++) {
    uint32_t dead = ts->dead[gr & 7][lane];
#pragma unroll
    for (int i = 0; i < (int)kTinyP; i++) {
      if ((uint32_t)i >= p) continue;
      if (i < 5) {
        dead |= (gr & ~row[i]) ? kWith[i < 5 ? i : 0] : dead_in[i];
      } else {
        const uint32_t own = 1u << (i < 5 ? 0 : i - 5);
        const uint32_t w = (gr & ~own & ~row[i]) ? 0u : dead_in[i];
        dead |= (gr & own) ? ~w : w;
      }
    }
    uint32_t E = p && gr <= high ? all & ~dead : 0u;
    if (!__any_sync(kFull, E != 0)) continue;
    uint64_t g1 = s10, g2 = s20;
    uint32_t rest = E ? gr : 0;
    while (rest) {
      const uint32_t w = __ldg(g.adj + first + 5 + (__ffs(rest) - 1));
      rest &= rest - 1;
      g1 += g.h1[w];
      g2 += g.h2[w];
    }
    while (E) {
      const uint32_t sset = __ffs(E) - 1;
      E &= E - 1;
      uint64_t a = g1, bsum = g2;
#pragma unroll
      for (int i = 0; i < 5; i++)
        if ((sset >> i) & 1) {
          a += h1[i];
          bsum += h2[i];
        }
      const uint32_t members = __popc(sset) + __popc(gr);
      chk += clique_hash(a, bsum, members + 1);
      sizes += 1ull << (8 * (members - 1));
    }
  }
  *chk_out += chk;
  return sizes;
}

__global__ void __launch_bounds__(32 * kTinyWarps) k_tiny(const __grid_constant__ EnumParams P) {
  __shared__ TinyWarp s_warp[kTinyWarps];
  __shared__ uint32_t s_hist[kTinyP];
  const DevGraph &g = P.g;
  const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
  if (threadIdx.x < kTinyP) s_hist[threadIdx.x] = 0;
  __syncthreads();
  uint64_t chk = 0;
  unsigned long long roots = 0;
  const uint32_t nwarps = gridDim.x * kTinyWarps;
  const uint32_t last = range_last(P), items = range_vertices(P);
  for (uint64_t k = range_singles(P) + (uint64_t)(blockIdx.x * kTinyWarps + wid) * 32; k < items; k += (uint64_t)nwarps * 32) {
    uint32_t v = 0, b = 0, d = 0, p = 0;
    bool left = false, tiny = false;
    if (k + lane < items) {
      v = last - (uint32_t)(k + lane);
      const uint32_t r0 = g.root_off[v], r1 = g.root_off[v + 1];
      b = g.off[v];
      d = g.off[v + 1] - b;
      p = r1 - r0;
      left = p && r1 > P.rb && r0 < P.re;  // some of its roots are in the range
      tiny = left && p <= kTinyP && d <= kTinyDegree && r0 >= P.rb && r1 <= P.re;
      left = left && !tiny;
    }
    const uint32_t lb = __ballot_sync(kFull, left);
    if (lb) {
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(P.vert_n, (uint32_t)__popc(lb));
      at = __shfl_sync(kFull, at, 0);
      if (left) P.vert_list[at + __popc(lb & lanemask_lt())] = v;
    }
    if (!__any_sync(kFull, tiny)) continue;
    if (tiny) roots += p;
    uint64_t one = 0;
    const uint64_t sizes = tiny_vertex(g, &s_warp[wid], v, b, d - p, tiny ? p : 0, &one);
    if (g.slot) {  // many graphs: each lane's results go to its own
      if (sizes) {
        const uint32_t slot = g.slot[v];
        uint32_t count = 0, largest = 0;
        for (uint32_t i = 0; i < kTinyP; i++) {
          const uint32_t n = (uint32_t)(sizes >> (8 * i)) & 0xff;
          if (!n) continue;
          count += n;
          largest = i + 2;
          const uint32_t bin = i + 2 < P.hist_len ? i + 2 : P.hist_len - 1;
          atomicAdd(&P.hist[(uint64_t)slot * P.hist_len + bin], (unsigned long long)n);
        }
        atomicAdd(&P.slots[slot].count, (unsigned long long)count);
        atomicAdd(&P.slots[slot].checksum, (unsigned long long)one);
        atomicMax(&P.slots[slot].max_size, largest);
      }
    } else {
      chk += one;
      for (uint32_t i = 0; i < kTinyP; i++) {
        const uint32_t n = __reduce_add_sync(kFull, (uint32_t)(sizes >> (8 * i)) & 0xff);
        if (lane == 0 && n) atomicAdd(&s_hist[i], n);
      }
    }
  }
  chk = warp_sum_u64(chk);
  roots = warp_sum_u64(roots);
  if (lane == 0) {
    if (chk) atomicAdd(&P.slots[0].checksum, (unsigned long long)chk);
    if (roots) atomicAdd(P.stat_roots, roots);
  }
  __syncthreads();
  if (threadIdx.x < kTinyP && s_hist[threadIdx.x]) {
    const uint32_t n = s_hist[threadIdx.x], size = threadIdx.x + 2;
    const uint32_t bin = size < P.hist_len ? size : P.hist_len - 1;
    atomicAdd(&P.hist[bin], (unsigned long long)n);
    atomicAdd(&P.slots[0].count, (unsigned long long)n);
    atomicMax(&P.slots[0].max_size, size);
  }
}

}  // namespace

mce_status launch_tiny(const EnumParams &P, uint32_t sms, cudaStream_t st) {
  const uint64_t blocks = (P.g.n - P.single_items + 32ULL * kTinyWarps - 1) / (32ULL * kTinyWarps);
  k_tiny<<<(uint32_t)std::min<uint64_t>(blocks, sms * 8ULL), 32 * kTinyWarps, 0, st>>>(P);
  note_launch();
  MCE_CUDA_TRY(cudaGetLastError());
  return MCE_OK;
}

}  // namespace mce
