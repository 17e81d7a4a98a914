// enum.cu -- edge-rooted bitmap Bron-Kerbosch with pivot on the GPU.
//
// Method (the reference's, src/kernels/BkPivotBitBalance.cuh):
//   root = undirected edge (v0 < v1) in the degeneracy order (:428-469);
//   C = N(v0) & N(v1); P = {c in C : c > v1}, X = {c in C : c < v1};
//   an edge in no triangle is a maximal clique of size 2 (:535-539);
//   ego bitmap: row r = P[r] for r < p, then the X members; bit j = adjacency
//   to P[j]; X rows without a P neighbour are dropped (include/graph_gpu.cuh:59-107);
//   node: pivot = argmin over rows containing R of |P \ row| (:229-257),
//   branch on VP = P \ row(pivot) in ascending order; child P' = P & row(q);
//   EXPAND_R moves every i in P' with |P' \ row(i)| == 1 into R (:368-382);
//   leaf: P empty and no row contains R -> one maximal clique (:276-294);
//   root-down exposure: the shallowest level with open candidates is handed
//   to other warps when they run dry (:87-138, :552-598).
//
// B200 design:
//   * Three tiers by subproblem size.  Nearly every search-tree node has at
//     most 32 candidate columns and 32 rows that contain R: there each lane
//     holds one row as a 32-bit word, P / VP / the active-row set are
//     warp-uniform 32-bit masks, and a node is one redux.sync (pivot argmin),
//     two ballots (EXPAND_R, the child's active rows) and a few shuffles.  Up to 64
//     columns and 128 rows, each lane holds 4 rows as 64-bit words.  Larger
//     subproblems run in the general tier (W 64-bit words per row in a global
//     scratch slab, per-level lists of active rows).  A child small enough for
//     a smaller tier has its rows compressed to its own columns (parallel bit
//     compress) and gathered, and continues there.
//   * In the 32-bit tier R is a column mask and leaves are hashed 32 at a
//     time, one per lane.  A node or child with few candidates is decided in
//     one step: its maximal cliques are the cliques K of the candidates that
//     no active row contains, found on words of subsets.  To expose work the
//     node loop steps out and is resumed.
//   * A range of roots is taken vertex by vertex first: one ego network and one
//     pivot for all roots of a vertex (run_vertex); small vertices of large
//     graphs are decided 32 to a warp before that (tiny.cu).
//   * Root-down exposure with self-contained tasks.  When warps are idle, a
//     busy warp turns every open candidate of the shallowest open level with
//     |P| >= tau -- outer tiers of a nested solve first -- into a task record
//     (rows restricted to the child's columns, X rows empty on them left out)
//     in a global pool, published through lock-free bounded MPMC rings.  A
//     task owns its data, so no warp ever waits on another warp's stack (the
//     reference's owner waits for its thieves, :87-138).  Every wait is bounded.
//   * Pivot ties go to the lowest row index; every leaf feeds the clique-size
//     histogram and the order-independent checksum.
//   * Roots whose ego network exceeds the per-warp slab are deferred to a
//     second pass with large slabs, never skipped (the reference prints and
//     skips them, :480-487).
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "engine.h"

// This file is compiled once per register budget of the enumeration kernel:
// MCE_ENUM_BPS resident 8-warp blocks per SM (3, 4 or 5: at most 85, 64 or 51
// registers a thread).  Each build keeps its own copies of the device
// functions, so one budget never forces spills on another; enum_dispatch.cu
// picks the build per solve (the autotuner's occupancy choice).
#ifndef MCE_ENUM_BPS
#define MCE_ENUM_BPS 4
#endif
#define MCE_CAT2(a, b) a##b
#define MCE_CAT(a, b) MCE_CAT2(a, b)
#define MCE_ENUM_FN(name) MCE_CAT(name, MCE_CAT(_b, MCE_ENUM_BPS))

namespace mce {

namespace {

constexpr uint32_t kIdent = 0xffffffffu;  // level-0 list = all rows
constexpr uint32_t kHistCache = 128;      // per-warp shared-memory histogram bins
constexpr int kRPL = 4;                   // 64-bit tier: rows per lane
constexpr uint32_t kT1Rows = 32 * kRPL;   // 64-bit tier: rows per subproblem
constexpr uint32_t kT1Depth = 66;         // 64-bit tier: levels (<= 64 columns + root)
constexpr uint32_t kT0Depth = 34;         // 32-bit tier: levels (<= 32 columns + root)
constexpr uint32_t kHdr = 64;             // task record header bytes
constexpr uint32_t kLocalRec = 2048;      // per-warp local task record (64-bit-tier size)
// Default tau inside the register tiers (64 or fewer candidates): the same 24
// as the general tier measured as fast as smaller values on R-MAT inputs,
// with fewer, larger tasks, once nested tiers expose their outer levels first.
constexpr uint32_t kRegShareBound = 24;
constexpr uint32_t kShareMin = 128, kShareMax = 8192;
// A graph with more vertices than this for each warp has the others' small
// vertices decided up front, 32 to a warp (tiny.cu); the late-peeled ones, up
// to this many, are items in order either way.
// Measured (B200), ms, for 1, 8, 32: Chung-Lu 10^6 6.89, 6.77, 6.73, R-MAT 18 of
// edge factor 4 11.03, 10.88, 11.10, G(10^6, mean degree 6) 0.23, 0.30, 0.59.
constexpr uint32_t kVertexSingles = 8;
// 32-bit-tier nodes with up to this many candidates are decided in one step,
// at 2^(n - 5) groups of about 12 instructions each (t0_small_sets).
#ifndef MCE_SMALL_P
#define MCE_SMALL_P 9
#endif
constexpr int kSmallP = MCE_SMALL_P;
static_assert(kSmallP >= 6 && kSmallP <= 12, "t0_batch has an array of the kSmallP - 5 group candidates; groups double with each");
// phases of the per-warp cycle accounting
// (kCycReg: the 64-bit tier; kCycT0: the 32-bit tier)
enum { kCycBuild = 0, kCycReg = 1, kCycGen = 2, kCycSpawn = 3, kCycIdle = 4, kCycQueue = 5, kCycT0 = 6, kCycPhases = 7 };

struct TaskHdr {
  uint32_t pc;     // candidate columns
  uint32_t nrows;  // rows: pc candidate rows, then the X rows
  uint32_t W;      // 64-bit words per row
  uint32_t rsize;  // |R| beyond the root edge
  uint64_t s1, s2; // label-hash sums of the clique so far (root edge included)
  uint32_t slot;   // result slot
  uint32_t pad0;
  uint64_t pad[3];
};
static_assert(sizeof(TaskHdr) == kHdr, "task header is 64 bytes");

__host__ __device__ __forceinline__ uint64_t align8(uint64_t x) { return (x + 7) & ~7ULL; }

__host__ __device__ __forceinline__ uint64_t task_bytes(uint32_t pc, uint32_t nrows, uint32_t W) {
  return kHdr + align8(4ULL * pc) + 8ULL * nrows * W;
}

// A compression plan (compress_plan): the selected bits and the six move masks.
struct CPlan {
  uint64_t m;
  uint64_t mv[6];
};
static_assert(sizeof(CPlan) == 56, "layout_for reserves this much a word");

// A general-tier subproblem laid out in the warp's slab.
struct Gen {
  const uint64_t *rows;
  const uint32_t *colv;
  const uint64_t *h1s, *h2s;
  uint64_t *stack;
  CPlan *plans;  // W of them, for the task being written
  uint32_t *alist;
  uint64_t alist_cap;
  uint32_t pc, nrows, W;
};

// Per-warp shared memory.  All mutable per-warp state outside the tier loops
// lives here (lane 0 updates the scalars), so the small Ctx handle can be
// passed by value.
struct WarpSmem {
  uint64_t rowbuf[64];
  // 32-bit tier frames: (P, VP, active rows, R as a column mask)
  uint4 t0f[kT0Depth];
  // exchange buffer for moving a subproblem into the 32-bit tier; xh1/xh2
  // hold the label hashes of the running 32-bit-tier subproblem's columns
  uint32_t xrow[32], xcv[32];
  uint64_t xh1[32], xh2[32];
  // the running 32-bit-tier subproblem's hash sums and |R| at entry, and the
  // R masks of leaves not yet hashed
  uint64_t t0_s1, t0_s2;
  uint32_t t0_rsize;
  uint32_t pend_rm[32];
  // collected small nodes (t0_batch): candidate k's row of node i at
  // [33 k + i] (a row stride of 33 keeps one node's rows in different banks),
  // the candidates and R
  uint32_t pr_row[33 * kSmallP];
  uint32_t pr_P[32], pr_RM[32];
  uint64_t lchk[32];  // per-lane checksum accumulators (batched leaves)
  // a 32-bit-tier solve that stepped out to expose work: its node state
  uint32_t y_P, y_A, y_RM, y_npend, y_nprob;
  int y_level;
  // nodes between the 32-bit tier's checks for idle warps; doubles (up to
  // kShareMax) while checks find nothing to expose, back to kShareMin after
  // one does
  uint32_t share_period;
  uint32_t hcache[kHistCache];
  // result accumulators for the current slot
  unsigned long long count, checksum, nodes, wops, bbytes;
  uint32_t max_size, slot, pending;
  uint32_t last, singles;  // vertex pass: range_last, range_singles
  unsigned long long cyc[kCycPhases];  // clock64 cycles by phase
  // The tiers enclosing the running subproblem.  A nested tier exposes their
  // open levels (shallower, so larger) before its own: the running
  // general-tier solve, and the level each enclosing tier is expanding (the
  // 64-bit tier's rows are in its T1Area).
  Gen gen;
  int t1_level, gen_level;
  uint32_t t1_pc;
  uint32_t nest;  // bit 0: a general-tier solve is running; bit 1: a 64-bit-tier solve
};

constexpr uint32_t kNestGen = 1, kNestT1 = 2;

// The 64-bit tier's frames and rows live at the tail of the warp's slab, not
// in shared memory: that tier holds few of the nodes, and shared memory kept
// small lets 4 blocks of 8 warps share an SM.
struct T1Area {
  uint64_t fP[kT1Depth], fVP[kT1Depth], fs1[kT1Depth], fs2[kT1Depth];
  uint32_t frs[kT1Depth];
  uint8_t fab[kT1Depth][32];
  uint64_t t1rows[kT1Rows];
  uint32_t t1cv[64];
};
constexpr uint32_t kT1Area = (sizeof(T1Area) + 255) & ~255u;
constexpr uint32_t kTail = kLocalRec + kT1Area;  // slab bytes reserved at its end

// Slab layout of a general-tier problem (bytes from the slab start).
struct Layout {
  uint64_t colv_off, hash_off, rows_off, stack_off, plan_off, alist_off, need;
};

__host__ __device__ __forceinline__ Layout layout_for(uint64_t cand_n, uint32_t pc, uint32_t nrows, uint32_t W) {
  Layout L;
  L.colv_off = 0;
  L.hash_off = align8(4ULL * cand_n);
  L.rows_off = L.hash_off + 16ULL * pc;
  L.stack_off = L.rows_off + 8ULL * (uint64_t)nrows * W;
  // pc + 1 levels, one scratch record past the deepest, one spare
  L.plan_off = L.stack_off + 8ULL * (uint64_t)(pc + 3) * (3ULL * W + 4);
  L.alist_off = L.plan_off + 56ULL * W;  // one compression plan a word (CPlan)
  L.need = L.alist_off + 4ULL * nrows + kTail;
  return L;
}

struct Ctx {
  const EnumParams *P;
  WarpSmem *sm;
  T1Area *ta;
  char *slab;
  uint64_t slab_bytes;
  uint32_t lane;
  bool sharing;
};

__device__ __forceinline__ unsigned long long now() { return clock64(); }

// Task records travel between SMs through reused pool blocks; read them from
// L2 (ld.global.cg) so no SM sees a stale L1 line of an earlier task.
__device__ __forceinline__ uint64_t ld_cg(const uint64_t *p) { return __ldcg((const unsigned long long *)p); }
__device__ __forceinline__ uint32_t ld_cg(const uint32_t *p) { return __ldcg((const unsigned int *)p); }

// ------------------------------------------------------------ accounting

__device__ __forceinline__ void acc_flush(const Ctx &c) {
  const EnumParams &P = *c.P;
  WarpSmem *sm = c.sm;
  __syncwarp();
  const uint64_t lc = warp_sum_u64(sm->lchk[c.lane]);
  sm->lchk[c.lane] = 0;
  if (c.lane == 0) sm->checksum += lc;
  __syncwarp();
  for (uint32_t b = c.lane; b < kHistCache; b += 32) {
    const uint32_t n = sm->hcache[b];
    if (n) {
      const uint32_t bin = b < P.hist_len ? b : P.hist_len - 1;
      atomicAdd(&P.hist[(uint64_t)sm->slot * P.hist_len + bin], (unsigned long long)n);
      sm->hcache[b] = 0;
    }
  }
  if (c.lane == 0) {
    if (sm->count || sm->max_size) {
      atomicAdd(&P.slots[sm->slot].count, sm->count);
      atomicAdd(&P.slots[sm->slot].checksum, sm->checksum);
      atomicMax(&P.slots[sm->slot].max_size, sm->max_size);
    }
    sm->count = 0;
    sm->checksum = 0;
    sm->max_size = 0;
    sm->pending = 0;
  }
  __syncwarp();
}

__device__ __forceinline__ void set_slot(const Ctx &c, uint32_t slot) {
  if (c.sm->slot != slot) {
    acc_flush(c);
    if (c.lane == 0) c.sm->slot = slot;
    __syncwarp();
  }
}

// lane 0 only
__device__ __forceinline__ void emit(const Ctx &c, uint32_t size, uint64_t s1, uint64_t s2) {
  WarpSmem *sm = c.sm;
  sm->count++;
  sm->checksum += clique_hash(s1, s2, size);
  sm->max_size = max(sm->max_size, size);
  if (size < kHistCache) {
    sm->hcache[size]++;
    sm->pending++;
  } else {
    const EnumParams &P = *c.P;
    const uint32_t bin = size < P.hist_len ? size : P.hist_len - 1;
    atomicAdd(&P.hist[(uint64_t)sm->slot * P.hist_len + bin], 1ULL);
  }
}

__device__ __forceinline__ void maybe_flush(const Ctx &c) {
  // keeps every u32 histogram bin far from overflow
  if (c.sm->pending > (1u << 30)) acc_flush(c);
}

// ------------------------------------------------------- bounded MPMC rings
// Vyukov's bounded queue: cell seq == pos means free for the producer of pos,
// seq == pos + 1 means filled for the consumer of pos.  Lane 0 only.
//
// A consumer first takes one of the ring's filled cells off its count, then
// draws its position with an unconditional add.  Advancing the head by
// compare-and-swap instead lets one consumer through in each round trip to L2
// while all others retry: with hundreds of idle warps polling, that capped the
// task rate at 1.3-2.8 tasks a microsecond however many warps were idle.
// Measured (B200): 1024 core roots of R-MAT 20 43.7 -> 27.7 ms, full R-MAT 14
// 31.9 -> 20.9 ms.

__device__ bool ring_push(uint32_t *slots, unsigned long long *seq, unsigned long long *tail, int *count,
                          uint32_t mask, uint32_t val, const EnumParams &P) {
  const unsigned long long pos = atomicAdd(tail, 1ULL);
  volatile unsigned long long *s = seq + (pos & mask);
  uint64_t n = 0;
  while (*s != pos) {
    if (++n > P.spin_limit) {
      atomicExch(P.error, 3u);
      return false;
    }
    __nanosleep(64);
  }
  ((volatile uint32_t *)slots)[pos & mask] = val;
  __threadfence();
  *s = pos + 1;
  __threadfence();
  atomicAdd(count, 1);
  return true;
}

__device__ bool ring_pop(uint32_t *slots, unsigned long long *seq, unsigned long long *head, int *count,
                         uint32_t mask, uint32_t *val, const EnumParams &P) {
  if (*(volatile int *)count <= 0) return false;
  if (atomicSub(count, 1) <= 0) {  // others were quicker
    atomicAdd(count, 1);
    return false;
  }
  const unsigned long long h = atomicAdd(head, 1ULL);
  volatile unsigned long long *s = seq + (h & mask);
  uint64_t n = 0;
  // a cell counted as filled may lie behind one whose producer is still writing
  while (*s != h + 1) {
    if (++n > P.spin_limit) {
      atomicExch(P.error, 3u);
      return false;
    }
    __nanosleep(32);
  }
  __threadfence();
  *val = ((volatile uint32_t *)slots)[h & mask];
  __threadfence();
  *s = h + (unsigned long long)mask + 1;
  return true;
}

// warp-uniform wrappers
__device__ __forceinline__ bool pool_alloc(const Ctx &c, uint32_t *blk) {
  const EnumParams &P = *c.P;
  uint32_t b = 0;
  bool ok = false;
  if (c.lane == 0) ok = ring_pop(P.free_slot, P.free_seq, P.free_head, P.free_count, P.pool_mask, &b, P);
  ok = __shfl_sync(kFull, ok, 0);
  *blk = __shfl_sync(kFull, b, 0);
  return ok;
}

__device__ __forceinline__ void pool_free(const Ctx &c, uint32_t blk) {
  const EnumParams &P = *c.P;
  __syncwarp();
  if (c.lane == 0) ring_push(P.free_slot, P.free_seq, P.free_tail, P.free_count, P.pool_mask, blk, P);
  __syncwarp();
}

// A task counts as busy from before it is published until its taker has
// finished it (see idle_wait).
__device__ __forceinline__ void pool_publish(const Ctx &c, uint32_t blk) {
  const EnumParams &P = *c.P;
  __threadfence();
  __syncwarp();
  if (c.lane == 0) {
    __threadfence();
    atomicAdd(P.active, 1u);  // ordered before the task by ring_push's fence
    if (!ring_push(P.ready_slot, P.ready_seq, P.ready_tail, P.ready_count, P.pool_mask, blk, P)) atomicSub(P.active, 1u);
    atomicAdd(P.stat_tasks, 1ULL);
  }
  __syncwarp();
}

__device__ __forceinline__ char *pool_block(const EnumParams &P, uint32_t blk) {
  return P.pool + (uint64_t)blk * P.block_bytes;
}

// busy warps expose work while fewer tasks are queued than warps are idle
__device__ __forceinline__ bool hungry(const Ctx &c) {
  const EnumParams &P = *c.P;
  uint32_t h = 0;
  if (c.lane == 0) h = *(volatile unsigned int *)P.active < P.nwarps;
  return __shfl_sync(kFull, h, 0) != 0;
}

// ------------------------------------------------------- bit compression
// compress(x, m): the bits of x at the set positions of m, packed to the low
// end (Hacker's Delight 2nd ed. section 7-4, parallel-suffix form).  The plan
// depends only on m, which is warp-uniform wherever it is used.

__device__ __forceinline__ CPlan compress_plan(uint64_t m) {
  CPlan p;
  p.m = m;
  uint64_t mk = ~m << 1;
#pragma unroll
  for (int i = 0; i < 6; i++) {
    uint64_t mp = mk ^ (mk << 1);
    mp ^= mp << 2;
    mp ^= mp << 4;
    mp ^= mp << 8;
    mp ^= mp << 16;
    mp ^= mp << 32;
    const uint64_t mv = mp & m;
    p.mv[i] = mv;
    m = (m ^ mv) | (mv >> (1 << i));
    mk = mk & ~mp;
  }
  return p;
}

__device__ __forceinline__ uint64_t compress_apply(uint64_t x, const CPlan &p) {
  x &= p.m;
#pragma unroll
  for (int i = 0; i < 6; i++) {
    const uint64_t t = x & p.mv[i];
    x = (x ^ t) | (t >> (1 << i));
  }
  return x;
}

// multi-word row compaction: out[0..W') = bits of row[0..W) at the masks of plans[0..W)
__device__ __forceinline__ void compress_row(const uint64_t *row, const CPlan *plans, uint32_t W, uint64_t *out) {
  uint64_t cur = 0;
  uint32_t cb = 0, wi = 0;
  for (uint32_t w = 0; w < W; w++) {
    const uint32_t n = __popcll(plans[w].m);
    if (n == 0) continue;
    const uint64_t c = compress_apply(row[w], plans[w]);
    cur |= c << cb;
    if (cb + n >= 64) {
      out[wi++] = cur;
      cur = cb ? (c >> (64 - cb)) : 0;
      cb = cb + n - 64;
    } else {
      cb += n;
    }
  }
  if (cb) out[wi] = cur;
}

// Expose open levels of the enclosing general-tier / 64-bit-tier solve, if one
// is running; true if anything was exposed.  Defined after those tiers.
__device__ __noinline__ bool spawn_outer_gen(Ctx c);
__device__ __noinline__ bool spawn_outer_t1(Ctx c);
// Exposure for a 32-bit-tier solve that stepped out: enclosing tiers first,
// then its own levels.
struct T0;
__device__ __noinline__ bool t0_share(Ctx c, const T0 t, int level);

// ---------------------------------------------------------- 32-bit tier
// At most 32 candidate columns and 32 rows: lane l holds row l as a 32-bit
// word (rows 0..pc-1 are the column vertices, the rest X rows).  P, VP, the
// active-row set and R -- the columns added since the subproblem began -- are
// warp-uniform masks, so a child costs a few bitwise ops and two ballots.
// Label-hash sums are not carried down the tree: a leaf records its R mask,
// and every 32 leaves the lanes hash one clique each (t0_flush).

struct T0 {
  uint32_t row;
  uint32_t cv;      // vertex id of column lane
  uint64_t h1, h2;  // label hashes of column lane
};

// One clique per live lane: its hash, histogram bin and size.
__device__ __forceinline__ void leaves_out(const EnumParams *Pm, WarpSmem *sm, bool live, uint64_t a, uint64_t b,
                                           uint32_t size) {
  const uint32_t lane = lane_id();
  if (live) {
    sm->lchk[lane] += clique_hash(a, b, size);
    if (size < kHistCache) {
      atomicAdd(&sm->hcache[size], 1u);
    } else {
      const uint32_t bin = size < Pm->hist_len ? size : Pm->hist_len - 1;
      atomicAdd(&Pm->hist[(uint64_t)sm->slot * Pm->hist_len + bin], 1ULL);
    }
  }
  const uint32_t n = __popc(__ballot_sync(kFull, live));
  const uint32_t mx = __reduce_max_sync(kFull, live ? size : 0u);
  if (lane == 0) {
    sm->count += n;
    sm->pending += n;
    sm->max_size = max(sm->max_size, mx);
  }
  __syncwarp();
}

// Hash one leaf per live lane (R = rm): sums of the entry sums and the R
// columns' hashes, then as above.
// Out of line: it runs once per 32 leaves, and one copy keeps the hot node
// loop's code small (instruction-cache misses, not issue slots, bound it).
__device__ __noinline__ void t0_hash(const EnumParams *Pm, WarpSmem *sm, uint32_t rm, bool live) {
  const uint32_t size = sm->t0_rsize + 2 + __popc(rm);
  uint64_t a = sm->t0_s1, b = sm->t0_s2;
  while (rm) {
    const uint32_t i = __ffs(rm) - 1;
    rm &= rm - 1;
    a += sm->xh1[i];
    b += sm->xh2[i];
  }
  leaves_out(Pm, sm, live, a, b, size);
}

// hash the pending leaves
__device__ __forceinline__ void t0_flush(const Ctx &c, uint32_t npend) {
  __syncwarp();
  const bool live = c.lane < npend;
  t0_hash(c.P, c.sm, live ? c.sm->pend_rm[c.lane] : 0u, live);
}

// hash sums of a frame's R mask (lanes of R contribute their column hash)
__device__ __forceinline__ void t0_sums(const Ctx &c, uint32_t rm, uint64_t *s1, uint64_t *s2) {
  const bool in = (rm >> c.lane) & 1;
  *s1 = c.sm->t0_s1 + warp_sum_u64(in ? c.sm->xh1[c.lane] : 0);
  *s2 = c.sm->t0_s2 + warp_sum_u64(in ? c.sm->xh2[c.lane] : 0);
}

// Child task of candidate q at a 32-bit-tier level, as a W = 1 record.
__device__ void t0_materialize(const Ctx &c, const T0 &t, uint32_t Pbase, uint32_t A, uint32_t q, uint32_t RM,
                               char *rec) {
  const uint32_t lane = c.lane;
  const uint32_t CP = Pbase & __shfl_sync(kFull, t.row, q);
  const uint32_t pc = __popc(CP);
  const CPlan plan = compress_plan(CP);
  uint64_t s1, s2;
  t0_sums(c, RM | (1u << q), &s1, &s2);
  uint32_t *colv = (uint32_t *)(rec + kHdr);
  uint64_t *rows = (uint64_t *)(rec + kHdr + align8(4ULL * pc));
  const uint64_t cr = compress_apply(t.row, plan);
  if ((CP >> lane) & 1) {
    const uint32_t k = __popc(CP & ((1u << lane) - 1));
    colv[k] = t.cv;
    rows[k] = cr;
  }
  const bool isx = ((A >> lane) & 1) && ((t.row >> q) & 1) && !((CP >> lane) & 1) &&
                   (CP == 0 || (t.row & CP) != 0);  // X rows empty on the child's columns left out
  const uint32_t bal = __ballot_sync(kFull, isx);
  if (isx) rows[pc + __popc(bal & lanemask_lt())] = cr;
  if (lane == 0) {
    TaskHdr *h = (TaskHdr *)rec;
    h->pc = pc;
    h->nrows = pc + __popc(bal);
    h->W = 1;
    h->rsize = c.sm->t0_rsize + __popc(RM) + 1;
    h->s1 = s1;
    h->s2 = s2;
    h->slot = c.sm->slot;
  }
  __syncwarp();
}

// expose every open candidate of the shallowest open level with |P| >= tau
// (the reference's TASK_SHARE_BOUND, BkPivotBitBalance.cuh:271-273)
__device__ bool t0_spawn(const Ctx &c, const T0 &t, int level) {
  WarpSmem *sm = c.sm;
  int l = 0;
  uint32_t open = 0;
  for (; l < level; l++) {
    const uint4 f = sm->t0f[l];
    open = f.x & f.y;
    if (open && (uint32_t)__popc(f.x) + 1 >= c.P->reg_share_bound) break;
    open = 0;
  }
  if (!open) return false;
  const uint4 f = sm->t0f[l];
  uint32_t VPl = f.y;
  // Highest candidate first: the child of q excludes every open candidate
  // below q, all still open at that point; whatever stays with this warp is
  // the lowest candidates, whose children correctly keep the exposed (later)
  // ones in P.
  while (open) {
    const uint32_t q = 31 - __clz(open);
    open &= ~(1u << q);
    uint32_t blk;
    if (!pool_alloc(c, &blk)) break;
    const uint32_t Pbase = f.x & ~(VPl & ((1u << q) - 1));
    t0_materialize(c, t, Pbase, f.z, q, f.w, pool_block(*c.P, blk));
    pool_publish(c, blk);
    VPl &= ~(1u << q);
  }
  if (c.lane == 0) sm->t0f[l].y = VPl;
  __syncwarp();
  return true;
}

// A node with 2 to kSmallP candidates P, active rows A and R = RM, decided in
// one step.  R + K is a maximal clique for exactly the cliques K of the
// candidates that no active row contains (a candidate outside K that extends K
// is itself such a row).  A subset is a lane number b (bit k: the k-th lowest
// candidate, for the low five) and a set of the others (a group); the subsets
// of one group are one 32-bit word.  Every lane marks the subsets that its row
// rules out: those the row contains and, if the row is a candidate, those that
// hold it and a candidate it is not adjacent to.  Inside a group both depend
// only on whether the row holds the group's members, so a lane has its two
// words ready, and a group costs a select, one redux over the warp and the
// leaves of what is left, which every lane knows; lane b writes subset b's.
// A search tree spends about 250 instructions on a node and its share of
// leaves; a group takes about 12.
__device__ __forceinline__ void t0_small_sets(const Ctx &c, uint32_t row, uint32_t P, uint32_t A, uint32_t RM,
                                              uint32_t &npend) {
  WarpSmem *sm = c.sm;
  const uint32_t lane = c.lane, lanebit = 1u << lane;
  uint32_t sub = 1;   // subsets of the low candidates that the row contains
  uint32_t mask = RM; // R and this lane's subset of the low candidates
  uint32_t high = P;
#pragma unroll
  for (int k = 0; k < 5; k++) {  // past the last candidate: qb = 0, nothing happens
    const uint32_t qb = high & (0u - high);
    high ^= qb;
    if (row & qb) sub |= sub << (1 << k);
    if ((lane >> k) & 1) mask |= qb;
  }
  const bool active = A & lanebit, mine = high & lanebit;
  // subsets ruled out where the row holds the group's (other) members, and where not
  uint32_t dead_in = active ? sub : 0, dead_out = 0;
  const uint32_t low = P ^ high;
  if (low & lanebit) {  // candidate i of the low five: subsets with i need the row to hold the rest
    const uint32_t i = __popc(low & lanemask_lt());
    const uint32_t with_i = i == 0   ? 0xAAAAAAAAu
                            : i == 1 ? 0xCCCCCCCCu
                            : i == 2 ? 0xF0F0F0F0u
                            : i == 3 ? 0xFF00FF00u
                                     : 0xFFFF0000u;
    dead_in |= with_i & ~(sub << (1u << i));
    dead_out = with_i;
  }
  const uint32_t miss = high & ~row & ~lanebit;  // members the row does not hold
  const uint32_t n = __popc(P);
  const uint32_t all = n >= 5 ? 0xffffffffu : (1u << (1u << n)) - 1;
  uint32_t members = 0;
#pragma unroll 1
  do {
    const bool out_row = members & miss;
    uint32_t dead = out_row ? dead_out : dead_in;
    if (mine && (members & lanebit)) dead = out_row ? 0xffffffffu : ~sub;
    const uint32_t E = all & ~__reduce_or_sync(kFull, dead);
    if (E) {
      const bool out = E & lanebit;
      const uint32_t pos = npend + __popc(E & lanemask_lt());
      const uint32_t leaf = mask | members;
      if (out && pos < 32) sm->pend_rm[pos] = leaf;
      npend += __popc(E);
      if (npend >= 32) {
        t0_flush(c, 32);
        if (out && pos >= 32) sm->pend_rm[pos - 32] = leaf;
        npend -= 32;
      }
    }
    members = (members - high) & high;  // the next set of high candidates, back to none after the last
  } while (members);
}

// The leaf of an entry of t0_batch: its fixed columns and the low candidates
// its subset number selects.
__device__ __forceinline__ uint32_t batch_leaf(const WarpSmem *sm, uint32_t fixed, uint32_t entry) {
  uint32_t P = sm->pr_P[entry >> 5], leaf = fixed;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const uint32_t qb = P & (0u - P);
    P ^= qb;
    if ((entry >> k) & 1) leaf |= qb;
  }
  return leaf;
}

// Collected small nodes without X rows, one node per lane: the same subset
// words as t0_small_sets, with the candidates' rows taken in turn instead of
// one per lane, so 32 nodes cost what 3 to 5 cost there.  Leaves are queued
// and hashed 32 at a time.
// Measured (B200): full R-MAT 15 (edge factor 16; 5.4e9 cliques, nine small
// nodes in ten have no X rows) 482 -> 391 ms against deciding each by itself
// (t0_small_sets), 562 ms with one-step decisions up to 6 candidates only.
__device__ __noinline__ void t0_batch(const EnumParams *Pm, WarpSmem *sm, uint32_t nprob) {
  const uint32_t lane = lane_id();
  constexpr int NH = kSmallP - 5;
  uint32_t *ent_leaf = sm->xrow, *ent_sub = sm->xcv;  // the exchange buffer is free inside a solve
  __syncwarp();
  const bool live = lane < nprob;
  const uint32_t P = live ? sm->pr_P[lane] : 0u, RM = live ? sm->pr_RM[lane] : 0u;
  uint32_t q[5], high = P;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    q[k] = high & (0u - high);
    high ^= q[k];
  }
  // per candidate: the subsets it rules out in a group whose members its row
  // holds, and the group members its row misses (see t0_small_sets)
  constexpr uint32_t kWith[5] = {0xAAAAAAAAu, 0xCCCCCCCCu, 0xF0F0F0F0u, 0xFF00FF00u, 0xFFFF0000u};
  uint32_t dead_in[kSmallP], miss[kSmallP], hb[NH];
  uint32_t hrest = high;
#pragma unroll
  for (int k = 0; k < NH; k++) {
    hb[k] = hrest & (0u - hrest);
    hrest ^= hb[k];
  }
#pragma unroll
  for (int i = 0; i < kSmallP; i++) {
    const uint32_t own = i < 5 ? q[i < 5 ? i : 0] : hb[i < 5 ? 0 : i - 5];
    const uint32_t row = own ? sm->pr_row[33 * i + lane] : 0u;
    uint32_t sub = 1;
#pragma unroll
    for (int k = 0; k < 5; k++)
      if (row & q[k]) sub |= sub << (1 << k);
    dead_in[i] = i < 5 ? sub | (kWith[i < 5 ? i : 0] & ~(sub << (1 << (i < 5 ? i : 0)))) : sub;
    if (!own) dead_in[i] = 0;
    miss[i] = own ? high & ~row & ~own : 0u;
  }
  const uint32_t n = __popc(P);
  const uint32_t all = n >= 5 ? 0xffffffffu : live ? (1u << (1u << n)) - 1 : 0u;
  uint32_t members = 0, queued = 0;
  bool more = live;
#pragma unroll 1
  do {
    uint32_t dead = 0;
#pragma unroll
    for (int i = 0; i < 5; i++) dead |= (members & miss[i]) ? kWith[i] : dead_in[i];
#pragma unroll
    for (int k = 0; k < NH; k++) {
      const uint32_t w = (members & miss[5 + k]) ? 0u : dead_in[5 + k];
      dead |= (members & hb[k]) ? ~w : w;
    }
    uint32_t E = more ? all & ~dead : 0u;
    const uint32_t fixed = RM | members;
    for (uint32_t bal = __ballot_sync(kFull, E != 0); bal; bal = __ballot_sync(kFull, E != 0)) {
      const bool out = E != 0;
      const uint32_t pos = queued + __popc(bal & lanemask_lt());
      const uint32_t sub = lane << 5 | (__ffs(E) - 1);
      E &= E - 1;
      if (out && pos < 32) {
        ent_leaf[pos] = fixed;
        ent_sub[pos] = sub;
      }
      queued += __popc(bal);
      if (queued >= 32) {
        __syncwarp();
        t0_hash(Pm, sm, batch_leaf(sm, ent_leaf[lane], ent_sub[lane]), true);
        if (out && pos >= 32) {
          ent_leaf[pos - 32] = fixed;
          ent_sub[pos - 32] = sub;
        }
        queued -= 32;
      }
    }
    members = (members - high) & high;
    more = more && members;
  } while (__any_sync(kFull, more));
  __syncwarp();
  if (queued) {
    const bool have = lane < queued;
    t0_hash(Pm, sm, have ? batch_leaf(sm, ent_leaf[lane], ent_sub[lane]) : 0u, have);
  }
}

// A subproblem that collected fewer small nodes than this decides them one at
// a time: a batch costs as much for one node as for 32.
// Measured (B200), ms, for limits of 1, 8, 16, 24 and 33 (only full batches):
// G(1000, mean degree 200) 6.32, 5.65, 5.64, 5.60, 5.62; 300 G(n, p) graphs 10.7,
// 9.5, 9.4, 9.4, 9.4; full R-MAT 15 222, 220, 220, 223, 227.
constexpr uint32_t kBatchMin = 16;

// ------------------------------------------------ join decomposition
// A node whose active rows are all candidates (no X row contains R) has as
// its maximal cliques R + K for exactly the maximal cliques K of G[P].  Let H
// be the complement of G[P].  G[P] is the join of the complements of H's
// connected components, so its maximal cliques are the products of one
// maximal clique of each component's complement, i.e. one maximal independent
// set (in H) per component.  When every component is small, the node is
// decided without a search tree: count, histogram and largest size in closed
// form, and the checksum by walking the products, 32 lanes at a time.
//
// The caller has checked that no closed H-neighbourhood P \ row is larger than
// a component may be.  Components: breadth-first search with ballots over
// those.  Component j's maximal independent sets come from the 2^s
// subsets of its s members, one per lane, and are packed into a table of at
// most 32 entries in shared memory (hash sums and size of each set).  Lane j
// holds component j's first entry and entry count.
//
// Walking the products: the first components whose entry counts multiply to
// at most 32 (Q) are carried by the lane index (each lane adds up its own
// entries once); the others form a warp-uniform mixed-radix counter, whose
// steps swap one entry per digit that moves.
constexpr int kJoinComp = 5;    // largest component decided this way
#ifndef MCE_JOIN_MIN
#define MCE_JOIN_MIN 10
#endif
constexpr int kJoinMin = MCE_JOIN_MIN;  // smallest |P| worth the decomposition

__device__ __noinline__ bool t0_join(const EnumParams *Pm, WarpSmem *sm, uint32_t row, uint32_t P, uint32_t RM) {
  const uint32_t lane = lane_id();
  const bool inP = (P >> lane) & 1;
  const uint32_t nb = inP ? (P & ~row) : 0u;  // closed non-neighbourhood in P (rows carry no self bit)
  const uint32_t single = __ballot_sync(kFull, inP && nb == (1u << lane));  // adjacent to every candidate
  // components first: a node is abandoned before any set is built
  uint32_t rem = P & ~single;
  uint32_t comp = 0, ncomp = 0;  // lane j: component j's members
  #pragma unroll 1
  while (rem) {
    uint32_t C = rem & (0u - rem), fr = C;
    do {
      const uint32_t nbr = __ballot_sync(kFull, (nb & fr) != 0);
      fr = nbr & ~C;
      C |= nbr;
    } while (fr && __popc(C) <= kJoinComp);
    if (__popc(C) > kJoinComp) return false;
    if (lane == ncomp) comp = C;
    ncomp++;
    rem &= ~C;
  }
  // Scratch while the node is decided: the exchange buffer and the row buffer
  // (free inside a 32-bit-tier solve).  xrow: closed non-neighbourhoods by
  // column; rowbuf[e], rowbuf[32 + e], xcv[e]: entry e's hash sums and size.
  uint64_t *E1 = sm->rowbuf, *E2 = sm->rowbuf + 32;
  uint32_t *ES = sm->xcv;
  sm->xrow[lane] = nb;
  __syncwarp();
  uint32_t nent = 0, c_off = 0, c_r = 0;  // lane j: component j's first entry and entry count
  uint64_t total = 1;
  #pragma unroll 1
  for (uint32_t j = 0; j < ncomp; j++) {
    const uint32_t C = __shfl_sync(kFull, comp, j);
    const uint32_t ns = __popc(C);
    // lane l tests the subset l of C's members (bit k = k-th lowest member)
    uint32_t sub = 0;
    uint64_t a1 = 0, a2 = 0;
    uint32_t cm = C;
    #pragma unroll 1
    for (uint32_t k = 0; k < ns; k++) {
      const uint32_t b = cm & (0u - cm);
      cm ^= b;
      if ((lane >> k) & 1) {
        const uint32_t m = __ffs(b) - 1;
        sub |= b;
        a1 += sm->xh1[m];
        a2 += sm->xh2[m];
      }
    }
    bool ok = lane != 0 && lane < (1u << ns);
    cm = C;
    #pragma unroll 1
    for (uint32_t k = 0; k < ns; k++) {
      const uint32_t b = cm & (0u - cm);
      cm ^= b;
      const uint32_t nbk = sm->xrow[__ffs(b) - 1];
      // independent: no other member of the subset is a non-neighbour;
      // maximal: every member outside has a non-neighbour inside
      ok = ok && ((sub & b) ? (nbk & sub) == b : (nbk & sub) != 0);
    }
    const uint32_t mis = __ballot_sync(kFull, ok);
    const uint32_t r = __popc(mis);
    if (nent + r > 32) return false;
    if (ok) {
      const uint32_t e = nent + __popc(mis & lanemask_lt());
      E1[e] = a1;
      E2[e] = a2;
      ES[e] = __popc(sub);
    }
    if (lane == j) {
      c_off = nent;
      c_r = r;
    }
    nent += r;
    total *= r;
  }
  __syncwarp();
  // the part every clique shares: R and the candidates adjacent to all others
  const uint32_t base_cols = RM | single;
  const uint64_t b1 = sm->t0_s1 + warp_sum_u64(((base_cols >> lane) & 1) ? sm->xh1[lane] : 0);
  const uint64_t b2 = sm->t0_s2 + warp_sum_u64(((base_cols >> lane) & 1) ? sm->xh2[lane] : 0);
  const uint32_t size0 = sm->t0_rsize + 2 + __popc(base_cols);
  // sizes: the product of the components' size polynomials, lane = size - size0
  // (a component's sets leave out at least one member, so sizes stay below size0 + 32)
  uint32_t poly = lane == 0 ? 1u : 0u;
  #pragma unroll 1
  for (uint32_t j = 0; j < ncomp; j++) {
    const uint32_t off = __shfl_sync(kFull, c_off, j), r = __shfl_sync(kFull, c_r, j);
    uint32_t acc = 0;
    #pragma unroll 1
    for (uint32_t d = 0; d < r; d++) {
      const uint32_t sz = ES[off + d];
      const uint32_t v = __shfl_up_sync(kFull, poly, sz);
      if (lane >= sz) acc += v;
    }
    poly = acc;
  }
  {
    const uint32_t size = size0 + lane;
    if (poly) {
      if (size < kHistCache) {
        atomicAdd(&sm->hcache[size], poly);
      } else {
        const uint32_t bin = size < Pm->hist_len ? size : Pm->hist_len - 1;
        atomicAdd(&Pm->hist[(uint64_t)sm->slot * Pm->hist_len + bin], (unsigned long long)poly);
      }
    }
    const uint32_t mx = __reduce_max_sync(kFull, poly ? size : 0u);
    if (lane == 0) {
      sm->count += total;
      sm->pending += (uint32_t)total;
      sm->max_size = max(sm->max_size, mx);
    }
  }
  // lane-carried components 0 .. a - 1 (Q products): each lane's own sums
  uint32_t a = 0, Q = 1;
  #pragma unroll 1
  while (a < ncomp) {
    const uint32_t r = __shfl_sync(kFull, c_r, a);
    if (Q * r > 32) break;
    Q *= r;
    a++;
  }
  uint64_t p1 = b1, p2 = b2;
  uint32_t psz = size0;
  {
    uint32_t rest = lane;
    #pragma unroll 1
    for (uint32_t j = 0; j < a; j++) {
      const uint32_t off = __shfl_sync(kFull, c_off, j), r = __shfl_sync(kFull, c_r, j);
      const uint32_t d = rest % r;
      rest /= r;
      p1 += E1[off + d];
      p2 += E2[off + d];
      psz += ES[off + d];
    }
  }
  // counter-carried components a .. ncomp - 1: digits in lanes, sums uniform
  uint32_t dig = 0;
  uint64_t h1 = 0, h2 = 0;
  uint32_t hsz = 0;
  #pragma unroll 1
  for (uint32_t j = a; j < ncomp; j++) {
    const uint32_t off = __shfl_sync(kFull, c_off, j);
    h1 += E1[off];
    h2 += E2[off];
    hsz += ES[off];
  }
  uint64_t chk = 0;
  const bool live = lane < Q;
  #pragma unroll 1
  for (;;) {
    if (live) chk += clique_hash(p1 + h1, p2 + h2, psz + hsz);
    // next value of the counter: the lowest digit below its top moves up,
    // the digits under it wrap to their first entry
    const uint32_t can = __ballot_sync(kFull, lane >= a && lane < ncomp && dig + 1 < c_r);
    if (!can) break;
    const uint32_t jmax = __ffs(can) - 1;
    #pragma unroll 1
    for (uint32_t j = a; j <= jmax; j++) {
      const uint32_t off = __shfl_sync(kFull, c_off, j);
      const uint32_t cur = off + __shfl_sync(kFull, dig, j);
      const uint32_t nxt = j == jmax ? cur + 1 : off;
      h1 += E1[nxt] - E1[cur];
      h2 += E2[nxt] - E2[cur];
      hsz += ES[nxt] - ES[cur];
    }
    if (lane >= a && lane < jmax) dig = 0;
    if (lane == jmax) dig++;
  }
  sm->lchk[lane] += chk;
  __syncwarp();
  return true;
}

// kStats: count search-tree nodes and row word-ops (a separate instance, so
// the counting costs nothing when it is off)
//
// The node loop makes no calls, which keeps its registers free.  To expose
// work it steps out instead: it saves its state and returns true; the caller
// (t0_run) exposes levels and calls it again with resume set.
template <bool kStats>
__device__ __noinline__ bool t0_solve_body(Ctx c, uint32_t row, uint32_t pc, uint32_t nrows, bool resume) {
  const uint32_t lane = c.lane;
  WarpSmem *sm = c.sm;
  const bool expand_r = c.P->expand_r != 0;
  uint32_t A, P, RM, npend, nprob;
  int level;
  if (!resume) {
    A = nrows >= 32 ? ~0u : ((1u << nrows) - 1);
    P = pc >= 32 ? ~0u : ((1u << pc) - 1);
    RM = 0;
    npend = 0;
    nprob = 0;
    level = 0;
  } else {
    P = sm->y_P;
    A = sm->y_A;
    RM = sm->y_RM;
    npend = sm->y_npend;
    nprob = sm->y_nprob;
    level = sm->y_level;
  }
  const uint32_t lanebit = 1u << lane;
  unsigned long long nodes = 0, wops = 0;  // uniform across lanes
  uint32_t tick = 0;
  const uint32_t period = sm->share_period;
  // A child whose candidate set comes out empty is a leaf: it is tested where
  // it is made, without a frame push, a descent and a backtrack.
  uint32_t VP = 0;
  uint32_t sP = 0, sA = 0, sRM = 0;  // a node or child that is decided in one step
node:  // a node with candidates P, active rows A and R = RM
  if (kStats) nodes++;
  if (P == 0) {  // only a subproblem without columns starts like this
    if (A == 0) {
      if (lane == 0) sm->pend_rm[npend] = RM;
      ++npend;
    }
    goto backtrack;
  }
  if (__popc(P) <= kSmallP) {
    if (kStats) nodes++;
    sP = P;
    sA = A;
    sRM = RM;
    P = 0;  // no candidate of this node is left: the way on is back
    goto small;
  }
  {
    const uint32_t far = (uint32_t)__popc(P & ~row);  // a candidate's row holds no self bit: it counts itself
    if (__popc(P) >= kJoinMin && (A & ~P) == 0 &&
        __reduce_max_sync(kFull, (P & lanebit) ? far : 0u) <= (uint32_t)kJoinComp &&
        t0_join(c.P, sm, row, P, RM))
      goto backtrack;
    const uint32_t key = (A & lanebit) ? ((far << 5) | lane) : 0xffffffffu;
    const uint32_t kmin = __reduce_min_sync(kFull, key);
    if (kStats) wops += 2 * __popc(A);  // ANDN + POPC per active row
    if ((kmin >> 5) == 0) goto backtrack;  // an X row covers P: nothing maximal below
    VP = P & ~__shfl_sync(kFull, row, kmin & 31);
  }
expand:  // next candidate of VP at this level
  {
    const uint32_t cand = P & VP;
    if (cand == 0) goto backtrack;
    const uint32_t q = __ffs(cand) - 1;
    P &= ~(1u << q);
    // the child's candidates and the rows holding q: two independent
    // collectives; rows holding R' = R + q (+ E) are A & those
    uint32_t P2 = P & __shfl_sync(kFull, row, q);
    uint32_t A2 = A & __ballot_sync(kFull, (row >> q) & 1);
    uint32_t M = 1u << q;
    if (expand_r && (P2 & (P2 - 1))) {
      // EXPAND_R: a candidate adjacent to every other candidate joins R at
      // once; rows carry no self bit, so that is P2 \ row == {itself}
      const uint32_t E = __ballot_sync(kFull, (P2 & ~row) == lanebit);
      if (kStats) wops += 2 * __popc(P2);
      if (E) {
        P2 &= ~E;
        M |= E;
        A2 &= __ballot_sync(kFull, (row & E) == E);
      }
    }
    if (kStats) wops += __popc(A) + 1;
    if (P2 == 0) {  // leaf child: maximal iff no row contains R + M
      if (kStats) nodes++;
      if (A2 == 0) {
        if (lane == 0) sm->pend_rm[npend] = RM | M;
        if (++npend == 32) {
          t0_flush(c, 32);
          npend = 0;
        }
      }
      goto expand;
    }
    if (__popc(P2) <= kSmallP) {  // small child: decided here, no descent
      if (kStats) nodes++;
      sP = P2;
      sA = A2;
      sRM = RM | M;
      goto small;
    }
    // a child that is its parent's last open candidate replaces the parent
    // (no frame: the parent would only backtrack after it)
    if (cand & (cand - 1)) {
      sm->t0f[level] = make_uint4(P, VP, A, RM);
      level++;
    }
    P = P2;
    A = A2;
    RM |= M;
    if (c.sharing && ++tick >= period) {
      tick = 0;
      if (hungry(c)) {
        // step out at this fresh node; t0_run exposes work and resumes
        __syncwarp();
        if (lane == 0) {
          sm->y_P = P;
          sm->y_A = A;
          sm->y_RM = RM;
          sm->y_npend = npend;
          sm->y_nprob = nprob;
          sm->y_level = level;
          if (kStats) {
            sm->nodes += nodes;
            sm->wops += wops;
          }
        }
        __syncwarp();
        return true;
      }
    }
    goto node;
  }
small:  // one copy of the small decisions, for nodes and children
  if ((sP & (sP - 1)) == 0) {
    // One candidate q: R + q is maximal iff no active row holds q (the pivot
    // step would prune on such a row, else branch on q into a leaf).
    if ((sA & __ballot_sync(kFull, (row & sP) != 0)) == 0) {
      if (lane == 0) sm->pend_rm[npend] = sRM | sP;
      if (++npend == 32) {
        t0_flush(c, 32);
        npend = 0;
      }
    }
    goto expand;
  }
  // X rows without a candidate rule nothing out
  if ((sA & ~sP) == 0 || !__any_sync(kFull, (sA & ~sP & lanebit) && (row & sP))) {
    if (sP & lanebit) sm->pr_row[33 * __popc(sP & lanemask_lt()) + nprob] = row;
    if (lane == 0) {
      sm->pr_P[nprob] = sP;
      sm->pr_RM[nprob] = sRM;
    }
    if (++nprob == 32) {
      t0_batch(c.P, sm, 32);
      nprob = 0;
    }
    goto expand;
  }
sets:
  t0_small_sets(c, row, sP, sA, sRM, npend);
  goto expand;
backtrack:
  if (level > 0) {
    level--;
    const uint4 f = sm->t0f[level];
    P = f.x;
    VP = f.y;
    A = f.z;
    RM = f.w;
    goto expand;
  }
  if (nprob >= kBatchMin) {
    t0_batch(c.P, sm, nprob);
  } else if (nprob) {  // too few for a batch: one at a time
    __syncwarp();
    nprob--;
    sP = sA = sm->pr_P[nprob];
    sRM = sm->pr_RM[nprob];
    P = VP = 0;
    goto sets;
  }
  if (npend) t0_flush(c, npend);
  if (kStats && lane == 0) {
    sm->nodes += nodes;
    sm->wops += wops;
  }
  __syncwarp();
  maybe_flush(c);
  return false;
}

__device__ __forceinline__ void t0_run(const Ctx &c, const T0 &t, uint32_t pc, uint32_t nrows, uint32_t rsize0,
                                       uint64_t s10, uint64_t s20) {
  WarpSmem *sm = c.sm;
  sm->xh1[c.lane] = t.h1;
  sm->xh2[c.lane] = t.h2;
  if (c.lane == 0) {
    sm->t0_s1 = s10;
    sm->t0_s2 = s20;
    sm->t0_rsize = rsize0;
  }
  __syncwarp();
  bool resume = false;
  for (;;) {
    const bool out = c.P->stats ? t0_solve_body<true>(c, t.row, pc, nrows, resume)
                                : t0_solve_body<false>(c, t.row, pc, nrows, resume);
    if (!out) break;
    const bool any = t0_share(c, t, c.sm->y_level);
    if (c.lane == 0) c.sm->share_period = any ? kShareMin : min(c.sm->share_period * 2, kShareMax);
    __syncwarp();
    resume = true;
  }
}

// timed wrapper: cycles go to the register-tier phase, spawning excluded
__device__ __forceinline__ void t0_solve(const Ctx &c, const T0 &t, uint32_t pc, uint32_t nrows, uint32_t rsize0,
                                         uint64_t s10, uint64_t s20) {
  const unsigned long long t0 = now(), sp0 = c.sm->cyc[kCycSpawn];
  t0_run(c, t, pc, nrows, rsize0, s10, s20);
  if (c.lane == 0) c.sm->cyc[kCycT0] += (now() - t0) - (c.sm->cyc[kCycSpawn] - sp0);
}

// a W = 1 record with pc <= 32 and nrows <= 32, from a pool block (cg loads)
// or from this warp's own slab
template <bool kCoherent>
__device__ __forceinline__ void t0_load(const Ctx &c, const char *rec, T0 &t, uint32_t pc, uint32_t nrows) {
  const uint32_t *colv = (const uint32_t *)(rec + kHdr);
  const uint64_t *rows = (const uint64_t *)(rec + kHdr + align8(4ULL * pc));
  const uint32_t lane = c.lane;
  if (kCoherent) {
    t.row = lane < nrows ? (uint32_t)ld_cg(rows + lane) : 0;
    t.cv = lane < pc ? ld_cg(colv + lane) : 0;
  } else {
    t.row = lane < nrows ? (uint32_t)rows[lane] : 0;
    t.cv = lane < pc ? colv[lane] : 0;
  }
  t.h1 = lane < pc ? c.P->g.h1[t.cv] : 0;
  t.h2 = lane < pc ? c.P->g.h2[t.cv] : 0;
}

// ---------------------------------------------------------- 64-bit tier

struct T1 {
  uint64_t r[kRPL];   // rows lane, lane+32, lane+64, lane+96
  uint64_t h1a, h1b;  // label hashes of columns lane, lane+32
  uint64_t h2a, h2b;
  uint32_t cva, cvb;  // vertex ids of columns lane, lane+32
};

__device__ __forceinline__ uint64_t sel_row(const T1 &t, uint32_t j) {
  return j == 0 ? t.r[0] : j == 1 ? t.r[1] : j == 2 ? t.r[2] : t.r[3];
}
__device__ __forceinline__ uint64_t bcast_row(const T1 &t, uint32_t idx) {
  return __shfl_sync(kFull, sel_row(t, idx >> 5), idx & 31);
}

__device__ __forceinline__ void t1_hashes(const Ctx &c, T1 &t, uint32_t pc) {
  const DevGraph &g = c.P->g;
  t.h1a = c.lane < pc ? g.h1[t.cva] : 0;
  t.h2a = c.lane < pc ? g.h2[t.cva] : 0;
  t.h1b = c.lane + 32 < pc ? g.h1[t.cvb] : 0;
  t.h2b = c.lane + 32 < pc ? g.h2[t.cvb] : 0;
}

// a W = 1 record with nrows <= 128 into registers
template <bool kCoherent>
__device__ __forceinline__ void t1_load(const Ctx &c, const char *rec, T1 &t, uint32_t pc, uint32_t nrows) {
  const uint32_t *colv = (const uint32_t *)(rec + kHdr);
  const uint64_t *rows = (const uint64_t *)(rec + kHdr + align8(4ULL * pc));
#pragma unroll
  for (int j = 0; j < kRPL; j++) {
    const uint32_t idx = 32 * j + c.lane;
    t.r[j] = idx < nrows ? (kCoherent ? ld_cg(rows + idx) : rows[idx]) : 0;
  }
  t.cva = c.lane < pc ? (kCoherent ? ld_cg(colv + c.lane) : colv[c.lane]) : 0;
  t.cvb = c.lane + 32 < pc ? (kCoherent ? ld_cg(colv + c.lane + 32) : colv[c.lane + 32]) : 0;
  t1_hashes(c, t, pc);
}

// Child task of candidate q of a 64-bit-tier level, into `rec`: columns =
// Pbase & row(q), rows = active rows holding bit q, compressed to the columns.
__device__ void t1_materialize(const Ctx &c, const T1 &t, uint64_t Pbase, uint32_t ab, uint32_t q, uint32_t rsize,
                               uint64_t s1, uint64_t s2, char *rec) {
  const uint32_t lane = c.lane;
  const uint64_t CP = Pbase & bcast_row(t, q);
  const uint32_t pc = __popcll(CP);
  const CPlan plan = compress_plan(CP);
  const uint64_t hq1 = __shfl_sync(kFull, q < 32 ? t.h1a : t.h1b, q & 31);
  const uint64_t hq2 = __shfl_sync(kFull, q < 32 ? t.h2a : t.h2b, q & 31);
  uint32_t *colv = (uint32_t *)(rec + kHdr);
  uint64_t *rows = (uint64_t *)(rec + kHdr + align8(4ULL * pc));
  // candidate rows (row index == column index < 64) in column order
  if ((CP >> lane) & 1) {
    const uint32_t k = __popcll(CP & ((1ULL << lane) - 1));
    colv[k] = t.cva;
    rows[k] = compress_apply(t.r[0], plan);
  }
  if ((CP >> (lane + 32)) & 1) {
    const uint32_t k = __popcll(CP & ((1ULL << (lane + 32)) - 1));
    colv[k] = t.cvb;
    rows[k] = compress_apply(t.r[1], plan);
  }
  // X rows: active, holding bit q, not a column of the child
  uint32_t base = pc;
#pragma unroll
  for (int j = 0; j < kRPL; j++) {
    const uint32_t idx = 32 * j + lane;
    const bool act = ((ab >> j) & 1) && ((t.r[j] >> q) & 1);
    const bool isc = idx < 64 && ((CP >> idx) & 1);
    const bool isx = act && !isc && (CP == 0 || (t.r[j] & CP) != 0);  // empty X rows left out
    const uint32_t bal = __ballot_sync(kFull, isx);
    if (isx) rows[base + __popc(bal & lanemask_lt())] = compress_apply(t.r[j], plan);
    base += __popc(bal);
  }
  if (lane == 0) {
    TaskHdr *h = (TaskHdr *)rec;
    h->pc = pc;
    h->nrows = base;
    h->W = 1;
    h->rsize = rsize + 1;
    h->s1 = s1 + hq1;
    h->s2 = s2 + hq2;
    h->slot = c.sm->slot;
  }
  __syncwarp();
}

// shallowest 64-bit-tier level below `level` with open candidates and
// |P| >= tau, or -1
__device__ __forceinline__ int t1_open_level(const Ctx &c, int level) {
  const T1Area *ta = c.ta;
  for (int l = 0; l < level; l++) {
    const uint64_t Pl = ta->fP[l];
    if ((Pl & ta->fVP[l]) && (uint32_t)__popcll(Pl) + 1 >= c.P->reg_share_bound) return l;
  }
  return -1;
}

__device__ bool t1_spawn(const Ctx &c, const T1 &t, int level) {
  T1Area *ta = c.ta;
  int l = 0;
  uint64_t open = 0;
  for (; l < level; l++) {
    open = ta->fP[l] & ta->fVP[l];
    if (open && (uint32_t)__popcll(ta->fP[l]) + 1 >= c.P->reg_share_bound) break;
    open = 0;
  }
  if (!open) return false;
  const uint64_t Pl = ta->fP[l];
  uint64_t VPl = ta->fVP[l];
  const uint32_t abl = ta->fab[l][c.lane];
  const uint32_t rs = ta->frs[l];
  const uint64_t s1 = ta->fs1[l], s2 = ta->fs2[l];
  // highest open candidate first (see t0_spawn)
  while (open) {
    const uint32_t q = 63 - __clzll((long long)open);
    open &= ~(1ULL << q);
    uint32_t blk;
    if (!pool_alloc(c, &blk)) break;
    const uint64_t Pbase = Pl & ~(VPl & ((1ULL << q) - 1));
    t1_materialize(c, t, Pbase, abl, q, rs, s1, s2, pool_block(*c.P, blk));
    pool_publish(c, blk);
    VPl &= ~(1ULL << q);
  }
  if (c.lane == 0) ta->fVP[l] = VPl;
  __syncwarp();
  return true;
}

// The children of a 64-bit-tier node that are small, one a lane.  Candidates
// are taken in ascending order, so the ones above the last child with more than
// 5 candidates of its own can be taken out of turn: each leaves out the open
// candidates below it.  Every lane decides its child on words of subsets (see
// t0_small_sets): the rows pass by in turn, the same one in every lane, and a
// lane marks the subsets that the row rules out if it holds the lane's
// candidate.  A sparse ego network's root has dozens of such children, and
// descending into each costs as much as all of them cost here.
// Measured (B200): 300 G(n, p) graphs in one launch 13.9 -> 10.1 ms.
// Returns the candidates taken.  a0..a3: active rows 0-31, 32-63, ...
__device__ __noinline__ uint64_t t1_children(const EnumParams *Pm, WarpSmem *sm, const T1Area *ta, uint64_t P,
                                             uint64_t VP, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t rsize, uint64_t s1, uint64_t s2) {
  const uint32_t lane = lane_id();
  const DevGraph &g = Pm->g;
  // this lane's two candidates and their children's candidates
  uint64_t cp[2];
  uint32_t big[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const uint32_t q = 32 * j + lane;
    const bool mine = (VP >> q) & 1;
    cp[j] = mine ? P & ~(VP & ((1ULL << q) - 1)) & ta->t1rows[q] & ~(1ULL << q) : 0;
    big[j] = __ballot_sync(kFull, __popcll(cp[j]) > 5);
  }
  const uint64_t large = (uint64_t)big[0] | ((uint64_t)big[1] << 32);
  const uint64_t take = large ? VP & ~((2ULL << (63 - __clzll((long long)large))) - 1) : VP;
  if (__popcll(take) < 4) return 0;
#pragma unroll 1
  for (int j = 0; j < 2; j++) {
    const uint32_t q = 32 * j + lane;
    const bool mine = (take >> q) & 1;
    if (!__any_sync(kFull, mine)) continue;
    const uint64_t C = j ? cp[1] : cp[0];
    uint64_t m[5];
    uint64_t rest = C;
#pragma unroll
    for (int k = 0; k < 5; k++) {
      m[k] = rest & (0ULL - rest);
      rest ^= m[k];
    }
    uint32_t dead = 0;
#pragma unroll 1
    for (int w = 0; w < 4; w++) {
      uint32_t act = w == 0 ? a0 : w == 1 ? a1 : w == 2 ? a2 : a3;
      while (act) {
        const uint64_t row = ta->t1rows[32 * w + __ffs(act) - 1];
        act &= act - 1;
        uint32_t sub = (uint32_t)(row >> q) & 1;  // nothing from a row without the candidate
#pragma unroll
        for (int k = 0; k < 5; k++)
          if (row & m[k]) sub |= sub << (1 << k);
        dead |= sub;
      }
    }
    // the candidates' own rows: subsets with a candidate need its row to hold the rest
    constexpr uint32_t kWith[5] = {0xAAAAAAAAu, 0xCCCCCCCCu, 0xF0F0F0F0u, 0xFF00FF00u, 0xFFFF0000u};
    const uint32_t n = __popcll(C);
    uint64_t h1[5], h2[5];
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const bool have = mine && (uint32_t)i < n;
      const uint32_t col = have ? __ffsll((long long)m[i]) - 1 : 0;
      const uint64_t row = ta->t1rows[col];
      uint32_t sub = 1;
#pragma unroll
      for (int k = 0; k < 5; k++)
        if (row & m[k]) sub |= sub << (1 << k);
      if (have) dead |= kWith[i] & ~(sub << (1 << i));
      const uint32_t v = ta->t1cv[col];
      h1[i] = have ? g.h1[v] : 0;
      h2[i] = have ? g.h2[v] : 0;
    }
    const uint32_t all = n >= 5 ? 0xffffffffu : (1u << (1u << n)) - 1;
    uint32_t E = mine ? all & ~dead : 0u;
    uint64_t b1 = s1, b2 = s2;
    if (E) {
      const uint32_t v = ta->t1cv[q];
      b1 += g.h1[v];
      b2 += g.h2[v];
    }
    while (__any_sync(kFull, E != 0)) {
      const bool live = E != 0;
      const uint32_t b = live ? __ffs(E) - 1 : 0;
      E &= E - 1;
      uint64_t x = b1, y = b2;
#pragma unroll
      for (int i = 0; i < 5; i++)
        if ((b >> i) & 1) {
          x += h1[i];
          y += h2[i];
        }
      leaves_out(Pm, sm, live, x, y, rsize + 3 + __popc(b));
    }
  }
  return take;
}

__device__ __noinline__ void t1_solve_body(Ctx c, T1 t, uint32_t pc, uint32_t nrows, uint32_t rsize0, uint64_t s10,
                                           uint64_t s20) {
  T1Area *ta = c.ta;
  const uint32_t lane = c.lane;
  WarpSmem *sm = c.sm;
  const bool expand_r = c.P->expand_r != 0;
  uint32_t ab = 0;
#pragma unroll
  for (int j = 0; j < kRPL; j++)
    if (32 * j + lane < nrows) ab |= 1u << j;
  uint64_t P = pc >= 64 ? ~0ULL : ((1ULL << pc) - 1);
  uint64_t VP = 0;
  uint32_t rsize = rsize0;
#pragma unroll
  for (int j = 0; j < kRPL; j++) ta->t1rows[32 * j + lane] = t.r[j];
  ta->t1cv[lane] = t.cva;
  ta->t1cv[lane + 32] = t.cvb;
  if (lane == 0) {
    sm->t1_pc = pc;
    sm->nest |= kNestT1;
  }
  __syncwarp();
  uint64_t s1 = s10, s2 = s20;
  unsigned long long nodes = 0, wops = 0;  // nodes uniform; wops per lane
  int level = 0;
  bool fresh = true;
  uint32_t tick = 0;
  for (;;) {
    if (fresh) {
      nodes++;
      if (P == 0) {
        if (!__any_sync(kFull, ab != 0) && lane == 0) emit(c, rsize + 2, s1, s2);
        goto backtrack;
      }
      {
        wops += 2 * __popc(ab);
        uint32_t key = 0xffffffffu;
#pragma unroll
        for (int j = 0; j < kRPL; j++)
          if ((ab >> j) & 1) key = min(key, ((uint32_t)__popcll(P & ~t.r[j]) << 8) | (32 * j + lane));
        key = __reduce_min_sync(kFull, key);
        if ((key >> 8) == 0) goto backtrack;  // an X row covers P: nothing maximal below
        VP = P & ~bcast_row(t, key & 0xff);
        fresh = false;
        if (__popcll(VP) >= 4) {
          uint32_t a[kRPL];
#pragma unroll
          for (int j = 0; j < kRPL; j++) a[j] = __ballot_sync(kFull, (ab >> j) & 1);
          const uint64_t done = t1_children(c.P, sm, ta, P, VP, a[0], a[1], a[2], a[3], rsize, s1, s2);
          VP &= ~done;
          nodes += __popcll(done);
        }
        if (level == 0 && c.sharing && hungry(c)) {  // as in the general tier
          const unsigned long long ts = now();
          if (!spawn_outer_gen(c)) {
            if (lane == 0) {
              ta->fP[0] = P;
              ta->fVP[0] = VP;
              ta->frs[0] = rsize;
              ta->fs1[0] = s1;
              ta->fs2[0] = s2;
            }
            ta->fab[0][lane] = (uint8_t)ab;
            __syncwarp();
            t1_spawn(c, t, 1);
            VP = ta->fVP[0];
          }
          if (lane == 0) sm->cyc[kCycSpawn] += now() - ts;
        }
      }
    }
    {
      const uint64_t cand = P & VP;
      if (cand == 0) goto backtrack;
      const uint32_t q = __ffsll((long long)cand) - 1;
      P &= ~(1ULL << q);
      if (lane == 0) {
        ta->fP[level] = P;
        ta->fVP[level] = VP;
        ta->frs[level] = rsize;
        ta->fs1[level] = s1;
        ta->fs2[level] = s2;
      }
      ta->fab[level][lane] = (uint8_t)ab;
      uint64_t P2 = P & bcast_row(t, q);
      uint64_t n1 = s1 + __shfl_sync(kFull, q < 32 ? t.h1a : t.h1b, q & 31);
      uint64_t n2 = s2 + __shfl_sync(kFull, q < 32 ? t.h2a : t.h2b, q & 31);
      uint32_t rs = rsize + 1;
      uint64_t M = 1ULL << q;
      if (expand_r && __popcll(P2) > 1) {
        wops += 2 * (((P2 >> lane) & 1) + ((P2 >> (lane + 32)) & 1));
        const bool e0 = ((P2 >> lane) & 1) && __popcll(P2 & ~t.r[0]) == 1;
        const bool e1 = ((P2 >> (lane + 32)) & 1) && __popcll(P2 & ~t.r[1]) == 1;
        const uint64_t E = (uint64_t)__ballot_sync(kFull, e0) | ((uint64_t)__ballot_sync(kFull, e1) << 32);
        if (E) {
          P2 &= ~E;
          M |= E;
          rs += __popcll(E);
          n1 += warp_sum_u64((e0 ? t.h1a : 0) + (e1 ? t.h1b : 0));
          n2 += warp_sum_u64((e0 ? t.h2a : 0) + (e1 ? t.h2b : 0));
        }
      }
      uint32_t ab2 = 0;
#pragma unroll
      for (int j = 0; j < kRPL; j++)
        if (((ab >> j) & 1) && (t.r[j] & M) == M) ab2 |= 1u << j;
      wops += __popc(ab) + (lane == 0 ? 1 : 0);
      // A child with <= 32 columns and <= 32 active rows drops to the 32-bit
      // tier: rows compressed to the child's columns and gathered, columns
      // first, through the warp's exchange buffer.
      // X rows with no bit on the child's candidates never matter below a
      // child that has candidates (a pivot among them leaves VP = P, and they
      // drop out at the next step), so the handoff leaves them out
      uint32_t ab3 = ab2;
      if (P2) {
#pragma unroll
        for (int j = 0; j < kRPL; j++) {
          const uint32_t idx = 32 * j + lane;
          const bool isc = idx < 64 && ((P2 >> idx) & 1);
          if (!isc && (t.r[j] & P2) == 0) ab3 &= ~(1u << j);
        }
      }
      const uint32_t nact = __reduce_add_sync(kFull, __popc(ab3));
      if (__popcll(P2) <= 32 && nact <= 32) {
        const uint32_t pc2 = __popcll(P2);
        const CPlan plan = compress_plan(P2);
        uint32_t base = pc2;
#pragma unroll
        for (int j = 0; j < kRPL; j++) {
          const uint32_t idx = 32 * j + lane;
          const bool act = (ab3 >> j) & 1;
          const bool isc = idx < 64 && ((P2 >> idx) & 1);
          if (act && isc) {
            const uint32_t k = __popcll(P2 & ((1ULL << idx) - 1));
            sm->xrow[k] = (uint32_t)compress_apply(t.r[j], plan);
            sm->xcv[k] = j == 0 ? t.cva : t.cvb;
            sm->xh1[k] = j == 0 ? t.h1a : t.h1b;
            sm->xh2[k] = j == 0 ? t.h2a : t.h2b;
          }
          const bool isx = act && !isc;
          const uint32_t bal = __ballot_sync(kFull, isx);
          if (isx) sm->xrow[base + __popc(bal & lanemask_lt())] = (uint32_t)compress_apply(t.r[j], plan);
          base += __popc(bal);
        }
        __syncwarp();
        T0 t0;
        t0.row = lane < nact ? sm->xrow[lane] : 0;
        t0.cv = lane < pc2 ? sm->xcv[lane] : 0;
        t0.h1 = lane < pc2 ? sm->xh1[lane] : 0;
        t0.h2 = lane < pc2 ? sm->xh2[lane] : 0;
        if (lane == 0) sm->t1_level = level;
        __syncwarp();
        const unsigned long long tn = now(), spn = sm->cyc[kCycSpawn];
        t0_run(c, t0, pc2, nact, rs, n1, n2);
        if (lane == 0) {
          // the child's cycles go to the 32-bit tier (t1_solve adds the whole
          // span to the 64-bit tier afterwards)
          const unsigned long long dt = (now() - tn) - (sm->cyc[kCycSpawn] - spn);
          sm->cyc[kCycT0] += dt;
          sm->cyc[kCycReg] -= dt;
        }
        // the child may have exposed open candidates of this level
        VP = ta->fVP[level];
        // While the child ran, the levels above it were exposed only through
        // the child's own checks; offer them here as well.
        if (c.sharing && ++tick >= 4) {
          tick = 0;
          if (hungry(c)) {
            const unsigned long long ts = now();
            if (!spawn_outer_gen(c)) t1_spawn(c, t, level + 1);
            if (lane == 0) sm->cyc[kCycSpawn] += now() - ts;
            VP = ta->fVP[level];
          }
        }
        continue;  // next candidate at this level
      }
      level++;
      P = P2;
      VP = 0;
      rsize = rs;
      s1 = n1;
      s2 = n2;
      ab = ab2;
      fresh = true;
      if (c.sharing && ++tick >= 64) {
        tick = 0;
        if (hungry(c)) {
          const unsigned long long t0 = now();
          if (!spawn_outer_gen(c)) t1_spawn(c, t, level);
          if (lane == 0) sm->cyc[kCycSpawn] += now() - t0;
        }
      }
      continue;
    }
  backtrack:
    if (level == 0) break;
    level--;
    P = ta->fP[level];
    VP = ta->fVP[level];
    rsize = ta->frs[level];
    s1 = ta->fs1[level];
    s2 = ta->fs2[level];
    ab = ta->fab[level][lane];
    fresh = false;
  }
  wops = warp_sum_u64(wops);
  if (lane == 0) {
    sm->nodes += nodes;
    sm->wops += wops;
    sm->nest &= ~kNestT1;
  }
  __syncwarp();
  maybe_flush(c);
}

__device__ __forceinline__ void t1_solve(const Ctx &c, const T1 &t, uint32_t pc, uint32_t nrows, uint32_t rsize0,
                                         uint64_t s10, uint64_t s20) {
  const unsigned long long t0 = now(), sp0 = c.sm->cyc[kCycSpawn];
  t1_solve_body(c, t, pc, nrows, rsize0, s10, s20);
  if (c.lane == 0) c.sm->cyc[kCycReg] += (now() - t0) - (c.sm->cyc[kCycSpawn] - sp0);
}

// a register-tier record (W == 1) in this warp's own slab
__device__ void reg_from_local(const Ctx &c, const char *rec) {
  const TaskHdr *h = (const TaskHdr *)rec;
  const uint32_t pc = h->pc, nrows = h->nrows, rsize = h->rsize;
  const uint64_t s1 = h->s1, s2 = h->s2;
  if (pc <= 32 && nrows <= 32) {
    T0 t0;
    t0_load<false>(c, rec, t0, pc, nrows);
    __syncwarp();
    t0_solve(c, t0, pc, nrows, rsize, s1, s2);
    return;
  }
  T1 t;
  t1_load<false>(c, rec, t, pc, nrows);
  __syncwarp();
  t1_solve(c, t, pc, nrows, rsize, s1, s2);
}

// --------------------------------------------------------- general tier

// Child of candidate q at a general-tier level (record rec_l) as a task
// record in `out`: columns = Pbase & row(q), rows = active rows holding bit q
// (and all of R' when the level's list is inherited), compressed to the child
// columns.  Returns false when the record would exceed max_bytes, or, for a
// pool record (to_pool), when a warp's slab could not lay it out for the
// general tier.
__device__ bool gen_materialize(const Ctx &c, const Gen &G, const uint64_t *rec_l, uint32_t q,
                                const uint64_t *Pbase, uint64_t max_bytes, bool to_pool, char *out) {
  const uint32_t lane = c.lane, W = G.W;
  if (W > 64) return false;  // the child's column mask lives in rowbuf (64 words)
  uint64_t *CP = c.sm->rowbuf;
  const uint64_t *rowq = G.rows + (uint64_t)q * W;
  uint32_t pc = 0;
  for (uint32_t w = lane; w < W; w += 32) {
    const uint64_t v = Pbase[w] & rowq[w];
    CP[w] = v;
    pc += __popcll(v);
  }
  pc = __reduce_add_sync(kFull, pc);
  __syncwarp();
  const uint32_t Wn = (pc + 63) / 64;
  const uint64_t m0 = rec_l[3 * W], m1 = rec_l[3 * W + 1];
  const uint32_t aoff = (uint32_t)m0, alen = (uint32_t)(m0 >> 32);
  const bool lazy = (m1 >> 63) != 0;
  const uint64_t *R = rec_l + 2 * W;
  const uint32_t wq = q >> 6;
  const uint64_t bq = 1ULL << (q & 63);
  auto keep_row = [&](uint32_t i) -> bool {
    const uint64_t *row = G.rows + (uint64_t)i * W;
    if (!(row[wq] & bq)) return false;
    if (lazy)
      for (uint32_t w = 0; w < W; w++)
        if ((R[w] & row[w]) != R[w]) return false;
    return true;
  };
  auto is_col = [&](uint32_t i) -> bool { return i < G.pc && ((CP[i >> 6] >> (i & 63)) & 1); };
  // X rows empty on the child's columns are left out when it has columns
  auto hits = [&](uint32_t i) -> bool {
    if (pc == 0) return true;
    const uint64_t *row = G.rows + (uint64_t)i * W;
    for (uint32_t w = 0; w < W; w++)
      if (row[w] & CP[w]) return true;
    return false;
  };
  if (task_bytes(pc, pc, Wn) > max_bytes) return false;
  // the plans depend on the columns alone: one word a lane, once for the task
  for (uint32_t w = lane; w < W; w += 32) G.plans[w] = compress_plan(CP[w]);
  __syncwarp();
  uint32_t *colv = (uint32_t *)(out + kHdr);
  uint64_t *rows = (uint64_t *)(out + kHdr + align8(4ULL * pc));
  // child columns: parent candidate rows i < pc with CP bit i, in order
  for (uint32_t i = lane; i < G.pc; i += 32) {
    if (is_col(i)) {
      uint32_t k = 0;
      for (uint32_t w = 0; w < (i >> 6); w++) k += __popcll(CP[w]);
      k += __popcll(CP[i >> 6] & ((1ULL << (i & 63)) - 1));
      colv[k] = G.colv[i];
      compress_row(G.rows + (uint64_t)i * W, G.plans, W, rows + (uint64_t)k * Wn);
    }
  }
  uint32_t pos = pc;
  for (uint32_t base = 0; base < alen; base += 32) {
    const uint32_t t = base + lane;
    bool x = false;
    uint32_t i = 0;
    if (t < alen) {
      i = aoff == kIdent ? t : G.alist[aoff + t];
      x = !is_col(i) && keep_row(i) && hits(i);
    }
    const uint32_t bal = __ballot_sync(kFull, x);
    if (task_bytes(pc, pos + __popc(bal), Wn) > max_bytes) return false;
    if (x) compress_row(G.rows + (uint64_t)i * W, G.plans, W, rows + (uint64_t)(pos + __popc(bal & lanemask_lt())) * Wn);
    pos += __popc(bal);
  }
  const uint32_t nrows = pos;
  if (to_pool && layout_for(pc, pc, nrows, Wn).need > c.slab_bytes) return false;
  if (lane == 0) {
    TaskHdr *h = (TaskHdr *)out;
    h->pc = pc;
    h->nrows = nrows;
    h->W = Wn;
    h->rsize = ((uint32_t)(m1 >> 32) + 1) & 0x7fffffffu;
    h->s1 = rec_l[3 * W + 2] + G.h1s[q];
    h->s2 = rec_l[3 * W + 3] + G.h2s[q];
    h->slot = c.sm->slot;
  }
  __syncwarp();
  return true;
}

__device__ bool gen_spawn(const Ctx &c, const Gen &G, int level) {
  const uint32_t W = G.W, lane = c.lane;
  const uint64_t LREC = 3ULL * W + 4;
  int l = -1;
  for (int k = 0; k < level && l < 0; k++) {
    const uint64_t *rec = G.stack + (uint64_t)k * LREC;
    bool any = false;
    uint32_t pc = 0;
    for (uint32_t w = lane; w < W; w += 32) {
      any |= (rec[w] & rec[W + w]) != 0;
      pc += __popcll(rec[w]);
    }
    pc = __reduce_add_sync(kFull, pc);
    if (__any_sync(kFull, any) && pc + 1 >= c.P->share_bound) l = k;
  }
  if (l < 0) return false;
  uint64_t *rec = G.stack + (uint64_t)l * LREC;
  uint64_t *Pl = rec, *VPl = rec + W;
  // scratch record past the deepest level holds Pbase
  uint64_t *Pbase = G.stack + (uint64_t)(G.pc + 2) * LREC;
  // highest open candidate first (see t0_spawn)
  uint32_t spawned = 0;
  for (int wq = (int)W - 1; wq >= 0 && spawned < 256; wq--) {
    for (;;) {
      const uint64_t open = Pl[wq] & VPl[wq];
      if (!open) break;
      const uint32_t q = wq * 64 + (63 - __clzll((long long)open));
      uint32_t blk;
      if (!pool_alloc(c, &blk)) return spawned > 0;
      for (uint32_t w = lane; w < W; w += 32) {
        const uint64_t below = (int)w < wq ? ~0ULL : ((int)w == wq ? ((1ULL << (q & 63)) - 1) : 0);
        Pbase[w] = Pl[w] & ~(VPl[w] & below);
      }
      __syncwarp();
      const bool ok = gen_materialize(c, G, rec, q, Pbase, c.P->block_bytes, true, pool_block(*c.P, blk));
      if (!ok) {
        pool_free(c, blk);
        return spawned > 0;
      }
      pool_publish(c, blk);
      if (lane == 0) VPl[wq] &= ~(1ULL << (q & 63));
      __syncwarp();
      spawned++;
    }
  }
  return spawned > 0;
}

// Solve a general-tier ego network laid out in the slab.
__device__ __noinline__ void gen_solve_body(Ctx c, Gen G, uint32_t rsize0, uint64_t s10, uint64_t s20) {
  const uint32_t lane = c.lane, W = G.W;
  WarpSmem *sm = c.sm;
  const uint64_t LREC = 3ULL * W + 4;
  uint64_t *stack = G.stack;
  uint32_t *alist = G.alist;
  const uint64_t *rows = G.rows;
  char *local = c.slab + c.slab_bytes - kLocalRec;  // inside kTail, after the T1Area
  unsigned long long nodes = 0, wops = 0;
  if (lane == 0) {
    sm->gen = G;
    sm->nest |= kNestGen;
  }
  for (uint32_t w = lane; w < W; w += 32) {
    const uint32_t lo = w * 64;
    stack[w] = (G.pc - lo >= 64) ? ~0ULL : ((1ULL << (G.pc - lo)) - 1);
    stack[W + w] = 0;
    stack[2 * W + w] = 0;
  }
  if (lane == 0) {
    uint64_t *m = stack + 3 * W;
    m[0] = (uint64_t)kIdent | ((uint64_t)G.nrows << 32);
    m[1] = (uint64_t)(rsize0 & 0x7fffffffu) << 32;  // a root vertex starts at -1
    m[2] = s10;
    m[3] = s20;
  }
  __syncwarp();
  int level = 0;
  bool fresh = true;
  uint32_t tick = 0;
  for (;;) {
    uint64_t *rec = stack + (uint64_t)level * LREC;
    uint64_t *Pv = rec, *VP = rec + W, *R = rec + 2 * W;
    const uint64_t m0 = rec[3 * W], m1 = rec[3 * W + 1];
    const uint32_t aoff = (uint32_t)m0, alen = (uint32_t)(m0 >> 32);
    const uint32_t atop = (uint32_t)m1, rsize = (uint32_t)(m1 >> 32) & 0x7fffffffu;
    const bool lazy = (m1 >> 63) != 0;
    if (fresh) {
      nodes++;
      uint32_t pcnt = 0;
      for (uint32_t w = lane; w < W; w += 32) pcnt += __popcll(Pv[w]);
      pcnt = __reduce_add_sync(kFull, pcnt);
      if (pcnt == 0) {
        bool blocked;
        if (!lazy) {
          blocked = alen > 0;
        } else {
          bool hit = false;
          for (uint32_t base = 0; base < alen && !hit; base += 32) {
            const uint32_t t = base + lane;
            bool h = false;
            if (t < alen) {
              const uint32_t i = aoff == kIdent ? t : alist[aoff + t];
              const uint64_t *row = rows + (uint64_t)i * W;
              h = true;
              for (uint32_t w = 0; w < W && h; w++) h = (R[w] & ~row[w]) == 0;
            }
            hit = __any_sync(kFull, h);
          }
          blocked = hit;
        }
        if (!blocked && lane == 0) emit(c, (rsize + 2) & 0x7fffffffu, rec[3 * W + 2], rec[3 * W + 3]);
        fresh = false;
        if (level == 0) break;
        level--;
        continue;
      }
      uint32_t best_c = 0xffffffffu, best_t = 0xffffffffu;
      for (uint32_t base = 0; base < alen; base += 32) {
        const uint32_t t = base + lane;
        if (t < alen) {
          const uint32_t i = aoff == kIdent ? t : alist[aoff + t];
          const uint64_t *row = rows + (uint64_t)i * W;
          bool ok = true;
          if (lazy)
            for (uint32_t w = 0; w < W && ok; w++) ok = (R[w] & ~row[w]) == 0;
          if (ok) {
            uint32_t cnt = 0;
            wops += 2 * W;
            for (uint32_t w = 0; w < W; w++) cnt += __popcll(Pv[w] & ~row[w]);
            if (cnt < best_c) {
              best_c = cnt;
              best_t = t;
            }
          }
        }
        if (__any_sync(kFull, best_c == 0)) break;
      }
      const uint32_t minc = __reduce_min_sync(kFull, best_c);
      if (minc == 0 || minc == 0xffffffffu) {
        fresh = false;
        if (level == 0) break;
        level--;
        continue;
      }
      const uint32_t tmin = __reduce_min_sync(kFull, best_c == minc ? best_t : 0xffffffffu);
      const uint32_t piv = aoff == kIdent ? tmin : alist[aoff + tmin];
      const uint64_t *prow = rows + (uint64_t)piv * W;
      for (uint32_t w = lane; w < W; w += 32) VP[w] = Pv[w] & ~prow[w];
      __syncwarp();
      fresh = false;
      // idle warps wait for the top of this subproblem's tree: offer it before
      // the first child, not after eight
      if (level == 0 && c.sharing && hungry(c)) {
        const unsigned long long ts = now();
        gen_spawn(c, G, 1);
        if (lane == 0) sm->cyc[kCycSpawn] += now() - ts;
      }
      continue;
    }
    uint32_t q = 0xffffffffu;
    for (uint32_t wb = 0; wb < W; wb += 32) {
      const uint32_t w = wb + lane;
      const uint64_t val = w < W ? (Pv[w] & VP[w]) : 0;
      const uint32_t bal = __ballot_sync(kFull, val != 0);
      if (bal) {
        const uint32_t src = __ffs(bal) - 1;
        const uint64_t vv = __shfl_sync(kFull, val, src);
        q = (wb + src) * 64 + (__ffsll((long long)vv) - 1);
        break;
      }
    }
    if (q == 0xffffffffu) {
      if (level == 0) break;
      level--;
      continue;
    }
    const uint32_t wq = q >> 6;
    const uint64_t bq = 1ULL << (q & 63);
    if (lane == 0) Pv[wq] &= ~bq;
    __syncwarp();
    uint64_t *crec = rec + LREC;
    uint64_t *CP = crec, *CE = crec + W, *CR = crec + 2 * W;
    const uint64_t *rowq = rows + (uint64_t)q * W;
    uint32_t cpc = 0;
    for (uint32_t w = lane; w < W; w += 32) {
      const uint64_t cp = Pv[w] & rowq[w];
      CP[w] = cp;
      CR[w] = R[w] | (w == wq ? bq : 0);
      CE[w] = 0;
      cpc += __popcll(cp);
    }
    cpc = __reduce_add_sync(kFull, cpc);
    __syncwarp();
    // a child small enough for the register tiers leaves the general tier here
    if (cpc <= 64 && cpc > 0) {
      uint32_t ccount = 0;
      for (uint32_t base = 0; base < alen; base += 32) {
        const uint32_t t = base + lane;
        bool keep = false;
        if (t < alen) {
          const uint32_t i = aoff == kIdent ? t : alist[aoff + t];
          const uint64_t *row = rows + (uint64_t)i * W;
          keep = (row[wq] & bq) != 0;
          if (lazy)
            for (uint32_t w = 0; w < W && keep; w++) keep = (R[w] & row[w]) == R[w];
          // an X row empty on the child's columns is left out of the record
          if (keep && !(i < G.pc && ((CP[i >> 6] >> (i & 63)) & 1))) {
            bool hit = false;
            for (uint32_t w = 0; w < W && !hit; w++) hit = (row[w] & CP[w]) != 0;
            keep = hit;
          }
        }
        ccount += __popc(__ballot_sync(kFull, keep));
      }
      if (ccount <= kT1Rows && gen_materialize(c, G, rec, q, Pv, kLocalRec, false, local)) {
        if (lane == 0) sm->gen_level = level;
        __syncwarp();
        const unsigned long long t0 = now(), sp0 = sm->cyc[kCycSpawn];
        reg_from_local(c, local);
        // the register-tier time is booked there; keep it out of this phase
        if (lane == 0) sm->cyc[kCycGen] -= (now() - t0) - (sm->cyc[kCycSpawn] - sp0);
        if (c.sharing && ++tick >= 8) {
          tick = 0;
          if (hungry(c)) {
            const unsigned long long ts = now();
            gen_spawn(c, G, level + 1);
            if (lane == 0) sm->cyc[kCycSpawn] += now() - ts;
          }
        }
        continue;  // next candidate at this level
      }
    }
    uint32_t rs = rsize + 1;
    uint64_t t1 = rec[3 * W + 2] + G.h1s[q], t2 = rec[3 * W + 3] + G.h2s[q];
    uint32_t nE = 0;
    if (c.P->expand_r && cpc > 1) {
      uint64_t e1 = 0, e2 = 0;
      uint32_t ne = 0;
      for (uint32_t base = 0; base < G.pc; base += 32) {
        const uint32_t i = base + lane;
        bool e = false;
        if (i < G.pc && ((CP[i >> 6] >> (i & 63)) & 1)) {
          const uint64_t *ri = rows + (uint64_t)i * W;
          uint32_t cc = 0;
          for (uint32_t w = 0; w < W && cc <= 1; w++) cc += __popcll(CP[w] & ~ri[w]);
          e = (cc == 1);
        }
        const uint32_t bal = __ballot_sync(kFull, e);
        if (bal) {
          if (lane == 0) CE[base >> 6] |= (uint64_t)bal << (base & 32);
          if (e) {
            e1 += G.h1s[i];
            e2 += G.h2s[i];
            ne++;
          }
        }
      }
      nE = __reduce_add_sync(kFull, ne);
      if (nE) {
        e1 = warp_sum_u64(e1);
        e2 = warp_sum_u64(e2);
        __syncwarp();
        for (uint32_t w = lane; w < W; w += 32) {
          const uint64_t ew = CE[w];
          CP[w] &= ~ew;
          CR[w] |= ew;
        }
        rs += nE;
        t1 += e1;
        t2 += e2;
      }
    }
    __syncwarp();
    uint32_t caoff, calen, catop;
    bool clazy;
    if ((uint64_t)atop + alen <= G.alist_cap) {
      uint32_t n2 = 0;
      const bool single = !lazy && nE == 0;
      const bool child_has_p = cpc > nE;  // X rows empty on P' matter only at a leaf
      for (uint32_t base = 0; base < alen; base += 32) {
        const uint32_t t = base + lane;
        bool keep = false;
        uint32_t i = 0;
        if (t < alen) {
          wops += single ? 1 : W;
          i = aoff == kIdent ? t : alist[aoff + t];
          const uint64_t *row = rows + (uint64_t)i * W;
          keep = (row[wq] & bq) != 0;
          if (!single) {
            const uint64_t *need = lazy ? CR : CE;
            for (uint32_t w = 0; w < W && keep; w++) keep = (row[w] & need[w]) == need[w];
          }
          if (keep && child_has_p && !(i < G.pc && ((CP[i >> 6] >> (i & 63)) & 1))) {
            bool hit = false;
            for (uint32_t w = 0; w < W && !hit; w++) hit = (row[w] & CP[w]) != 0;
            keep = hit;
          }
        }
        const uint32_t bal = __ballot_sync(kFull, keep);
        if (keep) alist[atop + n2 + __popc(bal & lanemask_lt())] = i;
        n2 += __popc(bal);
      }
      caoff = atop;
      calen = n2;
      catop = atop + n2;
      clazy = false;
    } else {
      caoff = aoff;
      calen = alen;
      catop = atop;
      clazy = true;
    }
    if (lane == 0) {
      crec[3 * W] = (uint64_t)caoff | ((uint64_t)calen << 32);
      crec[3 * W + 1] = (uint64_t)catop | ((uint64_t)(rs & 0x7fffffffu) << 32) | (clazy ? (1ULL << 63) : 0);
      crec[3 * W + 2] = t1;
      crec[3 * W + 3] = t2;
    }
    __syncwarp();
    level++;
    fresh = true;
    if (c.sharing && ++tick >= 8) {
      tick = 0;
      if (hungry(c)) {
        const unsigned long long ts = now();
        gen_spawn(c, G, level);
        if (lane == 0) sm->cyc[kCycSpawn] += now() - ts;
      }
    }
  }
  wops = warp_sum_u64(wops);
  if (lane == 0) {
    sm->nodes += nodes;
    sm->wops += wops;
    sm->nest &= ~kNestGen;
  }
  __syncwarp();
  maybe_flush(c);
}

__device__ __noinline__ bool spawn_outer_gen(Ctx c) {
  if (!(c.sm->nest & kNestGen)) return false;
  const Gen G = c.sm->gen;
  return gen_spawn(c, G, c.sm->gen_level + 1);
}

__device__ __noinline__ bool spawn_outer_t1(Ctx c) {
  WarpSmem *sm = c.sm;
  T1Area *ta = c.ta;
  if (!(sm->nest & kNestT1)) return false;
  if (t1_open_level(c, sm->t1_level + 1) < 0) return false;  // before loading rows
  T1 t;
#pragma unroll
  for (int j = 0; j < kRPL; j++) t.r[j] = ta->t1rows[32 * j + c.lane];
  t.cva = ta->t1cv[c.lane];
  t.cvb = ta->t1cv[c.lane + 32];
  t1_hashes(c, t, sm->t1_pc);
  return t1_spawn(c, t, sm->t1_level + 1);
}

__device__ __noinline__ bool t0_share(Ctx c, const T0 t, int level) {
  const unsigned long long ts = now();
  const bool any = spawn_outer_gen(c) || spawn_outer_t1(c) || t0_spawn(c, t, level);
  if (c.lane == 0) c.sm->cyc[kCycSpawn] += now() - ts;
  return any;
}

__device__ __forceinline__ void gen_solve(const Ctx &c, const Gen &G, uint32_t rsize0, uint64_t s10, uint64_t s20) {
  const unsigned long long t0 = now(), sp0 = c.sm->cyc[kCycSpawn];
  gen_solve_body(c, G, rsize0, s10, s20);
  if (c.lane == 0) c.sm->cyc[kCycGen] += (now() - t0) - (c.sm->cyc[kCycSpawn] - sp0);
}

// ------------------------------------------------------------ root build

// Which of four sorted values per lane occur in the sorted list b[0..n), as
// four branchless binary searches in step: n is warp-uniform, so every lane
// runs the same trip count and the four dependent load chains overlap.
__device__ __forceinline__ void contains4(const uint32_t *b, uint32_t n, const uint32_t (&val)[4], bool (&hit)[4]) {
  uint32_t pos[4] = {0, 0, 0, 0};
  uint32_t len = n;
  while (len > 1) {
    const uint32_t half = len >> 1;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (__ldg(b + pos[k] + half - 1) < val[k]) pos[k] += half;
    len -= half;
  }
#pragma unroll
  for (int k = 0; k < 4; k++) hit[k] = n && __ldg(b + pos[k]) == val[k];
}

// The shorter of two adjacency lists in (a, da), the longer in (b, db).
__device__ __forceinline__ void shorter_first(const DevGraph &g, uint32_t v0, uint32_t v1, const uint32_t *&a,
                                              uint32_t &da, const uint32_t *&b, uint32_t &db) {
  a = g.adj + g.off[v0];
  b = g.adj + g.off[v1];
  da = g.off[v0 + 1] - g.off[v0];
  db = g.off[v1 + 1] - g.off[v1];
  if (da > db) {
    const uint32_t *t = a;
    a = b;
    b = t;
    const uint32_t td = da;
    da = db;
    db = td;
  }
}

// How many elements of the sorted list b[0..n) to look at for every value <=
// vmax to be among them (rounded up), and in *sure how many certainly are
// <= vmax.  The warp probes 32 places at a time, eight times further apart
// each time all of them are still below.
__device__ __forceinline__ uint32_t window_for(const uint32_t *b, uint32_t n, uint32_t vmax, uint32_t *sure) {
  const uint32_t lane = lane_id();
  uint32_t from = 0, stride = 32;
  for (;;) {
    const uint32_t at = from + stride * (lane + 1) - 1;
    const uint32_t below = __popc(__ballot_sync(kFull, at < n && __ldg(b + at) <= vmax));
    from += stride * below;
    if (below < 32) {
      *sure = from;
      return min(n, from + stride);
    }
    stride = min(stride * 8, 1u << 24);
  }
}

// C = N(v0) & N(v1) (sorted) into cand[]; |C|, or 0xffffffff beyond cap.
// Bound by the latency of the searches in the longer list, so four of the
// shorter list's 32-element groups are searched at a time, and where the lists
// are long and of like lengths only in the part of the longer one that the
// groups span (a few cache lines instead of the whole list).  Lists of up to 512
// are found faster whole: G(12000, mean degree 150) 2.99 ms instead of 3.14,
// G(4000, 400) 31.9 instead of 33.0 (B200).
__device__ uint32_t intersect(const DevGraph &g, uint32_t v0, uint32_t v1, uint32_t *cand, uint64_t cap) {
  const uint32_t lane = lane_id();
  const uint32_t *a, *b;
  uint32_t da, db;
  shorter_first(g, v0, v1, a, da, b, db);
  uint32_t nc = 0;
  const bool windows = da > 128 && db > 512 && db / 64 < da;
  uint32_t done = 0;  // elements of b below every value still to come
  for (uint32_t base = 0; base < da; base += 128) {
    uint32_t val[4];
    bool hit[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t t = base + 32 * k + lane;
      val[k] = t < da ? __ldg(a + t) : 0;
    }
    if (windows) {
      uint32_t sure = 0;
      const uint32_t n = window_for(b + done, db - done, __ldg(a + min(base + 127, da - 1)), &sure);
      contains4(b + done, n, val, hit);
      done += sure;
    } else {
      contains4(b, db, val, hit);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      hit[k] = hit[k] && base + 32 * k + lane < da;
      const uint32_t bal = __ballot_sync(kFull, hit[k]);
      if (nc + __popc(bal) > cap) return 0xffffffffu;
      if (hit[k]) cand[nc + __popc(bal & lanemask_lt())] = val[k];
      nc += __popc(bal);
    }
  }
  __syncwarp();
  return nc;
}

// |N(v0) & N(v1)| and how many of those lie below v1, without storing them:
// sizes the large-scratch pass for a root whose ego network overflowed the slab.
__device__ void intersect_count(const DevGraph &g, uint32_t v0, uint32_t v1, uint32_t *nc_out, uint32_t *nx_out) {
  const uint32_t lane = lane_id();
  const uint32_t *a, *b;
  uint32_t da, db;
  shorter_first(g, v0, v1, a, da, b, db);
  uint32_t nc = 0, nx = 0;
  for (uint32_t base = 0; base < da; base += 32) {
    const uint32_t t = base + lane;
    const uint32_t val = t < da ? __ldg(a + t) : 0;
    const bool hit = t < da && contains_u32(b, db, val);
    nc += __popc(__ballot_sync(kFull, hit));
    nx += __popc(__ballot_sync(kFull, hit && val < v1));
  }
  *nc_out = nc;
  *nx_out = nx;
}

// Scratch of the root build: the candidates P and the rows in flight.  It
// overlays per-warp state that only a running solve uses.
struct BuildScratch {
  uint32_t P[256];     // candidates, padded to a power of two with 0xffffffff (p <= 256)
  uint32_t obase[32];  // non-empty row o of the batch: element t of the flattened lists is adj[obase[o] + t]
  uint32_t orow[32];   // its row in the batch
};
static_assert(offsetof(WarpSmem, t0_s1) - offsetof(WarpSmem, t0f) >= sizeof(BuildScratch),
              "the build scratch fits over the 32-bit tier's frames and exchange buffer");

// First index whose value is >= key in a sorted list in the warp's slab
// (written by this kernel, so read with ordinary loads).
__device__ __forceinline__ uint32_t slab_lower_bound(const uint32_t *a, uint32_t n, uint32_t key) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// The only j < p at which P[j] can be y, over the candidates in shared memory
// (padded) or in the slab.
__device__ __forceinline__ uint32_t find_cand(const BuildScratch *bs, uint32_t top, const uint32_t *Pl, uint32_t p,
                                              uint32_t y) {
  if (top == 0) return slab_lower_bound(Pl, p, y);
  uint32_t pos = 0;
  for (uint32_t s = top; s; s >>= 1)
    if (bs->P[pos + s - 1] < y) pos += s;
  return pos;
}

// Ego bitmap rows (candidate rows, then X rows with a candidate neighbour), up
// to 4096 candidates.
//
// A row of member u is N(u) & P.  One row at a time leaves the warp waiting on
// two binary searches and a few loads for each row, so rows are built in
// batches of up to 32 (64 words of bitmap): every lane finds the part of one
// member's list that spans P -- most X members have no neighbour above v1 and
// end there -- and the parts are read as one flattened list, 32 neighbouring
// elements at a time whatever the rows' lengths.  An element's row comes from
// the row starts inside the window (one OR-reduction), its column from a
// search in shared memory.  A part much longer than P is probed for the
// candidates instead (a member's part is found from the end of its list: it
// has few neighbours after the root's vertices).  Up to 64 candidates, their own rows come from testing
// every pair once, in the shorter of the two lists, a pair a lane: late
// candidates are hubs whose lists between two candidates are long (Chung-Lu
// 10^6 enumeration 9.3 -> 7.3 ms).
// Measured (B200), against a row at a time: Chung-Lu 10^4 1.07 -> 0.28 ms (the
// longest root 1.9e6 -> 0.28e6 cycles); planted cliques of 40-200 vertices in
// 10^5, edge roots only (99 % of the time is this build) 297 -> 202 ms.
__device__ uint32_t build_rows(const DevGraph &g, const uint32_t *cand, uint32_t x, uint32_t p, uint32_t W,
                               uint64_t *rows, WarpSmem *sm) {
  const uint32_t lane = lane_id();
  const uint32_t *Pl = cand + x;
  BuildScratch *bs = (BuildScratch *)sm->t0f;
  uint64_t *acc = sm->rowbuf;  // rows of the batch, W words each
  uint32_t *acc32 = (uint32_t *)acc;
  const uint32_t pmin = Pl[0], pmax = Pl[p - 1];
  // top: first step of the column search, a power of two with 2 * top >= p (0: search the slab)
  uint32_t top = 0;
  if (p <= 256) {
    top = p <= 2 ? 1u : 1u << (31 - __clz(p - 1));
    for (uint32_t i = lane; i < 2 * top; i += 32) bs->P[i] = i < p ? Pl[i] : 0xffffffffu;
  }
  const uint32_t nb = min(32u, 64u / W);
  uint32_t nrows = 0;
  if (W == 1) {
    // candidate rows, a pair of candidates a lane
    uint32_t *Pb = bs->P + 128, *Pn = bs->P + 192;  // list starts and lengths (p <= 64 leaves them free)
    for (uint32_t i = lane; i < 64; i += 32) {
      acc[i] = 0;
      if (i < p) {
        const uint32_t b = g.off[Pl[i]];
        Pb[i] = b;
        Pn[i] = g.off[Pl[i] + 1] - b;
      }
    }
    __syncwarp();
    const uint32_t inv = (1u << 22) / p + 1, pairs = p * (p >> 1);  // t / p == t * inv >> 22 for t < pairs
    for (uint32_t t0 = 0; t0 < pairs; t0 += 32) {
      const uint32_t t = t0 + lane;
      if (t < pairs) {
        const uint32_t o = t * inv >> 22, i = t - o * p;
        uint32_t j = i + o + 1;  // the candidate o + 1 further on, around the end
        if (j >= p) j -= p;
        const bool in_i = Pn[i] <= Pn[j];
        if (contains_u32(g.adj + (in_i ? Pb[i] : Pb[j]), in_i ? Pn[i] : Pn[j], in_i ? bs->P[j] : bs->P[i])) {
          atomicOr(&acc32[2 * i + (j >> 5)], 1u << (j & 31));
          atomicOr(&acc32[2 * j + (i >> 5)], 1u << (i & 31));
        }
      }
    }
    __syncwarp();
    for (uint32_t i = lane; i < p; i += 32) rows[i] = acc[i];
    __syncwarp();
    nrows = p;
  }
  for (uint32_t mb = nrows; mb < p + x; mb += nb) {
    const uint32_t m = mb + lane;
    const bool mine = lane < nb && m < p + x;
    uint32_t lo = 0, len = 0;
    if (mine) {
      const uint32_t u = m < p ? Pl[m] : cand[m - p];
      const uint32_t b = g.off[u], e = g.off[u + 1];
      const uint32_t last = __ldg(g.adj + e - 1);
      if (last >= pmin) {
        // from the end: a member's list has few neighbours after v
        uint32_t at = 1, step = 1;  // the last `at` elements are >= pmin
        while (at < e - b) {
          const uint32_t next = min(at + step, e - b);
          if (__ldg(g.adj + e - next) < pmin) {
            // the first element >= pmin is among the next - at before those
            const uint32_t o = e - next;
            lo = o + lower_bound_u32(g.adj + o, next - at, pmin);
            break;
          }
          at = next;
          step *= 2;
        }
        if (at == e - b) lo = b;
        len = last <= pmax ? e - lo : lower_bound_u32(g.adj + lo, e - lo, pmax + 1);
      }
    }
    for (uint32_t w = lane; w < nb * W; w += 32) acc[w] = 0;
    // probing costs p searches of a warp's lanes, reading the part len / 32 loads.
    // Measured (B200), ms, for 2, 8, 32 times p and never: 1024 core roots of
    // R-MAT 20 27.4, 32.4, 31.7, 30.9, planted cliques of 40-200 vertices 7.15,
    // 7.50, 7.46, 7.38; R-MAT 14, Chung-Lu 10^6 and 300 G(n, p) graphs the same
    const bool probe = len > 8 * p + 64;
    const uint32_t sl = probe ? 0 : len;
    uint32_t incl = sl;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, d);
      if (lane >= (uint32_t)d) incl += y;
    }
    const uint32_t T = __shfl_sync(kFull, incl, 31), first = incl - sl;
    const uint32_t ne = __ballot_sync(kFull, sl != 0);
    if (sl) {
      const uint32_t o = __popc(ne & lanemask_lt());
      bs->obase[o] = lo - first;
      bs->orow[o] = lane;
    }
    __syncwarp();
    // window t0: row starts inside it, and this lane's element and its row
    uint32_t started = 0, heads = 0, row = 0, y = 0;
    auto fetch = [&](uint32_t t0) {
      heads = __reduce_or_sync(kFull, sl && first - t0 < 32 ? 1u << (first - t0) : 0u);
      const uint32_t o = started + __popc(heads & (lanemask_lt() | (1u << lane))) - 1;
      started += __popc(heads);
      row = bs->orow[o];
      y = t0 + lane < T ? __ldg(g.adj + (bs->obase[o] + t0 + lane)) : 0;
    };
    if (T) fetch(0);
    for (uint32_t t0 = 0; t0 < T; t0 += 32) {
      const uint32_t nheads = __popc(heads), yc = y;
      const uint32_t rowkey = row * 2 * W;
      const bool in = t0 + lane < T;
      if (t0 + 32 < T) fetch(t0 + 32);  // the next window's loads run under this one's search
      const uint32_t j = find_cand(bs, top, Pl, p, yc);
      const bool hit = in && j < p && (top ? bs->P[j] : Pl[j]) == yc;
      const uint32_t key = rowkey + (j >> 5);
      const uint32_t bit = 1u << (j & 31);
      uint32_t rem = __ballot_sync(kFull, hit);
      if (__popc(rem) <= 8 || nheads > 2) {
        if (hit) atomicOr(&acc32[key], bit);
      } else {
        // long rows with many hits: neighbouring elements share a word, and
        // atomics on one word would run one after another
        while (rem) {
          const uint32_t l = __ffs(rem) - 1;
          const uint32_t kl = __shfl_sync(kFull, key, l);
          const bool same = hit && key == kl;
          const uint32_t bits = __reduce_or_sync(kFull, same ? bit : 0u);
          if (lane == l) acc32[key] |= bits;
          rem &= ~__ballot_sync(kFull, same);
        }
      }
      __syncwarp();
    }
    for (uint32_t pr = __ballot_sync(kFull, probe); pr; pr &= pr - 1) {
      const uint32_t l = __ffs(pr) - 1;
      const uint32_t *part = g.adj + __shfl_sync(kFull, lo, l);
      const uint32_t n = __shfl_sync(kFull, len, l);
      for (uint32_t base = 0; base < p; base += 32) {
        const uint32_t j = base + lane;
        const uint32_t bal = __ballot_sync(kFull, j < p && contains_u32(part, n, Pl[j]));
        if (lane == 0) acc32[l * 2 * W + (base >> 5)] = bal;
      }
    }
    __syncwarp();
    uint64_t any = 0;
    if (mine)
      for (uint32_t w = 0; w < W; w++) any |= acc[lane * W + w];
    const bool keep = mine && (m < p || any);
    const uint32_t bal = __ballot_sync(kFull, keep);
    if (keep) {
      uint64_t *row = rows + (uint64_t)(nrows + __popc(bal & lanemask_lt())) * W;
      for (uint32_t w = 0; w < W; w++) row[w] = acc[lane * W + w];
    }
    nrows += __popc(bal);
    __syncwarp();
  }
  return nrows;
}

// The same for more than 4096 candidates: one row at a time, probed for the
// candidates.
__device__ uint32_t build_rows_wide(const DevGraph &g, const uint32_t *cand, uint32_t x, uint32_t p, uint32_t W,
                                    uint64_t *rows) {
  const uint32_t lane = lane_id();
  const uint32_t *Pl = cand + x;
  const uint32_t pmin = Pl[0], pmax = Pl[p - 1];
  uint32_t nrows = 0;
  for (uint32_t r = 0; r < p + x; r++) {
    const uint32_t u = r < p ? Pl[r] : cand[r - p];
    const uint32_t *nu = g.adj + g.off[u];
    const uint32_t du = g.off[u + 1] - g.off[u];
    uint64_t *row = rows + (uint64_t)nrows * W;
    uint32_t lo = 0, hi = 0;
    if (lane == 0) {
      lo = lower_bound_u32(nu, du, pmin);
      hi = lower_bound_u32(nu, du, pmax + 1);
    }
    lo = __shfl_sync(kFull, lo, 0);
    hi = __shfl_sync(kFull, hi, 0);
    uint64_t word = 0;
    bool any = false;
    const uint32_t *sl = nu + lo;
    const uint32_t sn = hi - lo;
    for (uint32_t base = 0; base < p; base += 32) {
      const uint32_t j = base + lane;
      const bool hit = j < p && contains_u32(sl, sn, Pl[j]);
      const uint32_t bal = __ballot_sync(kFull, hit);
      any |= bal != 0;
      if (base & 32) {
        word |= (uint64_t)bal << 32;
        if (lane == 0) row[base >> 6] = word;
      } else {
        word = bal;
        if (base + 32 >= p && lane == 0) row[base >> 6] = word;
      }
    }
    __syncwarp();
    if (r < p || any) nrows++;
  }
  return nrows;
}

// Solve an ego network whose rows are in the slab, in the smallest tier that
// holds it.  colv: the candidates' vertex ids; rsize: |R| beyond two vertices.
__device__ __noinline__ void solve_ego(Ctx c, const uint32_t *colv, uint32_t nrows, uint32_t p, uint32_t W,
                                       const Layout &L, uint32_t rsize, uint64_t s1, uint64_t s2) {
  const DevGraph &g = c.P->g;
  const uint64_t *rows = (const uint64_t *)(c.slab + L.rows_off);
  if (p <= 32 && nrows <= 32) {
    T0 t0;
    t0.row = c.lane < nrows ? (uint32_t)rows[c.lane] : 0;
    t0.cv = c.lane < p ? colv[c.lane] : 0;
    t0.h1 = c.lane < p ? g.h1[t0.cv] : 0;
    t0.h2 = c.lane < p ? g.h2[t0.cv] : 0;
    __syncwarp();
    t0_solve(c, t0, p, nrows, rsize, s1, s2);
    return;
  }
  if (W == 1 && nrows <= kT1Rows) {
    T1 t;
#pragma unroll
    for (int j = 0; j < kRPL; j++) {
      const uint32_t idx = 32 * j + c.lane;
      t.r[j] = idx < nrows ? rows[idx] : 0;
    }
    t.cva = c.lane < p ? colv[c.lane] : 0;
    t.cvb = c.lane + 32 < p ? colv[c.lane + 32] : 0;
    t1_hashes(c, t, p);
    __syncwarp();
    t1_solve(c, t, p, nrows, rsize, s1, s2);
    return;
  }
  Gen G;
  G.rows = rows;
  G.colv = colv;
  uint64_t *h1s = (uint64_t *)(c.slab + L.hash_off);
  uint64_t *h2s = h1s + p;
  for (uint32_t j = c.lane; j < p; j += 32) {
    const uint32_t y = colv[j];
    h1s[j] = g.h1[y];
    h2s[j] = g.h2[y];
  }
  G.h1s = h1s;
  G.h2s = h2s;
  G.stack = (uint64_t *)(c.slab + L.stack_off);
  G.plans = (CPlan *)(c.slab + L.plan_off);
  G.alist = (uint32_t *)(c.slab + L.alist_off);
  G.alist_cap = (c.slab_bytes - kTail - L.alist_off) / 4;
  G.pc = p;
  G.nrows = nrows;
  G.W = W;
  __syncwarp();
  gen_solve(c, G, rsize, s1, s2);
}

// Solve root r.  Returns false when the root does not fit this slab.
__device__ bool solve_root(const Ctx &c, uint64_t r) {
  const DevGraph &g = c.P->g;
  const uint32_t v0 = g.root_v0[r], v1 = g.root_v1[r];
  set_slot(c, g.slot ? g.slot[v0] : 0);
  uint32_t *cand = (uint32_t *)c.slab;
  const uint64_t cap = (c.slab_bytes - kTail) / 4;
  const unsigned long long tb0 = now();
  const uint32_t nc = intersect(g, v0, v1, cand, cap);
  if (nc == 0xffffffffu) {
    if (c.lane == 0) c.sm->cyc[kCycBuild] += now() - tb0;
    return false;
  }
  const uint32_t x = slab_lower_bound(cand, nc, v1);
  const uint32_t p = nc - x;
  const uint64_t s1 = g.h1[v0] + g.h1[v1], s2 = g.h2[v0] + g.h2[v1];
  const uint32_t W = (p + 63) / 64;
  const Layout L = layout_for(nc, p, p + x, W);
  if (p > 0 && L.need > c.slab_bytes) {
    if (c.lane == 0) c.sm->cyc[kCycBuild] += now() - tb0;
    return false;
  }
  if (c.P->stats) {
    // algorithmic build bytes: both endpoint lists, then every member's
    // adjacency list and its bitmap row
    uint64_t du = 0;
    if (p > 0)
      for (uint32_t j = c.lane; j < nc; j += 32) du += g.off[cand[j] + 1] - g.off[cand[j]];
    du = warp_sum_u64(du);
    if (c.lane == 0)
      c.sm->bbytes += 4ULL * ((g.off[v0 + 1] - g.off[v0]) + (g.off[v1 + 1] - g.off[v1])) +
                      (p > 0 ? 4ULL * du + 8ULL * W * nc : 0);
  }
  if (p == 0) {
    if (x == 0 && c.lane == 0) emit(c, 2, s1, s2);
    if (c.lane == 0) c.sm->cyc[kCycBuild] += now() - tb0;
    return true;
  }
  uint64_t *rows = (uint64_t *)(c.slab + L.rows_off);
  const uint32_t nrows = W <= 64 ? build_rows(g, cand, x, p, W, rows, c.sm) : build_rows_wide(g, cand, x, p, W, rows);
  __syncwarp();
  if (c.lane == 0) c.sm->cyc[kCycBuild] += now() - tb0;
  solve_ego(c, cand + x, nrows, p, W, L, 0, s1, s2);
  return true;
}

// Vertices solved whole.  Up to kVertexCols later neighbours and kVertexDegree
// neighbours (a hub's members are many warps' work: Chung-Lu 10^6 6.4 ms with
// up to 16384, 5.6 with 4096, 5.8 with 2048, where full R-MAT 14 loses 10 %) a
// vertex's ego network is built once and searched with a pivot;
// from 65 later neighbours on (the general tier) only where at most
// kVertexBranches of them, and at most a quarter, are left to branch on.
// Measured (B200), ms, with all vertices of the G(n, p) graphs first (vertex_pass_for):
//   kVertexCols          64    128    256    512
//   planted 40-200    208.4  120.4    7.5    7.8
//   full R-MAT 14      25.2   18.9   18.8   18.4
//   G(4000, deg 400)   34.0   33.9   35.2   38.7
// kVertexBranches 4, 8, 16, 64: planted 16.4, 12.1, 7.5, 6.4, the others the
// same.  An eighth, a quarter or half of them: planted 8.8, 7.5, 7.5.  Without
// either bound planted 5.6, but G(4000, deg 400) 44.9 and G(1000, deg 200) 11.1
// instead of 5.7.  A vertex turned down has its rows built for nothing: none on
// R-MAT 14 and 15, 0.6 % of the warps' cycles on planted, 0.8 % on R-MAT 18 of
// edge factor 4, 2.1 % on G(1000, 200) and G(4000, 400).
constexpr uint32_t kVertexCols = 256, kVertexDegree = 4096, kVertexBranches = 16;

// Whether val is in each of four sorted lists, searched in step.
__device__ __forceinline__ void contains_each(const uint32_t *const (&list)[4], const uint32_t (&n)[4], uint32_t val,
                                              bool (&hit)[4]) {
  uint32_t pos[4] = {0, 0, 0, 0}, len[4] = {n[0], n[1], n[2], n[3]};
  while (max(max(len[0], len[1]), max(len[2], len[3])) > 1) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t half = len[k] >> 1;
      if (half && __ldg(list[k] + pos[k] + half - 1) < val) pos[k] += half;
      len[k] -= half;
    }
  }
#pragma unroll
  for (int k = 0; k < 4; k++) hit[k] = __ldg(list[k] + pos[k]) == val;
}

// Whether one of the four candidates Pl[0..p) of most neighbours is a pivot that
// leaves at most kVertexBranches of them, and at most a quarter, to branch on.
// Of the vertices with such a pivot, 96 to 100 % have one among these four
// (R-MAT 12 to 18, Chung-Lu 10^6, planted cliques).  A sample of 32 candidates
// turns most others down after one search.
__device__ __noinline__ bool good_pivot(const DevGraph &g, const uint32_t *Pl, uint32_t p) {
  if (p < 4) return false;
  const uint32_t lane = lane_id();
  uint32_t key[kVertexCols / 32];  // neighbours << 8 | candidate, 0: none
#pragma unroll
  for (int k = 0; k < (int)kVertexCols / 32; k++) {
    const uint32_t j = 32 * k + lane;
    key[k] = 0;
    if (j < p) {
      const uint32_t u = __ldg(Pl + j);
      key[k] = min(g.off[u + 1] - g.off[u], 0xffffffu) << 8 | j;
    }
  }
  const uint32_t *list[4];
  uint32_t n[4], hits[4] = {0, 0, 0, 0};
#pragma unroll
  for (int t = 0; t < 4; t++) {
    uint32_t top = 0;
#pragma unroll
    for (int k = 0; k < (int)kVertexCols / 32; k++) top = max(top, key[k]);
    top = __reduce_max_sync(kFull, top);
#pragma unroll
    for (int k = 0; k < (int)kVertexCols / 32; k++)
      if (key[k] == top) key[k] = 0;
    const uint32_t u = __ldg(Pl + (top & 0xff));
    list[t] = g.adj + g.off[u];
    n[t] = g.off[u + 1] - g.off[u];
  }
  bool hit[4];
  contains_each(list, n, __ldg(Pl + lane * p / 32), hit);
  uint32_t best = 0;
#pragma unroll
  for (int t = 0; t < 4; t++) best = max(best, (uint32_t)__popc(__ballot_sync(kFull, hit[t])));
  if (best < 16) return false;
  for (uint32_t base = 0; base < p; base += 32) {
    const uint32_t j = base + lane;
    contains_each(list, n, j < p ? __ldg(Pl + j) : 0, hit);
#pragma unroll
    for (int t = 0; t < 4; t++) hits[t] += __popc(__ballot_sync(kFull, j < p && hit[t]));
  }
  const uint32_t left = p - max(max(hits[0], hits[1]), max(hits[2], hits[3]));
  return left <= kVertexBranches && 4 * left <= p;
}

// Vertex item k of the vertex pass: the cliques whose first vertex (in the
// order) is v.  An edge root (v, w) builds its own ego network out of the
// members' lists, so a member's list is read once for every w it is adjacent
// to; here it is read once for v, and no intersection is needed, since v's
// own list is the ego network's vertex set.  The pivot also skips every w that
// it is adjacent to.  A vertex with many candidates and no good pivot is left
// to the edge pass: its roots are many warps' work.  Returns its solved roots.
// Measured (B200): planted cliques of 40-200 vertices in 10^5 202 -> 8.6 ms,
// Chung-Lu 10^6 15.4 -> 9.7 ms; the root build's share of full R-MAT 14 15 % -> 1 %.
__device__ __noinline__ uint32_t run_vertex(Ctx c, uint64_t k) {
  const EnumParams &P = *c.P;
  const DevGraph &g = P.g;
  // late-peeled vertices first: they are the heavy ones
  const uint32_t singles = c.sm->singles;
  const uint32_t v = k < singles ? c.sm->last - (uint32_t)k : P.vert_list[k - singles];
  const uint32_t r0 = g.root_off[v], r1 = g.root_off[v + 1];
  const uint32_t lo = (uint32_t)max((uint64_t)r0, P.rb), hi = (uint32_t)min((uint64_t)r1, P.re);
  if (lo >= hi) return 0;
  const unsigned long long t0 = now();
  const uint32_t b = g.off[v], d = g.off[v + 1] - b, p = r1 - r0, x = d - p, W = (p + 63) / 64;
  const Layout L = layout_for(0, p, d, W);
  const uint32_t *cand = g.adj + b;
  bool whole = hi - lo == p && p <= kVertexCols && d <= kVertexDegree && L.need <= c.slab_bytes &&
               (P.vertex_pass != kPivotVertices || good_pivot(g, cand + x, p));
  if (whole) {
    uint64_t *rows = (uint64_t *)(c.slab + L.rows_off);
    set_slot(c, g.slot ? g.slot[v] : 0);
    const uint32_t nrows = build_rows(g, cand, x, p, W, rows, c.sm);
    __syncwarp();
    if (W > 1) {
      uint32_t best = p;
      for (uint32_t r = c.lane; r < nrows; r += 32) {
        uint32_t n = 0;
        for (uint32_t w = 0; w < W; w++) n += __popcll(rows[(uint64_t)r * W + w]);
        best = min(best, p - n);
      }
      best = __reduce_min_sync(kFull, best);
      whole = best <= kVertexBranches && 4 * best <= p;
    }
    if (c.lane == 0) c.sm->cyc[kCycBuild] += now() - t0;
    // |R| is counted beyond a root edge: one less for a root vertex
    if (whole) solve_ego(c, cand + x, nrows, p, W, L, 0xffffffffu, g.h1[v], g.h2[v]);
  }
  if (!whole) {
    uint32_t at = 0;
    if (c.lane == 0) at = atomicAdd(P.edge_n, hi - lo);
    at = __shfl_sync(kFull, at, 0);
    for (uint32_t i = c.lane; i < hi - lo; i += 32) P.edge_out[at + i] = hi - 1 - i;
  }
  if (c.lane == 0) atomicMax(P.stat_max_item, now() - t0);
  __syncwarp();
  return whole ? p : 0;
}

// Solve a task popped from the pool; the block goes back to the free ring as
// soon as its contents are in registers or in the slab.
__device__ __noinline__ void solve_block(Ctx c, uint32_t blk) {
  const EnumParams &P = *c.P;
  const char *rec = pool_block(P, blk);
  const uint32_t *hw = (const uint32_t *)rec;
  const uint32_t pc = ld_cg(hw + 0), nrows = ld_cg(hw + 1), W = ld_cg(hw + 2), rsize = ld_cg(hw + 3);
  const uint64_t s1 = ld_cg((const uint64_t *)(rec + 16)), s2 = ld_cg((const uint64_t *)(rec + 24));
  const uint32_t slot = ld_cg(hw + 8);
  set_slot(c, slot);
  if (W == 1 && pc <= 32 && nrows <= 32) {
    T0 t0;
    t0_load<true>(c, rec, t0, pc, nrows);
    pool_free(c, blk);
    t0_solve(c, t0, pc, nrows, rsize, s1, s2);
    return;
  }
  if (W == 1 && nrows <= kT1Rows) {
    T1 t;
    t1_load<true>(c, rec, t, pc, nrows);
    pool_free(c, blk);
    t1_solve(c, t, pc, nrows, rsize, s1, s2);
    return;
  }
  const Layout L = layout_for(pc, pc, nrows, W);
  if (L.need > c.slab_bytes) {
    if (c.lane == 0) atomicExch(P.error, 2u);
    pool_free(c, blk);
    return;
  }
  uint32_t *colv = (uint32_t *)(c.slab + L.colv_off);
  const uint32_t *scol = (const uint32_t *)(rec + kHdr);
  for (uint32_t j = c.lane; j < pc; j += 32) colv[j] = ld_cg(scol + j);
  uint64_t *rows = (uint64_t *)(c.slab + L.rows_off);
  const uint64_t *srows = (const uint64_t *)(rec + kHdr + align8(4ULL * pc));
  const uint64_t nw = (uint64_t)nrows * W;
  for (uint64_t i = c.lane; i < nw; i += 32) rows[i] = ld_cg(srows + i);
  uint64_t *h1s = (uint64_t *)(c.slab + L.hash_off);
  uint64_t *h2s = h1s + pc;
  __syncwarp();
  for (uint32_t j = c.lane; j < pc; j += 32) {
    h1s[j] = P.g.h1[colv[j]];
    h2s[j] = P.g.h2[colv[j]];
  }
  pool_free(c, blk);
  Gen G;
  G.rows = rows;
  G.colv = colv;
  G.h1s = h1s;
  G.h2s = h2s;
  G.stack = (uint64_t *)(c.slab + L.stack_off);
  G.plans = (CPlan *)(c.slab + L.plan_off);
  G.alist = (uint32_t *)(c.slab + L.alist_off);
  G.alist_cap = (c.slab_bytes - kTail - L.alist_off) / 4;
  G.pc = pc;
  G.nrows = nrows;
  G.W = W;
  __syncwarp();
  gen_solve(c, G, rsize, s1, s2);
}

// Root k of this solve's work list: solve it, or defer it to the
// large-scratch pass (sized exactly), and record per-root values.  Not
// inlined: the persistent loop around it then keeps almost nothing live.
__device__ __noinline__ void run_root(Ctx c, uint64_t k) {
  const EnumParams &P = *c.P;
  WarpSmem *sm = c.sm;
  // wk: the root's index in this solve's work list (per-root results are
  // kept by it); the large-scratch pass walks a list of such indices
  const uint64_t wk = P.heavy_list ? P.heavy_list[k] : k;
  const uint64_t r = P.edge_list ? P.edge_list[wk] : P.root_list ? P.root_list[wk] : P.re - 1 - wk;  // range: late-peeled roots first
  const unsigned long long c0 = sm->count, h0 = sm->checksum;
  const unsigned long long tr = now();
  const bool fit = solve_root(c, r);
  if (c.lane == 0) atomicMax(P.stat_max_item, now() - tr);
  if (!fit) {
    if (P.push_heavy) {
      // defer the root, sized exactly: the slab must hold its candidate
      // list and an ego network of p columns and up to nc rows
      uint32_t nc = 0, nx = 0;
      intersect_count(P.g, P.g.root_v0[r], P.g.root_v1[r], &nc, &nx);
      if (c.lane == 0) {
        const uint32_t slot = atomicAdd(P.heavy_n, 1u);
        if (slot < P.heavy_cap) {
          P.heavy_out[slot] = (uint32_t)wk;
          const uint32_t p = nc - nx;
          atomicMax(P.heavy_need, (unsigned long long)layout_for(nc, p, nc, (p + 63) / 64).need);
        } else {
          atomicExch(P.error, 4u);  // more deferred roots than the list holds
        }
      }
    } else if (c.lane == 0) {
      atomicExch(P.error, 2u);
    }
  }
  if (P.per_root_count) {
    // fold the per-lane checksums of batched leaves into this root's
    const uint64_t lc = warp_sum_u64(sm->lchk[c.lane]);
    sm->lchk[c.lane] = 0;
    __syncwarp();
    if (c.lane == 0) {
      sm->checksum += lc;
      if (fit) {  // a deferred root's values come from the large-scratch pass
        P.per_root_count[wk] = sm->count - c0;
        P.per_root_checksum[wk] = sm->checksum - h0;
      }
    }
  }
  __syncwarp();
}

// Wait for a task while other warps are busy.  Returns a pool block taken
// from the ready queue (it counts as busy until its taker ends it), or -1 when no work is
// left anywhere (or the wait's bound ran out: the error word says so).
//
// At most one warp per block polls the global queue at a time (the block's
// poll token); the others sleep.  The busy count holds every warp that may
// still claim an item and every task from before it is published until its
// taker, unless that counts itself, has finished it.  Whoever adds to it is counted already (a task's
// producer; a warp before its first claim), so zero in this one word means that
// no task is queued or held: one look is enough, in any order of the ring's
// own counts.  (Warps that start late count themselves in, and wait for zero
// like any other before they leave.)  A count of busy warps alone needs the
// queue's count beside it, and no order of looks at the two sees a task that
// hops from warp to warp: blocks then left before the work it still held came
// out (full R-MAT 14 ran its second half on 1600 of 3552 warps, 25 ms instead
// of 16), and could leave a task behind.  The poller that sees zero leaves
// token value 2: the block's other warps look at the busy count themselves and
// leave, instead of each waiting for its turn.  Not inlined, so its loop holds
// only a few values: idle polling costs no reloads of the caller's state.
__device__ __noinline__ int idle_wait(Ctx c, unsigned int *s_poll) {
  const EnumParams &P = *c.P;
  WarpSmem *sm = c.sm;
  uint64_t idle_spins = 0;
  for (;;) {
    int result = -2;  // -2: keep waiting
    if (c.lane == 0) {
      const unsigned long long ti0 = now();
      bool polled = false, seen = false;
      const unsigned int token = atomicCAS(s_poll, 0u, 1u);
      if (token == 2u) {
        if (*(volatile unsigned int *)P.active == 0) result = -1;
        else atomicCAS(s_poll, 2u, 0u);  // a warp that started late holds work
      } else if (token == 0u) {
        polled = true;
        if (*(volatile unsigned int *)P.active == 0) {
          result = -1;
        } else if (*(volatile int *)P.ready_count > 0) {
          seen = true;
          uint32_t b = 0;
          if (ring_pop(P.ready_slot, P.ready_seq, P.ready_head, P.ready_count, P.pool_mask, &b, P)) result = (int)b;
        }
        atomicExch(s_poll, result == -1 ? 2u : 0u);
      }
      if (result == -2) {
        if (++idle_spins > P.spin_limit) {
          atomicExch(P.error, 1u);
          result = -1;
        } else if (!polled || seen) {
          __nanosleep(500u + ((uint32_t)(clock64() >> 3) & 511u));
        } else {
          // back off, with jitter, so idle warps do not hammer the control words
          const uint32_t shift = idle_spins < 6 ? (uint32_t)idle_spins : 6u;
          __nanosleep((256u << shift) + ((uint32_t)(clock64() >> 3) & 1023u));
        }
      }
      sm->cyc[kCycIdle] += now() - ti0;
    }
    result = __shfl_sync(kFull, result, 0);
    if (result != -2) return result;
  }
}

__global__ void __launch_bounds__(256, MCE_ENUM_BPS) k_enumerate(const __grid_constant__ EnumParams P) {
  extern __shared__ uint64_t smem_raw[];
  Ctx c;
  c.P = &P;
  c.lane = lane_id();
  WarpSmem *sm = (WarpSmem *)smem_raw + (threadIdx.x >> 5);
  c.sm = sm;
  for (uint32_t b = c.lane; b < kHistCache; b += 32) sm->hcache[b] = 0;
  if (c.lane == 0) {
    sm->count = sm->checksum = sm->nodes = sm->wops = sm->bbytes = 0;
    sm->max_size = sm->slot = sm->pending = 0;
    sm->nest = 0;
    sm->share_period = kShareMin;
    if (P.vertex_pass) {
      sm->last = range_last(P);
      sm->singles = range_singles(P);
    }
  }
  sm->lchk[c.lane] = 0;
  if (c.lane == 0) {
    for (int i = 0; i < kCycPhases; i++) sm->cyc[i] = 0;
  }
  __shared__ unsigned int s_poll;  // the block's poll token (see idle_wait)
  if (threadIdx.x == 0) s_poll = 0;
  __syncthreads();
  const uint64_t gwarp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  c.slab = P.slab + gwarp * P.slab_bytes;
  c.slab_bytes = P.slab_bytes;
  c.ta = (T1Area *)(c.slab + c.slab_bytes - kTail);
  c.sharing = P.sharing != 0;
  if (P.edge_list && !P.heavy_list && *P.edge_n == 0) return;  // the vertex pass left nothing (all blocks agree)
  const uint64_t total = P.heavy_list    ? P.n_heavy
                         : P.vertex_pass ? sm->singles + (uint64_t)(P.vert_list ? *P.vert_n : 0)
                         : P.edge_list   ? *P.edge_n
                         : P.root_list   ? P.n_list
                                         : P.re - P.rb;
  unsigned long long nroots = 0;
  // a warp counts itself busy from its first root claim until a claim fails,
  // so warps that start late (not co-resident) are never waited for
  if (c.lane == 0) atomicAdd(P.active, 1u);
  __syncwarp();
  for (;;) {
    // queued tasks first: they are the open top of the heaviest subtrees
    if (c.sharing) {
      bool got = false;
      uint32_t b = 0;
      const unsigned long long tq = now();
      if (c.lane == 0) got = ring_pop(P.ready_slot, P.ready_seq, P.ready_head, P.ready_count, P.pool_mask, &b, P);
      got = __shfl_sync(kFull, got, 0);
      const uint32_t blk = __shfl_sync(kFull, b, 0);
      if (c.lane == 0) sm->cyc[kCycQueue] += now() - tq;
      if (got) {
        const unsigned long long tb = now();
        // this warp counts itself; two for one busy warp would hide an idle one
        if (c.lane == 0) atomicSub(P.active, 1u);
        solve_block(c, blk);
        if (c.lane == 0) atomicMax(P.stat_max_item + 1, now() - tb);
        continue;
      }
    }
    unsigned long long k = 0;
    if (c.lane == 0) k = atomicAdd(P.next, 1ULL);
    k = __shfl_sync(kFull, k, 0);
    if (k >= total) break;
    if (P.vertex_pass) {
      nroots += run_vertex(c, k);
      continue;
    }
    nroots++;
    run_root(c, k);
  }
  if (c.lane == 0) atomicSub(P.active, 1u);
  if (c.sharing) {
    // roots are gone: take tasks until no warp has work left
    for (;;) {
      const int blk = idle_wait(c, &s_poll);
      if (blk < 0) break;
      const unsigned long long tb = now();
      solve_block(c, (uint32_t)blk);
      if (c.lane == 0) {
        atomicMax(P.stat_max_item + 1, now() - tb);
        atomicSub(P.active, 1u);
      }
      __syncwarp();
    }
  }
  acc_flush(c);
  if (c.lane == 0) {
    atomicAdd(P.stat_roots, nroots);
    if (P.stats) {
      atomicAdd(P.stat_nodes, sm->nodes);
      atomicAdd(P.stat_wops, sm->wops);
      atomicAdd(P.stat_bbytes, sm->bbytes);
    }
    for (int i = 0; i < kCycPhases; i++) atomicAdd(P.stat_cycles + i, sm->cyc[i]);
  }
}

// Control words; the contended ones each own a 128-byte line.
struct EnumCtl {
  alignas(128) unsigned long long next;
  alignas(128) unsigned long long next_edge;  // claims of the edge pass
  alignas(128) unsigned long long free_head;
  alignas(128) unsigned long long free_tail;
  alignas(128) unsigned long long ready_head;
  alignas(128) unsigned long long ready_tail;
  alignas(128) int ready_count;  // filled cells not yet claimed
  alignas(128) int free_count;
  alignas(128) unsigned int active;
  alignas(128) unsigned long long heavy_need, stat_roots, stat_tasks, stat_nodes, stat_wops, stat_bbytes;
  unsigned long long stat_cycles[kCycPhases];
  unsigned long long stat_max_item[2];
  unsigned int heavy_n, error, edge_n, vert_n;
};

// free ring full of every block, ready ring empty, counters reset
__global__ void k_pool_init(EnumCtl *ctl, uint32_t *free_slot, unsigned long long *free_seq,
                            unsigned long long *ready_seq, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    free_slot[i] = i;
    free_seq[i] = (unsigned long long)i + 1;  // filled for the consumer of position i
    ready_seq[i] = i;                        // free for the producer of position i
  }
  // word by word: the compiler takes minutes over a copy of the padded struct
  if (blockIdx.x == 0) {
    for (uint32_t w = threadIdx.x; w < sizeof(EnumCtl) / 4; w += blockDim.x) ((uint32_t *)ctl)[w] = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
      ctl->free_tail = n;
      ctl->free_count = (int)n;
    }
  }
}

mce_status reset_ctl(const EnumPlan &plan, cudaStream_t st) {
  k_pool_init<<<grid_for(plan.pool_blocks, 256), 256, 0, st>>>((EnumCtl *)plan.ctl, plan.params.free_slot,
                                                               plan.params.free_seq, plan.params.ready_seq,
                                                               plan.pool_blocks);
  note_launch();
  MCE_CUDA_TRY(cudaGetLastError());
  return MCE_OK;
}

// the launch behind the vertex pass: the roots that pass left
EnumParams edge_pass(const EnumPlan &plan) {
  EnumParams P = plan.params;
  P.vertex_pass = 0;
  P.edge_list = P.edge_out;
  P.next = &((EnumCtl *)plan.ctl)->next_edge;
  return P;
}

// How a range of a graph goes: root by root, or vertices first, all of them or
// those with a good pivot.  One warp solves all roots of a vertex: it takes
// longer than the longest root, and the roots left wait for the pass to end.
// Root by root, every root work of its own, where
//   * warps outnumber the roots;
//   * nobody takes over a heavy vertex's open work (no sharing) and there may
//     be some.
// Not all vertices, where
//   * warps outnumber the vertices two to one;
//   * vertices have many later neighbours on average: without a good pivot
//     their ego networks are searched no faster than their roots', and from 65
//     on built for nothing -- unless the mean vertex is adjacent to a sixth of
//     its graph (the graphs are many then), where a vertex's roots share most
//     of their networks.
// Looking for pivots takes a pass of its own, which pays from ego networks of 64
// later neighbours on.
// Measured (B200, 4736 warps), enumeration, ms, vertices first and root by root:
//   G(64, mean degree 32) 0.128, 0.077; G(500, 64) 0.43, 0.13
//   G(3000, 32) 0.091, 0.118; G(3000, 64) 0.46, 0.26; G(6000, 64) 0.36, 0.39
//   G(6000, 100) 1.20, 0.82; G(30000, 64) 0.69, 1.30; G(30000, 100) 2.75, 2.29
//   100 x G(300, 90) 13.6, 19.0; 40 x G(500, 100) 8.1, 8.6; 30 x G(1000, 100) 8.3,
//   8.4; 60 x G(1000, 150) 58, 49
//   R-MAT 12 and 13, edge factor 16: 1.82, 1.91 and 3.4, 4.1
//   without sharing: R-MAT 13 160, 45; G(200, 100) 2.7, 0.85; planted cliques of
//   10-60 in 20,000 vertices 0.14, 0.47
// and with pivots only: 300 cliques of 200 vertices 17.7, 972, 17.9; G(6000, 150)
// 3.3, 2.1, 2.1; G(3000, 64) 0.46, 0.26, 0.33.
VertexPass vertex_pass_for(const DeviceGraph &g, uint64_t nwork, uint64_t nwarps, uint64_t n_graphs, bool sharing) {
  if (nwork <= nwarps) return kNoVertices;
  if (!sharing && g.max_degree > 256) return kNoVertices;
  const uint64_t n = g.n;
  const bool dense = 12 * g.m * n_graphs >= n * n;
  const uint64_t later = n < nwarps ? 24 : dense ? 256 : 40;
  if (2 * n >= nwarps && g.m <= later * n) return kAllVertices;
  return g.degeneracy < 64 || (!sharing && 2 * n < nwarps) ? kNoVertices : kPivotVertices;
}

}  // namespace

mce_status MCE_ENUM_FN(enum_plan)(const DeviceGraph &g, const EnumConfig &cfg, Scratch *scr, SlotResult *slots,
                     unsigned long long *hist, EnumPlan *plan) {
  const int device = scr->device;
  int sms = 0;
  MCE_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const uint32_t wpb = cfg.warps_per_block ? std::min(cfg.warps_per_block, 8u) : 8u;
  const uint32_t bps = cfg.blocks_per_sm ? std::min<uint32_t>(cfg.blocks_per_sm, MCE_ENUM_BPS) : MCE_ENUM_BPS;
  EnumParams &P = plan->params;
  P = EnumParams{};
  P.g.n = g.n;
  P.g.m = g.m;
  P.g.off = g.off;
  P.g.adj = g.adj;
  P.g.labels = g.labels;
  P.g.h1 = g.h1;
  P.g.h2 = g.h2;
  P.g.root_v0 = g.root_v0;
  P.g.root_v1 = g.root_v1;
  P.g.root_off = g.root_off;
  P.g.slot = g.slot;
  P.slots = slots;
  P.hist = hist;
  P.hist_len = cfg.hist_len;
  P.expand_r = cfg.expand_r;
  P.per_root_count = cfg.per_root_count;
  P.per_root_checksum = cfg.per_root_checksum;
  P.spin_limit = cfg.spin_limit ? cfg.spin_limit : (1ULL << 34);
  P.sharing = (cfg.sharing && cfg.per_root_count == nullptr) ? 1 : 0;
  P.stats = cfg.stats;
  P.share_bound = cfg.share_bound ? cfg.share_bound : 24;
  P.reg_share_bound = std::min(P.share_bound, cfg.reg_share_bound ? cfg.reg_share_bound : kRegShareBound);
  mce_status s = MCE_OK;
  EnumCtl *ctl = (EnumCtl *)scr->get(1, sizeof(EnumCtl), &s);
  if (!ctl) return s;
  plan->ctl = ctl;
  P.next = &ctl->next;
  P.heavy_need = &ctl->heavy_need;
  P.heavy_n = &ctl->heavy_n;
  P.error = &ctl->error;
  P.stat_roots = &ctl->stat_roots;
  P.stat_tasks = &ctl->stat_tasks;
  P.stat_nodes = &ctl->stat_nodes;
  P.stat_wops = &ctl->stat_wops;
  P.stat_bbytes = &ctl->stat_bbytes;
  P.stat_cycles = ctl->stat_cycles;
  P.stat_max_item = ctl->stat_max_item;
  P.active = &ctl->active;
  P.free_head = &ctl->free_head;
  P.free_tail = &ctl->free_tail;
  P.ready_head = &ctl->ready_head;
  P.ready_tail = &ctl->ready_tail;
  P.ready_count = &ctl->ready_count;
  P.free_count = &ctl->free_count;

  uint64_t rb = cfg.root_begin, re = cfg.root_end ? std::min<uint64_t>(cfg.root_end, g.m) : g.m;
  if (rb > re) rb = re;
  const bool list_mode = cfg.root_list != nullptr;
  const uint64_t nwork = list_mode ? cfg.n_root_list : re - rb;
  plan->nwork = nwork;

  uint32_t blocks = (uint32_t)sms * bps;
  if (cfg.max_blocks && blocks > cfg.max_blocks) blocks = cfg.max_blocks;
  if (!P.sharing) {
    const uint64_t want_blocks = (nwork + wpb - 1) / wpb;
    if (want_blocks < blocks) blocks = (uint32_t)std::max<uint64_t>(want_blocks, 1);
  }
  const uint64_t nwarps = (uint64_t)blocks * wpb;
  P.nwarps = (uint32_t)nwarps;
  // slab: the largest ego network this graph can produce (p <= degeneracy,
  // rows <= max degree), capped at 4 MB per warp and by free memory
  const uint64_t kcap = std::max<uint32_t>(1, std::min(g.degeneracy, g.max_degree));
  const uint64_t dcap = std::max<uint32_t>(1, g.max_degree);
  const Layout LB = layout_for(dcap, (uint32_t)kcap, (uint32_t)(kcap + dcap), (uint32_t)((kcap + 63) / 64));
  const uint64_t bound = align8(LB.need + 3ULL * (kcap + dcap) * 4);
  const uint64_t slab_cap = cfg.slab_kib ? std::max<uint64_t>(16, cfg.slab_kib) << 10 : 4ULL << 20;
  uint64_t slab_bytes = std::max<uint64_t>(std::min<uint64_t>(bound, slab_cap), 16ULL << 10);
  // Free memory limits what is newly allocated: asking for it costs tens of
  // microseconds, so scratch that already holds the full sizes is used as it is.
  const uint32_t pool_max = 1u << 14;
  const auto block_size = [](uint64_t slab) {
    return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(4096, align8(slab / 4)), 64 << 10);
  };
  size_t freeb = SIZE_MAX, totalb = 0;
  if (scr->bytes[2] < ((slab_bytes + 255) & ~255ULL) * nwarps ||
      scr->bytes[5] < (uint64_t)pool_max * block_size((slab_bytes + 255) & ~255ULL))
    MCE_CUDA_TRY(cudaMemGetInfo(&freeb, &totalb));
  while (slab_bytes > (64ULL << 10) && slab_bytes * nwarps > freeb / 2) slab_bytes >>= 1;
  slab_bytes = (slab_bytes + 255) & ~255ULL;  // every warp's slab (and its T1Area) 256-byte aligned
  plan->fits_all = slab_bytes >= bound;
  char *slab = (char *)scr->get(2, slab_bytes * nwarps, &s);
  if (!slab) return s;
  // A range goes vertex by vertex first; per-root values and the counters of
  // the edge-rooted method (stats) need every root on its own.
  const VertexPass pass_kind = list_mode || P.per_root_count || P.stats
                                   ? kNoVertices
                                   : vertex_pass_for(g, nwork, nwarps, cfg.n_slots, P.sharing);
  plan->vertex_pass = pass_kind != kNoVertices;
  // One buffer of lists: the vertex pass's roots and vertices left, and the
  // roots whose ego network overflows the slab, deferred to a second pass.
  // Those are kept by work index (a solve of more than 2^32 roots is refused by
  // the callers).  One buffer, since each that grows with the graph costs a
  // first solve an allocation, which waits for the device.
  const uint64_t heavy_cap = std::min<uint64_t>(nwork, 1ULL << 26);
  uint32_t *heavy = nullptr;
  if (nwork) {
    const uint64_t pass = plan->vertex_pass ? nwork + g.n : 0;
    heavy = (uint32_t *)scr->get(3, (heavy_cap + pass) * 4, &s);
    if (!heavy && pass) {  // no room for the vertex pass's lists: root by root
      plan->vertex_pass = false;
      heavy = (uint32_t *)scr->get(3, heavy_cap * 4, &s);
    }
    if (!heavy) return s;
  }
  // task pool: one record per block; both rings have one cell per block
  const uint32_t block_bytes = block_size(slab_bytes);
  uint32_t nblocks = pool_max;
  while ((uint64_t)nblocks * block_bytes > (freeb / 8) && nblocks > 1024) nblocks >>= 1;
  char *pool = (char *)scr->get(5, (uint64_t)nblocks * block_bytes, &s);
  if (!pool) return s;
  char *rings = (char *)scr->get(6, (uint64_t)nblocks * 24, &s);
  if (!rings) return s;
  P.pool = pool;
  P.block_bytes = block_bytes;
  P.pool_mask = nblocks - 1;
  P.free_seq = (unsigned long long *)rings;
  P.ready_seq = (unsigned long long *)(rings + (uint64_t)nblocks * 8);
  P.free_slot = (uint32_t *)(rings + (uint64_t)nblocks * 16);
  P.ready_slot = (uint32_t *)(rings + (uint64_t)nblocks * 20);
  plan->pool_blocks = nblocks;
  P.slab = slab;
  P.slab_bytes = slab_bytes;
  P.rb = rb;
  P.re = re;
  P.root_list = list_mode ? cfg.root_list : nullptr;
  P.n_list = list_mode ? cfg.n_root_list : 0;
  if (plan->vertex_pass) {
    P.vertex_pass = pass_kind;
    P.edge_out = heavy + heavy_cap;
    P.edge_n = &ctl->edge_n;
    if (g.n > kVertexSingles * nwarps) {
      P.vert_list = P.edge_out + nwork;
      P.vert_n = &ctl->vert_n;
      P.single_items = kVertexSingles * nwarps;
    }
  }
  P.heavy_out = heavy;
  P.heavy_cap = (uint32_t)heavy_cap;
  P.push_heavy = 1;
  plan->heavy_warps = cfg.heavy_warps;
  plan->blocks = blocks;
  plan->sms = (uint32_t)sms;
  plan->threads = wpb * 32;
  plan->smem = (size_t)wpb * sizeof(WarpSmem);
  plan->nwarps = nwarps;
  plan->scr = scr;
  if (plan->smem > 48 * 1024)
    MCE_CUDA_TRY(cudaFuncSetAttribute(k_enumerate, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan->smem));
  return MCE_OK;
}

mce_status MCE_ENUM_FN(enum_launch)(const EnumPlan &plan, cudaStream_t st) {
  MCE_TRY(reset_ctl(plan, st));
  if (plan.nwork) {
    if (plan.params.vert_list) MCE_TRY(launch_tiny(plan.params, plan.sms, st));
    k_enumerate<<<plan.blocks, plan.threads, plan.smem, st>>>(plan.params);
    note_launch();
    if (plan.vertex_pass) {
      k_enumerate<<<plan.blocks, plan.threads, plan.smem, st>>>(edge_pass(plan));
      note_launch();
    }
    MCE_CUDA_TRY(cudaGetLastError());
  }
  return MCE_OK;
}

mce_status MCE_ENUM_FN(enum_finish)(const EnumPlan &plan, cudaStream_t st, EnumStats *stats) {
  EnumCtl *ctl = (EnumCtl *)plan.ctl;
  EnumCtl h{};
  MCE_CUDA_TRY(cudaMemcpyAsync(&h, ctl, sizeof(EnumCtl), cudaMemcpyDeviceToHost, st));
  MCE_CUDA_TRY(cudaStreamSynchronize(st));
  const uint64_t heavy_roots = h.heavy_n;
  uint64_t launches = plan.nwork ? (plan.params.vert_list ? 3 : plan.vertex_pass ? 2 : 1) : 0;
  uint64_t roots = h.stat_roots;
  uint64_t tasks = h.stat_tasks, nodes = h.stat_nodes, wops = h.stat_wops, bbytes = h.stat_bbytes;
  uint64_t cycles[kCycPhases];
  for (int i = 0; i < kCycPhases; i++) cycles[i] = h.stat_cycles[i];
  uint64_t max_item[2] = {h.stat_max_item[0], h.stat_max_item[1]};
  // 5: a task was left behind (cannot happen, see idle_wait): the totals are short
  const auto error_of = [](const EnumCtl &x) { return x.error ? x.error : x.active || x.ready_count ? 5u : 0u; };
  uint32_t err = error_of(h);
  if (h.heavy_n && !err) {
    // Deferred roots: one slab per warp, each sized for the largest deferred
    // ego network; every warp of the pass shares their work (unless per-root
    // values are being attributed, which keeps each root on one warp).  Only
    // warps that get a slab are launched: with fewer slabs than a block's
    // warps, the block shrinks to that many.
    size_t freeb = 0, totalb = 0;
    MCE_CUDA_TRY(cudaMemGetInfo(&freeb, &totalb));
    const uint64_t need = ((h.heavy_need + 4096) + 255) & ~255ULL;
    uint64_t hw = std::min<uint64_t>((uint64_t)(freeb * 0.7) / need, plan.nwarps);
    if (plan.heavy_warps) hw = std::min<uint64_t>(hw, plan.heavy_warps);
    hw = std::min<uint64_t>(hw, h.heavy_n);
    if (hw == 0) return MCE_ERR_OUT_OF_MEMORY;
    EnumPlan H = plan;
    if (H.vertex_pass) H.params = edge_pass(plan);  // the list holds indices of that pass
    H.params.next = &ctl->next;
    const uint32_t wpb = plan.threads / 32;
    if (hw < wpb) {
      H.blocks = 1;
      H.threads = (uint32_t)hw * 32;
      H.smem = (size_t)hw * sizeof(WarpSmem);
    } else {
      H.blocks = (uint32_t)(hw / wpb);
    }
    H.nwarps = (uint64_t)H.blocks * (H.threads / 32);
    mce_status s = MCE_OK;
    char *big = (char *)plan.scr->get(4, need * H.nwarps, &s);
    if (!big) return s;
    H.params.slab = big;
    H.params.slab_bytes = need;
    H.params.heavy_list = plan.params.heavy_out;
    H.params.n_heavy = h.heavy_n;
    H.params.push_heavy = 0;
    H.params.nwarps = (uint32_t)H.nwarps;
    cudaEvent_t he0, he1;
    MCE_CUDA_TRY(cudaEventCreate(&he0));
    MCE_CUDA_TRY(cudaEventCreate(&he1));
    cudaEventRecord(he0, st);
    mce_status ls = reset_ctl(H, st);
    if (ls == MCE_OK) {
      k_enumerate<<<H.blocks, H.threads, H.smem, st>>>(H.params);
      note_launch();
      launches++;
      if (cudaGetLastError() != cudaSuccess) ls = MCE_ERR_CUDA;
    }
    cudaEventRecord(he1, st);
    EnumCtl h2{};
    if (ls == MCE_OK && cudaMemcpyAsync(&h2, ctl, sizeof(EnumCtl), cudaMemcpyDeviceToHost, st) != cudaSuccess)
      ls = MCE_ERR_CUDA;
    if (ls == MCE_OK && cudaStreamSynchronize(st) != cudaSuccess) ls = MCE_ERR_CUDA;
    float hms = 0;
    if (ls == MCE_OK) cudaEventElapsedTime(&hms, he0, he1);
    cudaEventDestroy(he0);
    cudaEventDestroy(he1);
    if (ls != MCE_OK) return ls;
    if (stats) stats->ms_heavy = hms;
    roots = roots - heavy_roots + h2.stat_roots;
    tasks += h2.stat_tasks;
    nodes += h2.stat_nodes;
    wops += h2.stat_wops;
    bbytes += h2.stat_bbytes;
    for (int i = 0; i < kCycPhases; i++) cycles[i] += h2.stat_cycles[i];
    for (int i = 0; i < 2; i++) max_item[i] = std::max<uint64_t>(max_item[i], h2.stat_max_item[i]);
    err = error_of(h2);
  }
  if (stats) {
    stats->roots = roots;
    stats->heavy_roots = heavy_roots;
    stats->shared_tasks = tasks;
    stats->nodes = nodes;
    stats->word_ops = wops;
    stats->build_bytes = bbytes;
    for (int i = 0; i < kCycPhases; i++) stats->cycles[i] = cycles[i];
    for (int i = 0; i < 2; i++) stats->max_item[i] = max_item[i];
    stats->error = err;
    stats->launches = launches;
  }
  if (err == 2) return MCE_ERR_OUT_OF_MEMORY;
  if (err == 4) return MCE_ERR_CAPACITY;
  if (err == 5) return MCE_ERR_INTERNAL;
  if (err) return MCE_ERR_TIMEOUT;
  return MCE_OK;
}

#if MCE_ENUM_BPS == 4
namespace {
// Integer-pipe probe: per thread, 8 independent chains of the enumeration's
// word-op mix (a 64-bit ANDN feeding a 64-bit POPC, folded back by an add).
__global__ void k_int_probe(const uint64_t *seed, uint64_t *sink, int iters) {
  uint64_t a[8];
  const uint64_t b = seed[0] ^ (threadIdx.x * 0x9E3779B97F4A7C15ULL);
#pragma unroll
  for (int i = 0; i < 8; i++) a[i] = seed[1] + (uint64_t)i * 0x632BE59BD9B4E019ULL + blockIdx.x;
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int i = 0; i < 8; i++) a[i] += __popcll(a[i] & ~b) | (a[i] << 7);
  }
  uint64_t x = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) x ^= a[i];
  if (x == 0x123456789ULL) sink[0] = x;  // keeps the chains live
}

}  // namespace

mce_status probe_int_peak(int device, double *word_ops_per_s) {
  MCE_CUDA_TRY(cudaSetDevice(device));
  int sms = 0;
  MCE_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  uint64_t *buf = nullptr;
  MCE_CUDA_TRY(cudaMalloc(&buf, 64));
  MCE_CUDA_TRY(cudaMemset(buf, 0x5a, 64));
  const int iters = 4096, threads = 256, blocks = sms * 8;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_int_probe<<<blocks, threads>>>(buf, buf + 4, 64);
  note_launch();
  cudaEventRecord(e0);
  k_int_probe<<<blocks, threads>>>(buf, buf + 4, iters);
  note_launch();
  cudaEventRecord(e1);
  const cudaError_t e = cudaEventSynchronize(e1);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(buf);
  if (e != cudaSuccess || ms <= 0) return MCE_ERR_CUDA;
  // two word-ops (ANDN, POPC) per chain step
  *word_ops_per_s = 2.0 * 8.0 * iters * (double)threads * blocks / (ms * 1e-3);
  return MCE_OK;
}

#endif

}  // namespace mce
