// Whole traversals in one launch.
//
// A level-by-level run costs six or seven launches and a host round trip per
// level (about 30 us), whatever the level holds; on graphs up to a few
// million edges that is most of a call.  Here one cooperative launch runs
// every level: its CTAs keep the frontier on the device, meet at a grid
// barrier (about 1.3 us over the whole chip, a __syncthreads for the smallest
// graphs, which get one CTA) and take every decision from counters that all of
// them read after the barrier.  What bounds a small graph now is the chain of
// dependent loads of a level, about 5 us with its barrier (BFS, R-MAT edge
// factor 16: 2^10 vertices 182 -> 27 us, 2^16 298 -> 43 us); a large one is bound
// by its pulls' gathers, as level by level (2^24: 973 -> 450 us; the compactions
// between the levels are gone).
//
// The frontier is two unordered queues: vertices of degree <= kSmallDeg, four
// lanes each, and pieces of at most kPiece edges of the larger ones, a warp
// each, so a hub and a leaf cost the same per edge.  Winners are collected in a
// per-warp shared-memory buffer and appended with one counter update per flush.
//
// Every wait is bounded: a CTA that waits too long says so to the host and returns,
// and the host, whatever the other CTAs made of it, answers level by level.

#include <cuda_runtime.h>
#include <math_constants.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <utility>
#include <vector>

#include "fused.cuh"
#include "pr_exact.cuh"

namespace rg {

namespace {

constexpr int kFT = 1024;             // threads per CTA, one CTA per SM
constexpr int kFWarps = kFT / 32;
constexpr uint32_t kSmallDeg = 32;    // at most this degree: four lanes per vertex
constexpr uint32_t kPiece = 128;      // edges per piece of a larger vertex
constexpr int kFlushAt = 64;          // winners a warp collects before it appends them
constexpr int kBuf = kFlushAt + 32;
constexpr unsigned kAll = 0xffffffffu;
constexpr unsigned kPolls = 1u << 21;  // of the grid barrier: a second or two

// One level's frontier: queue lengths, members and their degree sum
// (PageRankDelta: and the round's L1; BFS and BC: the pieces of long lists that a
// pull puts off).
struct alignas(16) Slot {
  unsigned int ns, nl, count, heavy;
  unsigned long long degsum;
  double l1;
};

// A 128-bit sum that CTAs add to without waiting for a carry: 43-bit limbs in
// 64-bit words, so up to 2^21 additions fit.
struct L1Sum {
  unsigned long long limb[4];  // the fourth is padding
  __device__ __forceinline__ void add(const U128& x) {
    constexpr unsigned long long kMask = (1ull << 43) - 1;
    atomicAdd(&limb[0], x.lo & kMask);
    atomicAdd(&limb[1], ((x.lo >> 43) | (x.hi << 21)) & kMask);
    atomicAdd(&limb[2], x.hi >> 22);
  }
  __device__ __forceinline__ U128 read() const {
    const unsigned long long a = __ldcg(&limb[0]), b = __ldcg(&limb[1]), c = __ldcg(&limb[2]);
    U128 s{a, 0ull};
    add128(s, U128{b << 43, b >> 21});
    add128(s, U128{0ull, c << 22});
    return s;
  }
};

// Zero when a launch begins.  Two sets take turns: a launch clears the one that the
// launch before it used (a memset of its own cost a call 3 us: BFS 2^10 40 -> 37).
struct Ctl {
  unsigned int bar;
  unsigned int bar_all;  // of all groups (BC)
  int levels;            // of the group's source (BC)
  unsigned int pad0;
  unsigned long long edges;
  unsigned int pad[10];
  Slot lv[4];
};

// What every launch gets besides its own arguments (launch_fused fills it in).
struct Launch {
  Ctl *ctl, *stale;
  int nstale;
  unsigned polls, from;        // polls of a grid barrier, from the launch's `from`-th on, before it gives up
  volatile uint64_t* gave_up;  // mapped: set by a CTA that did.  (The last barrier's others pass and say that
                               // the run is done, without that CTA's share of the results.)
};

// The warp's sums of four values: of acc[p] in lanes 8p .. 8p + 7.  Six FP64 adds
// in place of twenty (GB300 issues one FP64 warp instruction per 16 clocks).
__device__ __forceinline__ double warp_sum4(const double (&acc)[4]) {
  const bool hi = threadIdx.x & 16, odd = threadIdx.x & 8;
  const double x0 = __shfl_xor_sync(kAll, hi ? acc[0] : acc[2], 16);
  const double x1 = __shfl_xor_sync(kAll, hi ? acc[1] : acc[3], 16);
  const double y0 = (hi ? acc[2] : acc[0]) + x0, y1 = (hi ? acc[3] : acc[1]) + x1;
  double z = (odd ? y1 : y0) + __shfl_xor_sync(kAll, odd ? y0 : y1, 8);
  z += __shfl_xor_sync(kAll, z, 4);
  z += __shfl_xor_sync(kAll, z, 2);
  return z + __shfl_xor_sync(kAll, z, 1);
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// A member of the next frontier and its edges.
struct Member {
  uint32_t v, b, e;
};

// The CTAs that meet at a barrier.
struct Team {
  unsigned* bar;
  unsigned target, ctas;
};

// What a CTA shares: its members' totals, what the last barrier completed and
// the barrier's verdict.
struct Shared {
  Team team[2];  // the group's CTAs, and all of them (BC)
  unsigned polls, from;
  volatile uint64_t* gave_up;
  unsigned int count;
  unsigned long long degsum;
  Slot slot;  // the frontier that the last barrier completed
  U128 l1;    // the sum that it completed (PageRank)
  uint32_t taken;  // work that the CTA's warps have taken since
  int ok;
};

__device__ __forceinline__ Slot read_slot(const Slot* s) {
  const uint4 a = __ldcg(reinterpret_cast<const uint4*>(s));
  const ulonglong2 b = __ldcg(reinterpret_cast<const ulonglong2*>(&s->degsum));
  return Slot{a.x, a.y, a.z, a.w, b.x, __longlong_as_double((long long)b.y)};
}

// The barrier's wait, after a first look.  0: it ran out.  (Out of line: what it needs
// of shared memory is read beside the polls, off the path of a wait that ends.)
__device__ __noinline__ int poll(Shared* sh, const Team& t) {
  unsigned left = t.target > (unsigned long long)sh->from * t.ctas ? sh->polls : kPolls;
  do {
    if (left-- == 0) {
      *sh->gave_up = 1;
      return 0;
    }
  } while ((int)(ld_acquire(t.bar) - t.target) < 0);
  return 1;
}

struct Grid {
  Shared* sh;
  int which;

  // All CTAs meet; this CTA's totals go into `slot` first (null: dropped) and the
  // completed slot comes back in sh->slot (and the completed sum `l1` in sh->l1).
  // keep: the totals stay for the next barrier.  What
  // any thread wrote before is visible to every thread after.  False: the wait
  // ran out.
  __device__ __forceinline__ bool sync(Slot* slot = nullptr, const L1Sum* l1 = nullptr, bool keep = false) {
    __syncthreads();
    if (threadIdx.x == 0) {
      Team& t = sh->team[which];
      if (slot && sh->count) {
        atomicAdd(&slot->count, sh->count);
        atomicAdd(&slot->degsum, sh->degsum);
      }
      const bool others = t.ctas > 1;
      if (others) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(t.bar) : "memory");
      else __threadfence();
      t.target += t.ctas;
      if (!keep) {
        sh->count = 0;
        sh->degsum = 0;
      }
      sh->taken = 0;
      int ok = 1;
      if (others && (int)(ld_acquire(t.bar) - t.target) < 0) ok = poll(sh, t);
      if (l1) sh->l1 = l1->read();
      if (slot) sh->slot = read_slot(slot);  // once per CTA: thousands of warps would queue on its line
      sh->ok = ok;
    }
    __syncthreads();
    return sh->ok != 0;
  }
};

// An entry: a vertex, the edges [y, z) of it that the entry stands for, and in w
// twice the vertex's number of entries, plus 1 on its first.
struct Queues {
  uint4* small;  // whole vertices
  uint4* large;  // pieces
};

// Appends a warp's n collected winners (buf) to the next frontier's queues and
// adds their number and degrees to the CTA's totals.  kEmpty: vertices without
// edges are queued too (the caller visits every member).
template <bool kEmpty>
__device__ __noinline__ void flush_winners(const Member* buf, int n, uint4* qs, uint4* ql, Slot* slot, uint32_t sbase,
                                           uint32_t lbase, Shared* sh) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  uint32_t v[kBuf / 32], b[kBuf / 32], d[kBuf / 32];
  unsigned small_total = 0;
  unsigned long long degsum = 0;
#pragma unroll
  for (int i = 0; i < kBuf / 32; i++) {
    v[i] = 0;
    d[i] = 0;
    b[i] = 0;
    const bool in = i * 32 + lane < n;
    if (in) {
      const Member x = buf[i * 32 + lane];
      v[i] = x.v;
      b[i] = x.b;
      d[i] = x.e - x.b;
      degsum += d[i];
    }
    small_total += __popc(__ballot_sync(kAll, d[i] <= kSmallDeg && (kEmpty ? in : d[i] > 0)));
  }
  degsum = warp_sum(degsum);
  unsigned at = 0;
  if (lane == 0) {
    atomicAdd(&sh->count, (unsigned)n);
    atomicAdd(&sh->degsum, degsum);
    if (small_total) at = atomicAdd(&slot->ns, small_total);
  }
  at = __shfl_sync(kAll, at, 0) + sbase;
#pragma unroll
  for (int i = 0; i < kBuf / 32; i++) {
    const bool is = d[i] <= kSmallDeg && (kEmpty ? i * 32 + lane < n : d[i] > 0);
    const unsigned m = __ballot_sync(kAll, is);
    if (is) qs[at + __popc(m & ((1u << lane) - 1u))] = make_uint4(v[i], b[i], b[i] + d[i], 3u);
    at += __popc(m);
    if (__any_sync(kAll, d[i] > kSmallDeg)) {
      const unsigned pieces = d[i] > kSmallDeg ? (d[i] + kPiece - 1) / kPiece : 0;
      unsigned inc = pieces;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(kAll, inc, o);
        if (lane >= o) inc += t;
      }
      unsigned lat = 0;
      if (lane == 31) lat = atomicAdd(&slot->nl, inc);
      lat = __shfl_sync(kAll, lat, 31) + lbase;
      // every lane writes every 32nd piece; its vertex is the first whose pieces
      // end past it (a hub's hundreds of pieces cost the warp no more than as
      // many vertices with one)
      const unsigned total = __shfl_sync(kAll, inc, 31);
      for (unsigned p0 = 0; p0 < total; p0 += 32) {
        const unsigned p = p0 + lane;
        int j = 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          if (__shfl_sync(kAll, inc, j + o - 1) <= p) j += o;
        }
        j &= 31;  // (past the last piece: unused)
        const uint32_t jv = __shfl_sync(kAll, v[i], j), jb = __shfl_sync(kAll, b[i], j);
        const uint32_t jend = jb + __shfl_sync(kAll, d[i], j);
        const unsigned np = __shfl_sync(kAll, pieces, j), k = p - (__shfl_sync(kAll, inc, j) - np);
        if (p < total) {
          const uint32_t y = jb + k * kPiece;
          ql[lat + p] = make_uint4(jv, y, min(y + kPiece, jend), 2 * np + (k == 0 ? 1u : 0u));
        }
      }
    }
  }
  __syncwarp();
}

// A warp's winners on their way into the next frontier's queues.
template <bool kEmpty>
struct Appender {
  Member* buf;
  Shared* sh;
  int n;

  // b, e: v's edges (the caller loads them beside the update that decides
  // `won`, so that an append waits for no memory)
  __device__ __forceinline__ void add(bool won, uint32_t v, uint32_t b, uint32_t e, const Queues& q, Slot* slot,
                                      uint32_t sbase, uint32_t lbase) {
    const unsigned m = __ballot_sync(kAll, won);
    if (!m) return;
    if (won) buf[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = Member{v, b, e};
    n += __popc(m);
    if (n >= kFlushAt) finish(q, slot, sbase, lbase);
  }

  __device__ __forceinline__ void finish(const Queues& q, Slot* slot, uint32_t sbase, uint32_t lbase) {
    if (n) flush_winners<kEmpty>(buf, n, q.small, q.large, slot, sbase, lbase, sh);
    n = 0;
  }
};

// fn(lane has an edge, source, neighbour) over every edge of a frontier, all
// lanes of a warp together, four edges per lane in flight.  The caller is CTA
// `cta` of the `ctas` that share the frontier.
template <class Fn>
__device__ __forceinline__ void expand(const DevGraph& g, const Queues& q, uint32_t sbase, uint32_t ns, uint32_t lbase,
                                       uint32_t nl, uint32_t cta, uint32_t ctas, Fn&& fn) {
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (threadIdx.x >> 5) * ctas + cta;  // neighbours on other SMs
  const uint32_t nwarps = ctas * kFWarps;
  // a short frontier is spread over more warps, a quarter of a piece or one vertex
  // each: few warps would also be left with all that it wins (one hub's 6933
  // neighbours, 2.8e5 pieces: 41 of 56 us on 55 warps)
  const int quarter = nl * 4 <= nwarps ? 2 : 0;
  for (uint32_t i = warp; i < nl << quarter; i += nwarps) {
    const uint4 it = q.large[lbase + (i >> quarter)];
    const uint32_t e0 = it.y + (quarter ? 32 * (i & 3) : 0) + lane;
    uint32_t d[4];
    bool in[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t e = e0 + 32 * k;
      in[k] = e < it.z && (k == 0 || !quarter);
      d[k] = in[k] ? g.adj[e] : 0u;
    }
    fn(in, it.x, d);
  }
  const int few = ns <= nwarps ? 5 : 2;  // lanes per vertex, as a shift
  const uint32_t groups = (ns + (31 >> few)) >> (5 - few);
  for (uint32_t i = warp; i < groups; i += nwarps) {
    const uint32_t j = (i << (5 - few)) + (lane >> few);
    const uint4 it = j < ns ? q.small[sbase + j] : make_uint4(0, 0, 0, 0);
    const uint32_t s = it.x, b = it.y, end = it.z;
    for (uint32_t e0 = b + (lane & ((1 << few) - 1)); __any_sync(kAll, e0 < end); e0 += 4 << few) {
      uint32_t d[4];
      bool in[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t e = e0 + (k << few);
        in[k] = e < end;
        d[k] = in[k] ? g.adj[e] : 0u;
      }
      fn(in, s, d);
    }
  }
}

__device__ __forceinline__ void begin(Grid& grid, Shared* sh, const Launch& L, Ctl* ctl) {
  if (blockIdx.x == 0 && blockIdx.y == 0) {  // what the launch before used, for the one after
    unsigned* w = reinterpret_cast<unsigned*>(L.stale);
    for (int i = threadIdx.x; i < L.nstale * (int)(sizeof(Ctl) / 4); i += kFT) w[i] = 0u;
  }
  grid.sh = sh;
  grid.which = 0;
  if (threadIdx.x == 0) {
    sh->team[0] = Team{&ctl->bar, 0, gridDim.x};
    sh->polls = L.polls;
    sh->from = L.from;
    sh->gave_up = L.gave_up;
    sh->count = 0;
    sh->degsum = 0;
    sh->taken = 0;
    sh->ok = 1;
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// BFS (BFS.C:122-188)
// ---------------------------------------------------------------------------
constexpr uint32_t kPullWords = 8;  // words of the visited bitmap that a warp takes together, at most
// A pull's warp reads this much of a vertex's list beyond its first 48 edges; the rest
// of a longer one, as a rule a hub's that the search does not reach at all, is put off
// and read in pieces by all warps.  (By one warp, 32 edges after 32: 2^20 vertices
// beside a star of 2e6 that they do not reach 32.8 ms, 0.11 now; beside as many
// vertices again, degree sorted, 17.3 and 0.43.)
constexpr uint32_t kRestList = 256, kRestPiece = 512;

struct BfsArgs : Launch {
  DevGraph out, in;  // push and pull lists
  bool same;         // the same lists (a symmetric graph)
  const uint32_t* new_ids;  // null: not sorted
  uint32_t root;            // original id
  int64_t threshold;
  uint32_t* vis[2];   // visited bitmaps, (n+31)/32 words
  int32_t* depth;
  uint32_t* parents;  // null: not wanted
  int32_t* depth_out;  // original-id order; null: not wanted (or not sorted)
  Queues q[2];
  uint4* rest;  // a pulled level's pieces: vertex, edges [y, z)
  volatile uint64_t* info;  // mapped: rounds, reached, edges, done
};

// The first edge among [b, e) of a list whose neighbour is visited, as the neighbour;
// kNone: none.  The whole warp, the same in every lane.
__device__ __noinline__ uint32_t first_visited(const uint32_t* adj, const uint32_t* vis, uint32_t b, uint32_t e) {
  const int lane = threadIdx.x & 31;
  for (uint32_t x = b; x < e; x += 128) {
    uint32_t u[4];
    bool hit[4];
#pragma unroll
    for (int k = 0; k < 4; k++) u[k] = x + 32 * k + lane < e ? adj[x + 32 * k + lane] : kNone;
#pragma unroll
    for (int k = 0; k < 4; k++) hit[k] = u[k] != kNone && bit_test(vis, u[k]);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const unsigned hits = __ballot_sync(kAll, hit[k]);
      if (hits) return __shfl_sync(kAll, u[k], __ffs(hits) - 1);
    }
  }
  return kNone;
}

// The same for the rest of an unvisited vertex's list, which is put off where it is long.
__device__ __noinline__ uint32_t read_on(const uint32_t* adj, const uint32_t* vis, uint32_t b, uint32_t e, uint32_t v,
                                         uint4* rest, unsigned* nrest) {
  const int lane = threadIdx.x & 31;
  const uint32_t near = min(b + kRestList, e);
  const uint32_t f = first_visited(adj, vis, b, near);
  if (f != kNone || near == e) return f;
  const uint32_t pieces = (e - near + kRestPiece - 1) / kRestPiece;
  uint32_t at = 0;
  if (lane == 0) at = atomicAdd(nrest, pieces);
  at = __shfl_sync(kAll, at, 0);
  for (uint32_t p = lane; p < pieces; p += 32) {
    const uint32_t y = near + p * kRestPiece;
    rest[at + p] = make_uint4(v, y, min(y + kRestPiece, e), 0u);
  }
  return kNone;
}

// What a pulled level has put off.
__device__ __noinline__ void read_rest(const BfsArgs& A, uint32_t pieces, const uint32_t* vis, uint32_t* nvis,
                                       int32_t level, Shared* sh) {
  const uint32_t nwarps = gridDim.x * kFWarps;
  for (uint32_t i = blockIdx.x * kFWarps + (threadIdx.x >> 5); i < pieces; i += nwarps) {
    const uint4 it = A.rest[i];
    if (__any_sync(kAll, (__ldcg(nvis + (it.x >> 5)) >> (it.x & 31)) & 1u)) continue;  // found by another piece
    const uint32_t f = first_visited(A.in.adj, vis, it.y, it.z);
    const uint32_t bit = 1u << (it.x & 31);
    if (f != kNone && (threadIdx.x & 31) == 0 && !(atomicOr(nvis + (it.x >> 5), bit) & bit)) {
      A.depth[it.x] = level;
      if (A.parents) A.parents[it.x] = f;
      atomicAdd(&sh->count, 1u);
      atomicAdd(&sh->degsum, (unsigned long long)(A.out.off[it.x + 1] - A.out.off[it.x]));
    }
  }
}

// A push level claims vertices with an atomicOr on the visited bitmap; a pull
// level reads one bitmap and writes the other (a visited in-neighbour of an
// unvisited vertex is in the frontier, so visited is all a pull has to test) and, on
// a symmetric graph, marks vertices without edges visited, so that later pulls pass
// them by.
__global__ void __launch_bounds__(kFT, 1) bfs_fused(const __grid_constant__ BfsArgs A) {
  __shared__ Shared sh;
  __shared__ Member buf[kFWarps][kBuf];
  Grid grid;
  Appender<false> ap{buf[threadIdx.x >> 5], &sh, 0};
  begin(grid, &sh, A, A.ctl);
  const uint32_t n = A.out.n, nwords = (n + 31) / 32;
  const uint32_t tid = blockIdx.x * kFT + threadIdx.x, nthreads = gridDim.x * kFT;
  const int lane = threadIdx.x & 31;
  const uint32_t warp = tid >> 5, nwarps = nthreads >> 5;
  const uint32_t take = min((nwords + nwarps - 1) / nwarps, kPullWords);
  const uint32_t root = A.new_ids ? A.new_ids[A.root] : A.root;
  for (uint32_t i = tid; i < n; i += nthreads) {
    A.depth[i] = i == root ? 0 : -1;
    if (A.parents) A.parents[i] = i == root ? root : kNone;
  }
  for (uint32_t w = tid; w < nwords; w += nthreads) A.vis[0][w] = w == root >> 5 ? 1u << (root & 31) : 0u;
  if (warp == 0) {
    ap.add(lane == 0, root, A.out.off[root], A.out.off[root + 1], A.q[0], &A.ctl->lv[0], 0, 0);
    ap.finish(A.q[0], &A.ctl->lv[0], 0, 0);
  }
  if (!grid.sync(&A.ctl->lv[0])) return;
  int cv = 0;             // the bitmap that is current
  int cq = 0;             // the queue pair that holds the frontier
  bool queued = true;
  int32_t level = 0;
  unsigned long long reached = 0, edges = 0;
  for (;;) {
    Slot* cs = &A.ctl->lv[level % 3];
    Slot* ns = &A.ctl->lv[(level + 1) % 3];
    Slot c = sh.slot;
    if (c.count == 0) break;
    reached += c.count;
    edges += c.degsum;
    if (tid == 0) A.ctl->lv[(level + 2) % 3] = Slot{};
    // a symmetric graph's unvisited vertices hold the edges that no frontier had:
    // where those are fewer, looking at them is cheaper than the frontier's pushes
    const bool few = A.same && c.degsum > 2 * (A.out.m - edges) + n / 8;
    const bool pull = ((int64_t)(c.count + c.degsum) > A.threshold || few) && c.degsum > 0;
    level++;
    uint32_t* vis = A.vis[cv];
    if (pull) {
      uint32_t* nvis = A.vis[cv ^ 1];
      unsigned count = 0;
      unsigned long long degsum = 0;
      for (uint32_t w0 = warp; w0 < nwords; w0 += nwarps * take) {
        const uint32_t mw = w0 + lane * nwarps;
        const bool mine = lane < (int)take && mw < nwords;
        uint32_t word = mine ? vis[mw] : kNone;
        unsigned todo = __ballot_sync(kAll, (word | (mw == n >> 5 ? ~0u << (n & 31) : 0u)) != kNone);
        uint32_t next = word;
        while (todo) {
          // two words at a time: the chain offset - neighbour - its bit is all latency
          int j[2];
          j[0] = __ffs(todo) - 1;
          todo &= todo - 1;
          j[1] = todo ? __ffs(todo) - 1 : j[0];
          const bool two = todo != 0;
          todo &= todo - 1;
          uint32_t v[2], b[2], e[2], from[2];
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const uint32_t seen = __shfl_sync(kAll, word, j[i]);
            v[i] = (w0 + j[i] * nwarps) * 32 + lane;
            const bool want = (i == 0 || two) && v[i] < n && !((seen >> lane) & 1u);
            b[i] = want ? A.in.off[v[i]] : 0u;
            e[i] = want ? A.in.off[v[i] + 1] : 0u;
            from[i] = kNone;
            const unsigned alone = __ballot_sync(kAll, want && b[i] == e[i]);
            if (A.same && lane == j[i]) next |= alone;
          }
          // each lane tries its first 16 neighbours, four at a time; the lists
          // that are longer are then read by the whole warp, one at a time
          for (int t = 0; t < 4; t++) {
            uint32_t u[2][4];
            bool more = false;
#pragma unroll
            for (int i = 0; i < 2; i++) {
              const bool go = from[i] == kNone && b[i] < e[i];
              more |= go;
#pragma unroll
              for (int k = 0; k < 4; k++) u[i][k] = go && b[i] + k < e[i] ? A.in.adj[b[i] + k] : kNone;
            }
            if (!__any_sync(kAll, more)) break;
#pragma unroll
            for (int i = 0; i < 2; i++) {
              bool hit[4];
#pragma unroll
              for (int k = 0; k < 4; k++) hit[k] = u[i][k] != kNone && bit_test(vis, u[i][k]);
#pragma unroll
              for (int k = 3; k >= 0; k--) {
                if (hit[k]) from[i] = u[i][k];
              }
              b[i] = min(b[i] + 4, e[i]);
            }
          }
#pragma unroll
          for (int i = 0; i < 2; i++) {
            unsigned rest = __ballot_sync(kAll, from[i] == kNone && b[i] < e[i]);
            while (rest) {
              const int l = __ffs(rest) - 1;
              rest &= rest - 1;
              const uint32_t jb = __shfl_sync(kAll, b[i], l), je = __shfl_sync(kAll, e[i], l);
              const uint32_t u = jb + lane < je ? A.in.adj[jb + lane] : kNone;
              const unsigned hits = __ballot_sync(kAll, u != kNone && bit_test(vis, u));
              uint32_t f = hits ? __shfl_sync(kAll, u, __ffs(hits) - 1) : kNone;
              if (!hits && je - jb > 32) {
                f = read_on(A.in.adj, vis, jb + 32, je, __shfl_sync(kAll, v[i], l), A.rest, &ns->heavy);
              }
              if (lane == l) from[i] = f;
            }
            const bool won = from[i] != kNone;
            const unsigned now = __ballot_sync(kAll, won);
            if (lane == j[i]) next |= now;
            if (won) {
              A.depth[v[i]] = level;
              if (A.parents) A.parents[v[i]] = from[i];
              count++;
              degsum += A.out.off[v[i] + 1] - A.out.off[v[i]];
            }
          }
        }
        if (mine) nvis[mw] = next;
      }
      count = __reduce_add_sync(kAll, count);
      if (count) {
        degsum = warp_sum(degsum);
        if (lane == 0) {
          atomicAdd(&sh.count, count);
          atomicAdd(&sh.degsum, degsum);
        }
      }
      cv ^= 1;
      queued = false;
      if (!grid.sync(ns)) return;
      const uint32_t put_off = sh.slot.heavy;
      if (!put_off) continue;
      read_rest(A, put_off, vis, nvis, level, &sh);
    } else {
      if (!queued) {  // after a pull: the frontier is what it added to the bitmap
        const uint32_t* old = A.vis[cv ^ 1];
        for (uint32_t w0 = warp; w0 < nwords; w0 += nwarps * take) {
          const uint32_t mw = w0 + lane * nwarps;
          const uint32_t word = lane < (int)take && mw < nwords ? vis[mw] & ~old[mw] : 0u;
          for (unsigned todo = __ballot_sync(kAll, word != 0u); todo; todo &= todo - 1) {
            const int j = __ffs(todo) - 1;
            const uint32_t x = __shfl_sync(kAll, word, j);
            const uint32_t v = min((w0 + j * nwarps) * 32 + lane, n - 1);
            ap.add((x >> lane) & 1u, v, A.out.off[v], A.out.off[v + 1], A.q[cq], cs, 0, 0);
          }
        }
        ap.finish(A.q[cq], cs, 0, 0);
        if (!grid.sync()) return;  // (its members were counted by the pull)
        c = read_slot(cs);
        queued = true;
      }
      const Queues nq = A.q[cq ^ 1];
      expand(A.out, A.q[cq], 0, c.ns, 0, c.nl, blockIdx.x, gridDim.x, [&](const bool (&in)[4], uint32_t s, const uint32_t (&d)[4]) {
        bool won[4];
        uint32_t b[4] = {}, e[4] = {};
#pragma unroll
        for (int k = 0; k < 4; k++) won[k] = in[k] && !bit_test(vis, d[k]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (won[k]) {
            const uint32_t bit = 1u << (d[k] & 31);
            b[k] = A.out.off[d[k]];
            e[k] = A.out.off[d[k] + 1];
            won[k] = !(atomicOr(vis + (d[k] >> 5), bit) & bit);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (won[k]) {
            A.depth[d[k]] = level;
            if (A.parents) A.parents[d[k]] = s;
          }
          ap.add(won[k], d[k], b[k], e[k], nq, ns, 0, 0);
        }
      });
      ap.finish(nq, ns, 0, 0);
      cq ^= 1;
    }
    if (!grid.sync(ns)) return;
  }
  if (A.depth_out) {
    for (uint32_t i = tid; i < n; i += nthreads) A.depth_out[i] = A.depth[A.new_ids ? A.new_ids[i] : i];
  }
  if (tid == 0) {
    A.info[0] = (uint64_t)level;
    A.info[1] = reached;
    A.info[2] = edges;
    __threadfence_system();
    A.info[3] = 1;
  }
}

// ---------------------------------------------------------------------------
// BC, one source (BC-manyiter-v2.C:205-367)
// ---------------------------------------------------------------------------
struct BcArgs : Launch {
  DevGraph g;   // the lists the forward phase pushes along (the backward phase reads them the other way)
  DevGraph gt;  // the same edges by target
  bool same;    // g and gt are the same lists (a symmetric graph)
  bool long_lists;  // gt may hold lists above kLongList
  const uint32_t* new_ids;
  uint32_t source[64];  // original ids
  int k;
  bool rows;  // k independent sources, source s to row s of deps_out; else one source, whose dependencies add to deps
  int32_t* lvl;
  uint32_t* vis;  // the vertices reached, as bits: what a large push tests
  double *sigma, *even, *odd;  // path counts; dependencies of even and of odd levels
  double* inv;                 // 1/sigma of the vertices reached
  double* deps;                // a chain's dependencies so far
  double* deps_out;  // original-id order; null: deps keeps the result
  Queues q;          // every level's frontier, one after another
  uint32_t *first_small, *first_large;  // per level, levels + 1 entries
  unsigned long long* level_deg;        // per level: its degree sum
  uint4* heavy;                         // a pulled level's pieces of long lists
  size_t n_small, n_large, n_heavy;     // a group's share of the queues
  bool first_source;
  volatile uint64_t* info;  // mapped, four words per source (or summed over the calls): levels, edges, counts (rows), done
};

// Path counts are integers: doubles hold them below the first of these, 64-bit
// integers below the second.
constexpr double kExactCounts = 0x1p53, kIntegerCounts = 0x1p64;

constexpr uint32_t kLaneList = 16;    // a pull reads lists up to this with one lane,
constexpr uint32_t kLongList = 1024;  // up to this with the warp, and longer ones in pieces
constexpr uint32_t kLongPiece = 512;  // of this many edges

// Sum of sigma over the members of level r among edges [b, e) of a list, read by
// the whole warp; the same in every lane.
__device__ __forceinline__ double bc_level_sum(const BcArgs& A, const DevGraph& g, const double* val, uint32_t b,
                                               uint32_t e, int32_t r) {
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
  for (uint32_t e0 = b; e0 < e; e0 += 128) {
    uint32_t d[4];
    int32_t l[4];
#pragma unroll
    for (int k = 0; k < 4; k++) d[k] = e0 + 32 * k + lane < e ? g.adj[e0 + 32 * k + lane] : kNone;
#pragma unroll
    for (int k = 0; k < 4; k++) l[k] = d[k] != kNone ? A.lvl[d[k]] : -2;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (l[k] == r) acc += val[d[k]];
    }
  }
  return warp_sum(acc);
}

// A forward level as a pull: every vertex not reached yet sums the path counts of
// its predecessors in level r = level - 1.  False: a wait ran out.
__device__ bool bc_pull_level(const BcArgs& A, int32_t level, Slot* ns, uint32_t sn, uint32_t ln, Grid& grid,
                              Appender<true>& ap) {
  const uint32_t n = A.g.n, nwords = (n + 31) / 32;
  const int lane = threadIdx.x & 31;
  const uint32_t gwarp = (uint32_t)((threadIdx.x >> 5) * gridDim.x + blockIdx.x), nwarps = gridDim.x * kFWarps;
  for (uint32_t w = gwarp; w < nwords; w += nwarps) {
    const uint32_t v = w * 32 + lane;
    uint32_t b = 0, e = 0;
    if (v < n && !((A.vis[w] >> lane) & 1u)) {
      b = A.gt.off[v];
      e = A.gt.off[v + 1];
    }
    if (!__any_sync(kAll, b < e)) continue;
    double sum = 0.0;
    if (e - b <= kLaneList) {
      for (uint32_t x = b; x < e; x += 4) {
        uint32_t u[4];
        int32_t l[4];
#pragma unroll
        for (int k = 0; k < 4; k++) u[k] = x + k < e ? A.gt.adj[x + k] : kNone;
#pragma unroll
        for (int k = 0; k < 4; k++) l[k] = u[k] != kNone ? A.lvl[u[k]] : -2;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (l[k] == level - 1) sum += A.sigma[u[k]];
        }
      }
    }
    for (unsigned rest = __ballot_sync(kAll, e - b > kLaneList); rest; rest &= rest - 1) {
      const int j = __ffs(rest) - 1;
      const uint32_t jb = __shfl_sync(kAll, b, j), je = __shfl_sync(kAll, e, j);
      if (je - jb <= kLongList) {
        const double t = bc_level_sum(A, A.gt, A.sigma, jb, je, level - 1);
        if (lane == j) sum = t;
      } else {
        const uint32_t pieces = (je - jb + kLongPiece - 1) / kLongPiece;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&ns->heavy, pieces);
        at = __shfl_sync(kAll, at, 0);
        for (uint32_t p = lane; p < pieces; p += 32) {
          const uint32_t y = jb + p * kLongPiece;
          A.heavy[at + p] = make_uint4(w * 32 + j, y, min(y + kLongPiece, je), 0u);
        }
      }
    }
    const bool won = sum != 0.0;
    const unsigned now = __ballot_sync(kAll, won);
    if (lane == 0 && now) A.vis[w] |= now;
    uint32_t ob = 0, oe = 0;
    if (won) {
      A.lvl[v] = level;
      A.sigma[v] = sum;
      ob = A.g.off[v];
      oe = A.g.off[v + 1];
    }
    ap.add(won, v, ob, oe, A.q, ns, sn, ln);
  }
  if (!A.long_lists) return true;
  ap.finish(A.q, ns, sn, ln);
  // (its totals are not published yet: they stay in the CTA until the level ends)
  if (!grid.sync(nullptr, nullptr, true)) return false;
  const uint32_t heavy = __ldcg(&ns->heavy);
  for (uint32_t i = gwarp; i < heavy; i += nwarps) {
    const uint4 it = A.heavy[i];
    const double t = bc_level_sum(A, A.gt, A.sigma, it.y, it.z, level - 1);
    bool won = false;
    if (lane == 0 && t != 0.0) {
      atomicAdd(A.sigma + it.x, t);
      won = atomicCAS(A.lvl + it.x, -1, level) == -1;
      if (won) atomicOr(A.vis + (it.x >> 5), 1u << (it.x & 31));
    }
    ap.add(won, it.x, A.g.off[it.x], A.g.off[it.x + 1], A.q, ns, sn, ln);
  }
  return true;
}

// Forward: sigma is pushed along the frontier's edges to vertices of the next
// level or, where far fewer edges lead to vertices not reached yet, pulled by
// those.  Backward: a level's vertices sum the dependencies of their successors
// or, where the successors' level has far fewer edges, take them pushed (each
// direction examines an edge of the level it starts from; on R-MAT s22 the four
// large steps of pushes examine 2.5e8 edges, the cheaper directions 1.2e8).  The
// CTAs of one blockIdx.y are a group with arrays and a barrier of its own;
// independent sources are dealt out to the groups, whose waits and loads overlap.
__device__ bool bc_forward(const BcArgs& A, int s, Grid& grid, Appender<true>& ap, Shared& sh) {
  const uint32_t n = A.g.n;
  const uint32_t tid = blockIdx.x * kFT + threadIdx.x, nthreads = gridDim.x * kFT;
  const int lane = threadIdx.x & 31;
  const uint32_t src = A.new_ids ? A.new_ids[A.source[s]] : A.source[s];
  for (uint32_t i = tid; i < n; i += nthreads) {
    A.lvl[i] = i == src ? 0 : -1;
    A.sigma[i] = i == src ? 1.0 : 0.0;
    A.even[i] = A.odd[i] = 0.0;
  }
  for (uint32_t w = tid; w < (n + 31) / 32; w += nthreads) A.vis[w] = w == src >> 5 ? 1u << (src & 31) : 0u;
  if ((tid >> 5) == 0) {
    if (lane < 3) A.ctl->lv[lane] = Slot{};
    __syncwarp();
    ap.add(lane == 0, src, A.g.off[src], A.g.off[src + 1], A.q, &A.ctl->lv[0], 0, 0);
    ap.finish(A.q, &A.ctl->lv[0], 0, 0);
  }
  if (!grid.sync(&A.ctl->lv[0])) return false;
  uint32_t sbase = 0, lbase = 0;
  int32_t level = 0;
  unsigned long long edges = 0, seen = 0;  // examined; of vertices reached
  for (;;) {
    Slot* ns = &A.ctl->lv[(level + 1) % 3];
    const Slot c = sh.slot;
    if (tid == 0) {
      A.first_small[level] = sbase;
      A.first_large[level] = lbase;
      A.level_deg[level] = c.degsum;
    }
    if (c.count == 0) break;
    if (tid == 0) A.ctl->lv[(level + 2) % 3] = Slot{};
    level++;
    seen += c.degsum;
    const uint32_t sn = sbase + c.ns, ln = lbase + c.nl;  // where the next level's entries begin
    const unsigned long long rest = A.g.m - seen;  // edges of the vertices not reached yet
    if (A.same && c.degsum > 2 * rest + n / 8) {
      edges += rest;
      if (!bc_pull_level(A, level, ns, sn, ln, grid, ap)) return false;
    } else if (c.degsum >= n / 4) {
      // a large level: counts are added without claiming their targets (a claim
      // is an atomic that returns, and L1 lags behind the claims of other SMs, so
      // nearly every edge would make one), then one pass over the vertices finds
      // the ones that now have paths
      edges += c.degsum;
      expand(A.g, A.q, sbase, c.ns, lbase, c.nl, blockIdx.x, gridDim.x, [&](const bool (&in)[4], uint32_t u, const uint32_t (&d)[4]) {
        bool open[4];
#pragma unroll
        for (int k = 0; k < 4; k++) open[k] = in[k] && !bit_test(A.vis, d[k]);
        const double x = A.sigma[u];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (open[k]) atomicAdd(A.sigma + d[k], x);
        }
      });
      if (!grid.sync()) return false;
      for (uint32_t w0 = (tid & ~31u); w0 < n; w0 += nthreads) {
        const uint32_t v = min(w0 + lane, n - 1), old = A.vis[w0 >> 5];
        const bool won = w0 + lane < n && !((old >> lane) & 1u) && A.sigma[v] != 0.0;
        const unsigned now = __ballot_sync(kAll, won);
        if (lane == 0 && now) A.vis[w0 >> 5] = old | now;
        uint32_t b = 0, e = 0;
        if (won) {
          A.lvl[v] = level;
          b = A.g.off[v];
          e = A.g.off[v + 1];
        }
        ap.add(won, v, b, e, A.q, ns, sn, ln);
      }
    } else {
      edges += c.degsum;
      expand(A.g, A.q, sbase, c.ns, lbase, c.nl, blockIdx.x, gridDim.x, [&](const bool (&in)[4], uint32_t u, const uint32_t (&d)[4]) {
        int32_t l[4];
#pragma unroll
        for (int k = 0; k < 4; k++) l[k] = in[k] ? A.lvl[d[k]] : -2;
        const double x = A.sigma[u];
        uint32_t b[4] = {}, e[4] = {};
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (l[k] == -1) {
            b[k] = A.g.off[d[k]];
            e[k] = A.g.off[d[k] + 1];
            l[k] = atomicCAS(A.lvl + d[k], -1, level);
          } else if (l[k] != level) {
            l[k] = -2;
          }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {  // l: -1 reached here first, level reached by another edge, else not next
          if (l[k] >= -1) atomicAdd(A.sigma + d[k], x);
          if (l[k] == -1) atomicOr(A.vis + (d[k] >> 5), 1u << (d[k] & 31));
          ap.add(l[k] == -1, d[k], b[k], e[k], A.q, ns, sn, ln);
        }
      });
    }
    ap.finish(A.q, ns, sn, ln);
    sbase = sn;
    lbase = ln;
    if (!grid.sync(ns)) return false;
  }
  if (tid == 0) {  // (first_* and level_deg too: a barrier follows before anyone reads them)
    A.ctl->levels = level;
    A.ctl->edges = edges;
  }
  return true;
}

// The backward phase of source s, whose levels the group `A` holds, by `ctas` CTAs.
// The dependencies of even and of odd levels are kept apart: a vertex of level r finds
// its successors' among all its neighbours' in the other array (level r - 1 is still
// zero there), one gather per edge in place of a level and a value (8e6 vertices,
// 2^27 edges: 1460 -> 1380 us a call).
__device__ bool bc_backward(const BcArgs& A, int s, bool last, Grid& grid, uint32_t cta, uint32_t ctas) {
  const uint32_t n = A.g.n;
  const int lane = threadIdx.x & 31;
  const uint32_t tid = cta * kFT + threadIdx.x, nthreads = ctas * kFT;
  const uint32_t gwarp = (threadIdx.x >> 5) * ctas + cta, nwarps = ctas * kFWarps;
  const int32_t level = __ldcg(&A.ctl->levels);
  unsigned long long edges = __ldcg(&A.ctl->edges);
  // what the sources before left: it counts among a vertex's own
  const double* left = A.rows || (A.first_source && s == 0) ? nullptr : A.deps;
  for (int32_t r = level - 1; r >= 0; r--) {
    const uint32_t s0 = A.first_small[r], s1 = A.first_small[r + 1];
    const uint32_t l0 = A.first_large[r], l1 = A.first_large[r + 1];
    double* dep = r & 1 ? A.odd : A.even;
    const double* next = r & 1 ? A.even : A.odd;
    const bool deepest = r == level - 1;  // its vertices have no successors: 1/sigma alone
    const unsigned long long own = A.level_deg[r], below = deepest ? 0 : A.level_deg[r + 1];
    const bool push = A.same && !deepest && 4 * below < own;
    const bool alone = deepest || push;  // this level's edges are not read
    if (!deepest) edges += push ? below : own;
    if (push) {
      expand(A.g, A.q, s1, A.first_small[r + 2] - s1, l1, A.first_large[r + 2] - l1, cta, ctas,
             [&](const bool (&in)[4], uint32_t u, const uint32_t (&d)[4]) {
               int32_t l[4];
#pragma unroll
               for (int k = 0; k < 4; k++) l[k] = in[k] ? A.lvl[d[k]] : -2;
               const double x = next[u];
#pragma unroll
               for (int k = 0; k < 4; k++) {
                 if (l[k] == r) atomicAdd(dep + d[k], x);
               }
             });
    }
    // 1/sigma of the level's vertices, a lane each: GB300 issues one FP64 warp
    // instruction per 16 clocks, a division is ten of them, and beside the sums
    // one lane of the warp would do it
    const uint32_t gtid = gwarp * 32 + lane;
    for (uint32_t i = l0 + gtid; i < l1; i += nthreads) {
      const uint4 it = A.q.large[i];
      if (it.w & 1u) {
        const double x = 1.0 / A.sigma[it.x];
        A.inv[it.x] = x;
        atomicAdd(dep + it.x, left ? left[it.x] + x : x);
      }
    }
    if (alone) {
      for (uint32_t i = s0 + gtid; i < s1; i += nthreads) {
        const uint32_t u = A.q.small[i].x;
        const double x = 1.0 / A.sigma[u];
        A.inv[u] = x;
        const double own = left ? left[u] + x : x;
        if (push) atomicAdd(dep + u, own);  // beside the pushes
        else dep[u] = own;
      }
    } else {
      auto successors = [&](const uint32_t (&d)[4]) {  // the sum over those of d in the next level
        double x[4];
#pragma unroll
        for (int k = 0; k < 4; k++) x[k] = d[k] != kNone ? next[d[k]] : 0.0;
        return (x[0] + x[1]) + (x[2] + x[3]);
      };
      // four pieces per warp, their sums reduced together (one where there are few)
      const uint32_t each = l1 - l0 > nwarps ? 4 : 1;
      for (uint32_t i0 = l0 + gwarp * each; i0 < l1; i0 += nwarps * each) {
        double acc[4];
        uint32_t v = 0;  // the vertex of piece lane / 8
#pragma unroll
        for (int p = 0; p < 4; p++) {
          const uint4 it = p < (int)each && i0 + p < l1 ? A.q.large[i0 + p] : make_uint4(0, 0, 0, 0);
          if (lane / 8 == p) v = it.x;
          uint32_t d[4];
#pragma unroll
          for (int k = 0; k < 4; k++) d[k] = it.y + 32 * k + lane < it.z ? A.g.adj[it.y + 32 * k + lane] : kNone;
          acc[p] = successors(d);
        }
        const double z = warp_sum4(acc);
        if ((lane & 7) == 0 && z != 0.0) atomicAdd(dep + v, z);
      }
      // 8 vertices at a time, of 32 where the level has enough for every warp: one
      // division serves them
      const uint32_t per = s1 - s0 >= nwarps * 32 ? 4 : 1;
      const bool few = s1 - s0 <= nwarps;  // a vertex per warp, an edge per lane
      for (uint32_t i = s0 + gwarp; few && i < s1; i += nwarps) {
        const uint4 it = A.q.small[i];
        const double x = 1.0 / A.sigma[it.x];
        const uint32_t d = it.y + lane < it.z ? A.g.adj[it.y + lane] : kNone;
        const double acc = warp_sum(d != kNone ? next[d] : 0.0);
        if (lane == 0) {
          A.inv[it.x] = x;
          dep[it.x] = (left ? left[it.x] + x : x) + acc;
        }
      }
      for (uint32_t i = gwarp * per; !few && i < (s1 - s0 + 7) / 8; i += nwarps * per) {
        const uint32_t own = s0 + i * 8 + lane;
        const bool mine = own < s1 && lane < (int)per * 8;
        const uint32_t w = mine ? A.q.small[own].x : 0u;
        double x = mine ? A.sigma[w] : 1.0;
        if (per > 1) x = 1.0 / x;
        for (uint32_t t = 0; t < per; t++) {
          const uint32_t j = s0 + (i + t) * 8 + (lane >> 2);
          const uint4 it = j < s1 ? A.q.small[j] : make_uint4(0, 0, 0, 0);
          const uint32_t u = it.x, b = it.y, end = it.z;
          double acc = 0.0;
          for (uint32_t e0 = b + (lane & 3); __any_sync(kAll, e0 < end); e0 += 16) {
            uint32_t d[4];
#pragma unroll
            for (int k = 0; k < 4; k++) d[k] = e0 + 4 * k < end ? A.g.adj[e0 + 4 * k] : kNone;
            acc += successors(d);
          }
          acc += __shfl_xor_sync(kAll, acc, 1);
          acc += __shfl_xor_sync(kAll, acc, 2);
          if (per == 1) x = 1.0 / x;  // (a short chain: the division waits for nothing)
          const double y = __shfl_sync(kAll, x, t * 8 + (lane >> 2));
          if (j < s1 && (lane & 3) == 0) dep[u] = (left ? left[u] + y : y) + acc;
        }
        if (mine) A.inv[w] = x;
      }
    }
    if (!grid.sync()) return false;
  }
  // D = (D - 1/sigma) / (1/sigma), as bc_final forms it (unreached: NaN); by original
  // id for the caller (page-locked results: behind the host link)
  double* out = A.deps_out && last ? A.deps_out + (A.rows ? (size_t)s * n : 0) : nullptr;
  double* to = out ? out : A.deps;
  unsigned long long most = 0;  // the largest path count's bits
  for (uint32_t i = tid; i < n; i += nthreads) {
    const uint32_t v = out && A.new_ids ? A.new_ids[i] : i;
    const double d = A.even[v] + A.odd[v];  // one of them is 0; both: not reached
    const double count = A.sigma[v];
    to[i] = d != 0.0 ? (d - A.inv[v]) * count : CUDART_NAN;
    most = max(most, bits_of(count));
  }
  if (A.rows) {
    volatile unsigned char* counts = reinterpret_cast<volatile unsigned char*>(A.info + 4 * s + 2);
    const bool rounded = __any_sync(kAll, most >= bits_of(kExactCounts));
    const bool past_integers = __any_sync(kAll, most >= bits_of(kIntegerCounts));
    if (rounded && lane == 0) counts[past_integers] = 1;
  }
  if (tid == 0) {
    volatile uint64_t* f = A.info + (A.rows ? 4 * s : 0);
    f[0] += (uint64_t)level;
    f[1] += edges;
    __threadfence_system();
    f[3] += 1;
  }
  return true;
}

// The arrays of group y.  s: its source; a chain's odd sources run on the transposed
// graph (the reference transposes a directed graph after every source).
__device__ void bc_group(const BcArgs& P, size_t y, int s, BcArgs* A) {
  const size_t n = P.g.n;
  *A = P;
  if (!P.rows && s % 2 == 1) {
    A->g = P.gt;
    A->gt = P.g;
  }
  A->lvl += y * n;
  A->vis += y * ((n + 31) / 32);
  A->sigma += y * n;
  A->even += y * n;
  A->odd += y * n;
  A->inv += y * n;
  A->q.small += y * P.n_small;
  A->q.large += y * P.n_large;
  A->first_small += y * (n + 2);
  A->first_large += y * (n + 2);
  A->level_deg += y * (n + 2);
  A->heavy += y * P.n_heavy;
  A->ctl += y;
}

// Group y of CTAs (blockIdx.y) takes every gridDim.y-th source, on its own arrays.
// Independent sources (rows) never meet.  The sources of a chain add to the
// dependencies that the ones before left, so only their forward phases run side by
// side; then all CTAs take the backward phases one after another.
__global__ void __launch_bounds__(kFT, 1) bc_fused(const __grid_constant__ BcArgs P) {
  __shared__ Shared sh;
  __shared__ Member buf[kFWarps][kBuf];
  __shared__ BcArgs A;  // with the group's own arrays
  Grid grid;
  Appender<true> ap{buf[threadIdx.x >> 5], &sh, 0};
  begin(grid, &sh, P, P.ctl + blockIdx.y);
  if (threadIdx.x == 0) sh.team[1] = Team{&P.ctl->bar_all, 0, gridDim.x * gridDim.y};
  const int groups = gridDim.y;
  for (int s0 = 0; s0 < P.k; s0 += groups) {
    const int s = s0 + (int)blockIdx.y;
    if (P.rows && s >= P.k) return;
    if (s < P.k) {
      __syncthreads();
      if (threadIdx.x == 0) bc_group(P, blockIdx.y, s, &A);
      __syncthreads();
      if (!bc_forward(A, s, grid, ap, sh)) return;
    }
    Grid team = grid;
    team.which = P.rows ? 0 : 1;
    if (!team.sync()) return;
    const int first = P.rows ? s : s0, end = P.rows ? s + 1 : min(s0 + groups, P.k);
    for (int t = first; t < end; t++) {
      if (!P.rows && groups > 1) {
        __syncthreads();
        if (threadIdx.x == 0) bc_group(P, t - s0, t, &A);
        __syncthreads();
      }
      const uint32_t cta = P.rows ? blockIdx.x : blockIdx.y * gridDim.x + blockIdx.x;
      if (!bc_backward(A, t, P.rows || t == P.k - 1, team, cta, sh.team[team.which].ctas)) return;
      if (t + (P.rows ? groups : 1) < P.k && !team.sync()) return;  // the arrays are free for the next source
    }
  }
}

// ---------------------------------------------------------------------------
// Radii (Radii.C:140-218)
// ---------------------------------------------------------------------------
struct RadiiArgs : Launch {
  DevGraph out, in;
  const uint32_t* chunk_v;  // the pull lists' partition
  uint32_t nchunks;
  const uint32_t* new_ids;
  uint32_t seed[64];  // original ids, each once
  unsigned long long mask[64];
  int k;  // seeds
  int64_t threshold;
  unsigned long long *vis, *nvis;
  int32_t* radii;
  int32_t* radii_out;  // original-id order; null: not wanted (or not sorted)
  uint32_t* bits[2];  // what a pull reached
  Queues q[2];
  // multi-source BFS: bit q of plane p of v is bit p of v's depth from source q
  unsigned long long* planes;  // as many as the bits of the largest depth there can be
  int32_t* depths;  // sources rows of n, original-id order
  int sources;
  volatile uint64_t* info;  // mapped: rounds, edges, -, done
};
// Chunks of kSweepChunk edges per warp from which a dense round takes them whole
// (16 edges per lane, a quarter of the scans) instead of in steps of 128.
constexpr uint32_t kWideChunks = 2;
constexpr int kFewPlanes = 6;  // depths up to 63

// The vertex's new mask becomes current.
template <bool kDepths>
__device__ __forceinline__ void radii_advance(const RadiiArgs& A, uint32_t v, int32_t round, unsigned long long now,
                                              unsigned long long old) {
  if (kDepths) {
    const unsigned long long w = now & ~old;
    for (unsigned b = (unsigned)round; b; b &= b - 1) A.planes[(size_t)(__ffs(b) - 1) * A.out.n + v] |= w;
  }
  A.vis[v] = now;
}

// The depth rows from the planes: a warp takes 32 vertices and writes one whole
// line per source (a depth stored where it is found costs a line each, and a fill
// of every row before).
template <int kUsed>
__device__ __forceinline__ void write_depths(const RadiiArgs& A) {
  static_assert(kUsed <= kFewPlanes, "held in registers");
  const uint32_t n = A.out.n;
  const uint32_t tid = blockIdx.x * kFT + threadIdx.x, nthreads = gridDim.x * kFT;
  for (uint32_t i = tid; i < n; i += nthreads) {
    const uint32_t v = A.new_ids ? A.new_ids[i] : i;
    const unsigned long long seen = A.vis[v];
    unsigned long long pl[kUsed];
#pragma unroll
    for (int p = 0; p < kUsed; p++) pl[p] = A.planes[(size_t)p * n + v];
#pragma unroll
    for (int half = 0; half < 2; half++) {
      uint32_t s = (uint32_t)(seen >> (32 * half)), x[kUsed];
#pragma unroll
      for (int p = 0; p < kUsed; p++) x[p] = (uint32_t)(pl[p] >> (32 * half));
      const int end = min(32, A.sources - 32 * half);
      int32_t* row = A.depths + (size_t)(32 * half) * n + i;
      for (int q = 0; q < end; q++, row += n) {
        uint32_t d = 0;
#pragma unroll
        for (int p = 0; p < kUsed; p++) d |= ((x[p] >> q) & 1u) << p;
        *row = (s >> q) & 1u ? (int32_t)d : -1;
      }
    }
  }
}

// The same for deep searches, whose rounds cost far more than reading the planes a
// source at a time.
__device__ __noinline__ void write_depths_deep(const RadiiArgs& A, int used) {
  const uint32_t n = A.out.n;
  const uint32_t tid = blockIdx.x * kFT + threadIdx.x, nthreads = gridDim.x * kFT;
  for (uint32_t i = tid; i < n; i += nthreads) {
    const uint32_t v = A.new_ids ? A.new_ids[i] : i;
    const unsigned long long seen = A.vis[v];
    for (int q = 0; q < A.sources; q++) {
      uint32_t d = 0;
      for (int p = 0; p < used; p++) d |= (uint32_t)((A.planes[(size_t)p * n + v] >> q) & 1u) << p;
      A.depths[(size_t)q * n + i] = (seen >> q) & 1u ? (int32_t)d : -1;
    }
  }
}

__device__ __forceinline__ void radii_flush(const RadiiArgs& A, uint32_t* bits, uint32_t row, unsigned long long part) {
  const unsigned long long w = part & ~A.vis[row];
  if (!w) return;
  atomicOr(A.nvis + row, w);
  bit_set(bits, row);
}

// Rounds push over the queue or, dense ones, pull every row's neighbour masks
// (4 edges per lane, one segmented OR scan per 128 edges, as mask_pull_sweep
// with shorter steps: a small graph has more warps than 512-edge chunks).  A
// vertex pass after either makes the new masks current.  What a pull reached is
// queued only before a push.  kDepths: the same propagation, one bit per source, is a
// multi-source BFS (BFS.C); the bits that arrive in a round have that depth.
template <bool kDepths>
__global__ void __launch_bounds__(kFT, 1) radii_fused(const __grid_constant__ RadiiArgs A) {
  __shared__ Shared sh;
  __shared__ Member buf[kFWarps][kBuf];
  Grid grid;
  Appender<true> ap{buf[threadIdx.x >> 5], &sh, 0};
  begin(grid, &sh, A, A.ctl);
  const uint32_t n = A.out.n, nwords = (n + 31) / 32;
  const uint32_t tid = blockIdx.x * kFT + threadIdx.x, nthreads = gridDim.x * kFT;
  const int lane = threadIdx.x & 31;
  const uint32_t warp = tid >> 5, nwarps = nthreads >> 5;
  const uint32_t take = min((nwords + nwarps - 1) / nwarps, kPullWords);
  for (uint32_t i = tid; i < n; i += nthreads) {
    A.vis[i] = 0ull;
    A.nvis[i] = 0ull;
    A.radii[i] = -1;
  }
  for (uint32_t w = tid; w < nwords; w += nthreads) A.bits[0][w] = A.bits[1][w] = 0u;
  for (uint32_t c = tid; c < A.nchunks; c += nthreads) {
    if (A.chunk_v[c + 1] - A.chunk_v[c] > kPullRows) A.ctl->lv[0].heavy = 1;
  }
  unsigned long long full = 0ull;  // the bits that can spread: seeds with out-edges
  for (int j = lane; j < A.k; j += 32) {
    const uint32_t v = A.new_ids ? A.new_ids[A.seed[j]] : A.seed[j];
    if (A.out.off[v + 1] > A.out.off[v]) full |= A.mask[j];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) full |= __shfl_xor_sync(kAll, full, o);
  if (!grid.sync()) return;
  if (warp == 0) {
    for (int j0 = 0; j0 < 64; j0 += 32) {
      const int j = j0 + lane;
      uint32_t v = 0;
      if (j < A.k) {
        v = A.new_ids ? A.new_ids[A.seed[j]] : A.seed[j];
        A.vis[v] = A.nvis[v] = A.mask[j];
        A.radii[v] = 0;
      }
      ap.add(j < A.k, v, A.out.off[v], A.out.off[v + 1], A.q[0], &A.ctl->lv[0], 0, 0);
    }
    ap.finish(A.q[0], &A.ctl->lv[0], 0, 0);
  }
  if (!grid.sync(&A.ctl->lv[0])) return;
  const int64_t threshold = sh.slot.heavy ? INT64_MAX : A.threshold;
  int cq = 0;  // the queue pair that holds the frontier
  int cb = 0;  // the bitmap that holds it after a pull; a bitmap that does not is clear
  bool queued = true;
  int32_t round = 0;
  unsigned long long edges = 0;
  for (;;) {
    Slot* cs = &A.ctl->lv[round % 3];
    Slot* ns = &A.ctl->lv[(round + 1) % 3];
    Slot c = sh.slot;
    if (c.count == 0) break;
    edges += c.degsum;
    if (tid == 0) A.ctl->lv[(round + 2) % 3] = Slot{};
    round++;
    if (kDepths) {
      if ((round & (round - 1)) == 0) {  // the first round of a plane (a barrier lies before its first use)
        unsigned long long* pl = A.planes + (size_t)(31 - __clz(round)) * n;
        for (uint32_t i = tid; i < n; i += nthreads) pl[i] = 0ull;
      }
    }
    const Queues nq = A.q[cq ^ 1];
    if ((int64_t)(c.count + c.degsum) > threshold && A.in.m > 0) {
      uint32_t *bits = A.bits[cb ^ 1], *old_bits = A.bits[cb];
      const uint32_t steps = (A.in.m + 127) / 128;
      // a CTA's warps take its share as they get done: chunks whose rows are complete
      // cost next to nothing (16 of 140 us idle otherwise)
      auto take_next = [&]() {
        const uint32_t t = lane == 0 ? atomicAdd(&sh.taken, 1u) : 0u;
        return __shfl_sync(kAll, t, 0) * gridDim.x + blockIdx.x;
      };
      const bool wide = A.nchunks >= kWideChunks * nwarps;
      if (wide) {
        for (uint32_t c = take_next(); c < A.nchunks; c = take_next()) {
          mask_pull_chunk<16, false>(A.in, c, A.chunk_v[c], A.chunk_v[c + 1], A.vis, A.nvis, bits, full);
        }
      }
      for (uint32_t t = wide ? steps : take_next(); t < steps; t = take_next()) {
        const uint32_t e = t * 128 + lane * 4;
        const uint32_t ch = t / (kSweepChunk / 128);
        uint32_t row = kNone;
        unsigned long long part = 0ull;
        if (e < A.in.m) {
          const uint4 w = __ldg(reinterpret_cast<const uint4*>(A.in.adj + e));  // adj is padded past m
          const uint32_t u[4] = {w.x, w.y, w.z, w.w};
          row = upper_index(A.in.off, A.chunk_v[ch], A.chunk_v[ch + 1], e);
          uint32_t r = row, nxt = A.in.off[r + 1], rows[4];
          bool need[4];
          bool open = full == 0ull || (A.vis[r] & full) != full;
#pragma unroll
          for (int k = 0; k < 4; k++) {
            if (e + k < A.in.m && e + k >= nxt) {
              do { r++; nxt = A.in.off[r + 1]; } while (e + k >= nxt);
              open = full == 0ull || (A.vis[r] & full) != full;
            }
            rows[k] = r;
            need[k] = e + k < A.in.m && open;
          }
          unsigned long long x[4];
#pragma unroll
          for (int k = 0; k < 4; k++) x[k] = need[k] ? A.vis[u[k]] : 0ull;
#pragma unroll
          for (int k = 0; k < 4; k++) {
            if (rows[k] != row) {
              radii_flush(A, bits, row, part);
              part = 0ull;
              row = rows[k];
            }
            part |= x[k];
          }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long p = __shfl_up_sync(kAll, part, o);
          const uint32_t tr = __shfl_up_sync(kAll, row, o);
          if (lane >= o && tr == row) part |= p;
        }
        const uint32_t next_row = __shfl_down_sync(kAll, row, 1);
        if (row != kNone && (lane == 31 || next_row != row)) radii_flush(A, bits, row, part);
      }
      if (!grid.sync()) return;
      // the members' masks become current, two words of them at a time (a chain of
      // latencies); they are queued only if the next round pushes
      unsigned count = 0;
      unsigned long long degsum = 0;
      for (uint32_t w0 = warp; w0 < nwords; w0 += nwarps * take) {
        const uint32_t mw = w0 + lane * nwarps;
        const bool mine = lane < (int)take && mw < nwords;
        const uint32_t word = mine ? bits[mw] : 0u;
        if (mine && !queued) old_bits[mw] = 0u;
        unsigned todo = __ballot_sync(kAll, word != 0u);
        while (todo) {
          int j[2];
          j[0] = __ffs(todo) - 1;
          todo &= todo - 1;
          j[1] = todo ? __ffs(todo) - 1 : j[0];
          const bool two = todo != 0;
          todo &= todo - 1;
          uint32_t v[2];
          bool in[2];
          unsigned long long now[2], old[2];
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const uint32_t x = __shfl_sync(kAll, word, j[i]);
            v[i] = (w0 + j[i] * nwarps) * 32 + lane;
            in[i] = (i == 0 || two) && ((x >> lane) & 1u);
            now[i] = in[i] ? A.nvis[v[i]] : 0ull;
            old[i] = kDepths && in[i] ? A.vis[v[i]] : 0ull;
            if (in[i]) degsum += A.out.off[v[i] + 1] - A.out.off[v[i]];
            count += in[i];
          }
#pragma unroll
          for (int i = 0; i < 2; i++) {
            if (!in[i]) continue;
            A.radii[v[i]] = round;
            radii_advance<kDepths>(A, v[i], round, now[i], old[i]);
          }
        }
      }
      count = __reduce_add_sync(kAll, count);
      if (count) {
        degsum = warp_sum(degsum);
        if (lane == 0) {
          atomicAdd(&sh.count, count);
          atomicAdd(&sh.degsum, degsum);
        }
      }
      cb ^= 1;
      queued = false;
      if (!grid.sync(ns)) return;
    } else {
      if (!queued) {  // after a pull
        uint32_t* bits = A.bits[cb];
        for (uint32_t w0 = warp; w0 < nwords; w0 += nwarps * take) {
          const uint32_t mw = w0 + lane * nwarps;
          const bool mine = lane < (int)take && mw < nwords;
          const uint32_t word = mine ? bits[mw] : 0u;
          if (word) bits[mw] = 0u;
          for (unsigned todo = __ballot_sync(kAll, word != 0u); todo; todo &= todo - 1) {
            const int j = __ffs(todo) - 1;
            const uint32_t x = __shfl_sync(kAll, word, j);
            const uint32_t v = min((w0 + j * nwarps) * 32 + lane, n - 1);
            ap.add((x >> lane) & 1u, v, A.out.off[v], A.out.off[v + 1], A.q[cq], cs, 0, 0);
          }
        }
        ap.finish(A.q[cq], cs, 0, 0);
        if (!grid.sync()) return;  // (its members were counted by the pull)
        c = read_slot(cs);
        queued = true;
      }
      expand(A.out, A.q[cq], 0, c.ns, 0, c.nl, blockIdx.x, gridDim.x, [&](const bool (&in)[4], uint32_t s, const uint32_t (&d)[4]) {
        unsigned long long vd[4];
#pragma unroll
        for (int k = 0; k < 4; k++) vd[k] = in[k] ? A.vis[d[k]] : ~0ull;
        const unsigned long long ms = A.vis[s];
        bool won[4];
        uint32_t b[4] = {}, e[4] = {};
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const unsigned long long w = ms & ~vd[k];
          won[k] = w != 0ull;
          if (w) {
            atomicOr(A.nvis + d[k], w);
            won[k] = A.radii[d[k]] != round;
          }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (won[k]) {
            b[k] = A.out.off[d[k]];
            e[k] = A.out.off[d[k] + 1];
            won[k] = atomicExch(A.radii + d[k], round) != round;
          }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) ap.add(won[k], d[k], b[k], e[k], nq, ns, 0, 0);
      });
      ap.finish(nq, ns, 0, 0);
      if (!grid.sync(ns)) return;
      const Slot nx = sh.slot;
      for (uint32_t i = tid; i < nx.ns; i += nthreads) {
        const uint32_t v = nq.small[i].x;
        radii_advance<kDepths>(A, v, round, A.nvis[v], A.vis[v]);
      }
      for (uint32_t i = tid; i < nx.nl; i += nthreads) {
        const uint4 it = nq.large[i];
        if (it.w & 1u) radii_advance<kDepths>(A, it.x, round, A.nvis[it.x], A.vis[it.x]);
      }
      if (!grid.sync()) return;
    }
    cq ^= 1;
  }
  if (kDepths) {
    switch (32 - __clz(round)) {
      case 1: write_depths<1>(A); break;
      case 2: write_depths<2>(A); break;
      case 3: write_depths<3>(A); break;
      case 4: write_depths<4>(A); break;
      case 5: write_depths<5>(A); break;
      case 6: write_depths<6>(A); break;
      default: write_depths_deep(A, 32 - __clz(round)); break;
    }
  }
  if (A.radii_out) {
    for (uint32_t i = tid; i < n; i += nthreads) A.radii_out[i] = A.radii[A.new_ids ? A.new_ids[i] : i];
  }
  if (tid == 0) {
    A.info[0] = (uint64_t)round;
    A.info[1] = edges;
    __threadfence_system();
    A.info[3] = 1;
  }
}

// ---------------------------------------------------------------------------
// PageRank (PageRank.C:120-189), the exact-sum pull of pagerank.cu
// ---------------------------------------------------------------------------
struct PrArgs : Launch {
  DevGraph in;
  const uint32_t* out_off;
  const uint32_t* chunk_v;
  const uint32_t* new_ids;
  uint32_t* lane_row;    // the row of every lane's first edge
  U128 *opens, *closes;  // per warp step: the piece of the row that goes on past it, and of the one that began before it
  double* p;
  double* contrib[2];  // read by even and by odd iterations
  unsigned long long* rmag;
  double* ranks_out;  // original-id order; null: not wanted (or not sorted)
  L1Sum* l1;          // per iteration
  uint32_t row_weight;  // a row counts as this many edges when rows are shared out
  int64_t max_iters;
  double p0, added;
  volatile uint64_t* info;  // mapped: iterations run, last L1 (2 words), done, broke
};

constexpr uint32_t kPrStep = 128;  // edges per warp step, four per lane

// PR_Vertex_F, the L1 term and the next contribution of one vertex.
__device__ __forceinline__ void pr_vertex(const PrArgs& A, uint32_t v, const U128& sum, uint32_t deg, double* next,
                                          U128& l1) {
  const bool has = (sum.lo | sum.hi) != 0ull;
  const double pn = has ? fma(kPrDamp, fx_to_double(sum), A.added) : A.added;
  const double po = A.p[v];
  if (bits_of(po) != bits_of(pn)) add128(l1, fx_from_double(fabs(po - pn)));
  A.p[v] = pn;
  // p'/deg by degree class (pr_quotient's; the reciprocals are written by this
  // kernel, so they are read as plain memory)
  if (deg == 0) next[v] = 0.0;
  else if ((deg & (deg - 1)) == 0) next[v] = double_of(bits_of(pn) - ((unsigned long long)(31 - __clz(deg)) << 52));
  else next[v] = div_by_magic(pn, deg, A.rmag[v]);
}

// One warp step: edges [s0, s0 + kPrStep) that lie in [elo, ehi), the edges of
// the CTA's rows.  pr_pull_sweep's step with four edges per lane (a small graph
// has few steps, so short ones keep more warps busy) and the row of a lane's
// first edge read instead of searched for.  A row inside the step is stored to
// acc; a row that it shares with other steps leaves its piece in opens (it
// begins here) or closes (it began before), which the row's thread adds up.
__device__ __forceinline__ void pr_step(const PrArgs& A, const double* c, uint32_t s0, uint32_t elo, uint32_t ehi,
                                        const uint32_t* rows, U128* acc, uint32_t lo, U128* opens, U128* closes) {
  const int lane = threadIdx.x & 31;
  const DevGraph& g = A.in;
  const uint32_t e = s0 + lane * 4, begin = max(s0, elo);
  uint32_t row = kNone, head_row = kNone;
  U128 part{0ull, 0ull}, head{0ull, 0ull};
  bool cont = false;
  if (e < ehi && e + 4 > elo) {
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(g.adj + e));  // adj is padded past m
    uint32_t v = rows[lane];
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
    double x[4];
#pragma unroll
    for (int j = 0; j < 4; j++) x[j] = e + j >= elo && e + j < ehi ? c[u[j]] : 0.0;
    uint32_t nxt = g.off[v + 1];
    const bool before = g.off[v] < e;
    row = v;
    bool at_first = true;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t ee = e + j;
      if (ee < elo || ee >= ehi) continue;
      if (ee >= nxt) {
        if (at_first && before) {
          head = part;
          head_row = row;
        } else {
          acc[row - lo] = part;
        }
        at_first = false;
        part = U128{0ull, 0ull};
        do { v++; nxt = g.off[v + 1]; } while (ee >= nxt);
        row = v;
      }
      add128(part, fx_from_double(x[j]));
    }
    cont = nxt > e + 4;
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const U128 y = shfl_up128(part, o);
    const uint32_t tr = __shfl_up_sync(kAll, row, o);
    if (lane >= o && tr == row) add128(part, y);
  }
  const U128 prev = shfl_up128(part, 1);
  const uint32_t prev_row = __shfl_up_sync(kAll, row, 1);
  if (head_row != kNone) {
    if (lane > 0 && prev_row == head_row) add128(head, prev);
    if (g.off[head_row] >= begin) acc[head_row - lo] = head;
    else *closes = head;
  }
  if (row != kNone && (!cont || lane == 31)) {
    const bool here = g.off[row] >= begin;
    if (!here) *closes = part;
    else if (cont) *opens = part;
    else acc[row - lo] = part;
  }
}

// Each CTA owns a run of rows of about the same number of edges and rows and
// keeps their sums in shared memory, so an iteration is one pass over its
// edges, one over its rows and one grid barrier: contributions are read from
// one array and written to the other.  The sums are exact (pr_exact.cuh).
__global__ void __launch_bounds__(kFT, 1) pagerank_fused(const __grid_constant__ PrArgs A) {
  __shared__ Shared sh;
  __shared__ uint32_t s_range[2];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  U128* acc = reinterpret_cast<U128*>(smem_raw);
  Grid grid;
  begin(grid, &sh, A, A.ctl);
  const uint32_t n = A.in.n, m = A.in.m;
  const uint32_t tid = blockIdx.x * kFT + threadIdx.x, nthreads = gridDim.x * kFT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 2) {  // first row whose edges and rows before reach this CTA's (and the next one's) share
    const uint64_t want = ((uint64_t)m + (uint64_t)n * A.row_weight) * (blockIdx.x + threadIdx.x) / gridDim.x;
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if (A.in.off[mid] + (uint64_t)mid * A.row_weight >= want) hi = mid;
      else lo = mid + 1;
    }
    s_range[threadIdx.x] = lo;
  }
  __syncthreads();
  const uint32_t lo = s_range[0], hi = s_range[1];
  const uint32_t elo = A.in.off[lo], ehi = A.in.off[hi], base = elo & ~3u;
  const uint32_t steps = ehi > elo ? (ehi - base + kPrStep - 1) / kPrStep : 0;
  // the CTA's part of the per-lane and per-step arrays: CTAs share at most one
  // group of four edges, so shifting each by one keeps them apart
  uint32_t* rows = A.lane_row + (base / 4 + blockIdx.x * 32);
  U128* opens = A.opens + (base / kPrStep + 2 * blockIdx.x);
  U128* closes = A.closes + (base / kPrStep + 2 * blockIdx.x);
  for (uint32_t v = lo + threadIdx.x; v < hi; v += kFT) {
    A.p[v] = A.p0;
    const uint32_t d = A.out_off[v + 1] - A.out_off[v];
    const unsigned long long R = (d & (d - 1)) ? recip_magic(d) : 0ull;
    A.contrib[0][v] = deg_quotient(A.p0, d, R);
    A.rmag[v] = R;
  }
  for (uint32_t i = threadIdx.x; i < steps * 32; i += kFT) {
    const uint32_t e = max(base + i * 4, elo);
    if (e < ehi) {
      const uint32_t ch = e / kSweepChunk;
      rows[i] = upper_index(A.in.off, A.chunk_v[ch], A.chunk_v[ch + 1], e);
    }
  }
  for (int64_t i = tid; i < A.max_iters; i += nthreads) A.l1[i] = L1Sum{};
  if (!grid.sync()) return;
  const U128 eps = pr_eps_fx();
  U128 last{0ull, 0ull};
  int64_t it = 0;
  bool broke = false;
  while (it < A.max_iters && !broke) {
    const double* c = A.contrib[it & 1];
    double* next = A.contrib[(it & 1) ^ 1];
    for (uint32_t t = warp; t < steps; t += kFWarps) {
      pr_step(A, c, base + t * kPrStep, elo, ehi, rows + t * 32, acc, lo, opens + t, closes + t);
    }
    __syncthreads();
    U128 local{0ull, 0ull};
    for (uint32_t v0 = lo + warp * 32; v0 < hi; v0 += kFT) {
      const uint32_t v = v0 + lane;
      U128 sum{0ull, 0ull};
      uint32_t first = 0, end = 0;  // steps whose `closes` hold pieces of the row
      if (v < hi) {
        const uint32_t b = A.in.off[v], e = A.in.off[v + 1];
        if (e > b) {
          const uint32_t s1 = (b - base) / kPrStep, s2 = (e - 1 - base) / kPrStep;
          sum = s1 == s2 ? acc[v - lo] : opens[s1];
          first = s1 + 1;
          end = s2 + 1;
        }
      }
      unsigned many = __ballot_sync(kAll, end > first + 8);  // long rows: the warp adds their pieces together
      while (many) {
        const int j = __ffs(many) - 1;
        many &= many - 1;
        const uint32_t jf = __shfl_sync(kAll, first, j), je = __shfl_sync(kAll, end, j);
        U128 s{0ull, 0ull};
        for (uint32_t k = jf + lane; k < je; k += 32) add128(s, closes[k]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          add128(s, U128{__shfl_xor_sync(kAll, s.lo, o), __shfl_xor_sync(kAll, s.hi, o)});
        }
        if (lane == j) {
          add128(sum, s);
          first = end;
        }
      }
      for (; first < end; first++) add128(sum, closes[first]);
      if (v < hi) pr_vertex(A, v, sum, A.out_off[v + 1] - A.out_off[v], next, local);
    }
    const U128 t = block_sum128(local);
    if (threadIdx.x == 0 && (t.lo | t.hi)) A.l1[it].add(t);
    if (!grid.sync(nullptr, A.l1 + it)) return;
    last = sh.l1;
    broke = less128(last, eps);
    it++;
  }
  if (A.ranks_out) {
    for (uint32_t i = tid; i < n; i += nthreads) A.ranks_out[i] = A.p[A.new_ids ? A.new_ids[i] : i];
  }
  if (tid == 0) {
    A.info[0] = (uint64_t)it;
    A.info[1] = last.lo;
    A.info[2] = last.hi;
    A.info[4] = broke ? 1 : 0;
    __threadfence_system();
    A.info[3] = 1;
  }
}

// ---------------------------------------------------------------------------
// PageRankDelta (PageRankDelta.C:98-155)
// ---------------------------------------------------------------------------
struct PrdArgs : Launch {
  DevGraph out, in;
  const uint32_t* new_ids;
  double *p, *ngh, *c;
  uint32_t* bits;  // the frontier, as the last filter left it
  uint32_t* touched;  // the vertices that a short push reached (0 between rounds)
  Queues rows;     // every row with in-edges (whole runs only)
  Queues q[2];
  int64_t start;   // rounds already run level by level (0: a whole run)
  int64_t max_iters;
  int64_t threshold;
  int64_t short_push;  // edges up to which a push notes what it reaches
  bool allow_pull;
  double one_over_n, added;
  double* ranks_out;  // original-id order; null: not wanted (or not sorted)
  volatile uint64_t* info;  // mapped: rounds, L1 (bits), edges, done
};

// A round pushes the frontier's contributions or, a dense one, sums every row's
// (c is 0 outside the frontier); a filter pass over the vertices then forms the
// next frontier as prd_filter does, skipping words that nothing reached and that
// held no member.  A run can be taken over after its dense first rounds, which
// large graphs sweep with a launch of their own.
//
// A round of few edges is a chain of latencies: two grid barriers, the push and the
// filter.  Its push notes the vertices that it reaches, so that the filter looks at
// up to 1024 vertices at a time and loads only what has changed: reading every sum
// instead, a word after the other, was most of such a round (2^21 vertices, 14
// rounds: 270 us).
__global__ void __launch_bounds__(kFT, 1) prd_fused(const __grid_constant__ PrdArgs A) {
  __shared__ Shared sh;
  __shared__ Member buf[kFWarps][kBuf];
  __shared__ double s_l1[kFWarps];
  Grid grid;
  Appender<false> ap{buf[threadIdx.x >> 5], &sh, 0};
  begin(grid, &sh, A, A.ctl);
  const uint32_t n = A.out.n, nwords = (n + 31) / 32;
  const uint32_t tid = blockIdx.x * kFT + threadIdx.x, nthreads = gridDim.x * kFT;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t warp = tid >> 5, nwarps = nthreads >> 5;
  uint32_t rs = 0, rl = 0;  // entries of the row queues
  if (A.start == 0) {
    for (uint32_t w = warp; w < nwords; w += nwarps) {
      const bool in = w * 32 + lane < n;
      const uint32_t v = in ? w * 32 + lane : n - 1;
      if (in) {
        A.p[v] = 0.0;
        A.ngh[v] = 0.0;
        const uint32_t d = A.out.off[v + 1] - A.out.off[v];
        A.c[v] = d ? A.one_over_n / d : 0.0;
      }
      if (lane == 0) A.bits[w] = A.touched[w] = 0u;
      const uint32_t b = A.in.off[v], e = A.in.off[v + 1];
      ap.add(in && e > b, v, b, e, A.rows, &A.ctl->lv[3], 0, 0);
    }
    ap.finish(A.rows, &A.ctl->lv[3], 0, 0);
    if (!grid.sync()) return;
    const Slot r = read_slot(&A.ctl->lv[3]);
    rs = r.ns;
    rl = r.nl;
    if (threadIdx.x == 0) {
      sh.slot = Slot{};  // every vertex starts in the frontier
      sh.slot.count = n;
      sh.slot.degsum = A.out.m;
    }
    __syncthreads();
  } else {
    for (uint32_t w = warp; w < nwords; w += nwarps) {
      const uint32_t x = A.bits[w];
      if (lane == 0) A.touched[w] = 0u;
      if (!x) continue;
      const uint32_t v = min(w * 32 + lane, n - 1);
      ap.add((x >> lane) & 1u, v, A.out.off[v], A.out.off[v + 1], A.q[0], &A.ctl->lv[0], 0, 0);
    }
    ap.finish(A.q[0], &A.ctl->lv[0], 0, 0);
    if (!grid.sync(&A.ctl->lv[0])) return;
  }
  int cq = 0;
  int64_t k = 0, round = A.start;  // k: rounds of this launch
  unsigned long long edges = 0;
  double l1 = 0.0;
  while (round++ < A.max_iters) {
    const Slot c = sh.slot;
    Slot* ns = &A.ctl->lv[(k + 1) % 3];
    if (tid == 0) A.ctl->lv[(k + 2) % 3] = Slot{};
    k++;
    edges += c.degsum;
    const bool whole = A.start == 0 && k == 1;  // the queue does not hold the first frontier of a whole run
    const bool pull = whole || (A.start == 0 && A.allow_pull && (int64_t)(c.count + c.degsum) > A.threshold);
    const bool noted = !pull && (int64_t)c.degsum <= A.short_push;
    if (pull) {
      const uint32_t gwarp = (uint32_t)(wid * gridDim.x + blockIdx.x);
      for (uint32_t i0 = gwarp * 4; i0 < rl; i0 += nwarps * 4) {
        double acc[4];
        uint4 mine = make_uint4(0, 0, 0, 0);  // piece lane / 8
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const uint4 it = i0 + q < rl ? A.rows.large[i0 + q] : make_uint4(0, 0, 0, 0);
          if (lane / 8 == q) mine = it;
          uint32_t u[4];
          double x[4];
#pragma unroll
          for (int j = 0; j < 4; j++) u[j] = it.y + 32 * j + lane < it.z ? A.in.adj[it.y + 32 * j + lane] : kNone;
#pragma unroll
          for (int j = 0; j < 4; j++) x[j] = u[j] != kNone ? A.c[u[j]] : 0.0;
          acc[q] = (x[0] + x[1]) + (x[2] + x[3]);
        }
        const double s = warp_sum4(acc);
        if ((lane & 7) == 0 && i0 + lane / 8 < rl) {
          if (mine.w == 3u) A.ngh[mine.x] = s;  // the row's only piece
          else if (s != 0.0) atomicAdd(A.ngh + mine.x, s);
        }
      }
      for (uint32_t i = gwarp; i < (rs + 7) / 8; i += nwarps) {
        const uint32_t j = i * 8 + (lane >> 2);
        const uint4 it = j < rs ? A.rows.small[j] : make_uint4(0, 0, 0, 0);
        double s = 0.0;
        for (uint32_t e0 = it.y + (lane & 3); __any_sync(kAll, e0 < it.z); e0 += 16) {
          uint32_t u[4];
          double x[4];
#pragma unroll
          for (int q = 0; q < 4; q++) u[q] = e0 + 4 * q < it.z ? A.in.adj[e0 + 4 * q] : kNone;
#pragma unroll
          for (int q = 0; q < 4; q++) x[q] = u[q] != kNone ? A.c[u[q]] : 0.0;
          s += (x[0] + x[1]) + (x[2] + x[3]);
        }
        s += __shfl_xor_sync(kAll, s, 1);
        s += __shfl_xor_sync(kAll, s, 2);
        if (j < rs && (lane & 3) == 0) A.ngh[it.x] = s;
      }
    } else {
      expand(A.out, A.q[cq], 0, c.ns, 0, c.nl, blockIdx.x, gridDim.x, [&](const bool (&in)[4], uint32_t s, const uint32_t (&d)[4]) {
        const double x = A.c[s];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (in[j]) {
            atomicAdd(A.ngh + d[j], x);
            if (noted) atomicOr(A.touched + (d[j] >> 5), 1u << (d[j] & 31));
          }
        }
      });
    }
    if (!grid.sync()) return;
    const Queues nq = A.q[cq ^ 1];
    double local = 0.0;
    auto filter = [&](uint32_t w) {
      const bool in = w * 32 + lane < n;
      const uint32_t v = in ? w * 32 + lane : n - 1;
      const double g = in ? A.ngh[v] : 0.0;
      // nothing arrived and nobody was active: delta is 0, the vertex stays as it is
      if (!noted && round > 1 && !A.bits[w] && !__any_sync(kAll, g != 0.0)) return;
      bool act = false;
      uint32_t b = 0, e = 0;
      if (in) {
        b = A.out.off[v];
        e = A.out.off[v + 1];
        double pv = A.p[v], d;
        if (round == 1) {  // PageRankDelta.C:46-61
          d = __dadd_rn(__dmul_rn(kPrDamp, g), A.added);
          pv = __dadd_rn(pv, d);
          d = __dsub_rn(d, A.one_over_n);
          act = fabs(d) > __dmul_rn(kPrdEps2, pv);
          A.p[v] = pv;
        } else {  // PageRankDelta.C:63-76
          d = __dmul_rn(g, kPrDamp);
          act = fabs(d) > __dmul_rn(kPrdEps2, pv);
          if (act) A.p[v] = __dadd_rn(pv, d);
        }
        A.ngh[v] = 0.0;
        A.c[v] = (act && e > b) ? __ddiv_rn(d, (double)(e - b)) : 0.0;
        local += fabs(d);
      }
      const unsigned now = __ballot_sync(kAll, act);
      if (lane == 0) A.bits[w] = now;
      ap.add(act, v, b, e, nq, ns, 0, 0);
    };
    if (noted) {
      const uint32_t take = min((nwords + nwarps - 1) / nwarps, 32u);  // words a warp looks at together
      for (uint32_t w0 = warp * take; w0 < nwords; w0 += nwarps * take) {
        const uint32_t w = w0 + lane;
        const bool mine = lane < (int)take && w < nwords;
        const uint32_t t = mine ? A.touched[w] : 0u;
        unsigned todo = __ballot_sync(kAll, t || (mine && A.bits[w]));
        if (t) A.touched[w] = 0u;
        for (; todo; todo &= todo - 1) filter(w0 + __ffs(todo) - 1);
      }
    } else {
      for (uint32_t w = warp; w < nwords; w += nwarps) filter(w);
    }
    ap.finish(nq, ns, 0, 0);
    local = warp_sum(local);
    if (lane == 0) s_l1[wid] = local;
    __syncthreads();
    if (wid == 0) {
      const double t = warp_sum(s_l1[lane]);
      if (lane == 0 && t != 0.0) atomicAdd(&ns->l1, t);
    }
    if (!grid.sync(ns)) return;
    l1 = sh.slot.l1;
    if (l1 < kPrdEps) break;  // PageRankDelta.C:144
    cq ^= 1;
  }
  if (A.ranks_out) {
    for (uint32_t i = tid; i < n; i += nthreads) A.ranks_out[i] = A.p[A.new_ids ? A.new_ids[i] : i];
  }
  if (tid == 0) {
    A.info[0] = (uint64_t)round;
    A.info[1] = bits_of(l1);
    A.info[2] = edges;
    __threadfence_system();
    A.info[3] = 1;
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// The largest in-degree of g (found once per graph); n if it cannot be found.
__global__ void find_max_degree(const uint32_t* __restrict__ off, uint32_t n, unsigned int* out) {
  unsigned int mx = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    mx = max(mx, off[v + 1] - off[v]);
  }
  mx = __reduce_max_sync(kAll, mx);
  if ((threadIdx.x & 31) == 0) atomicMax(out, mx);
}

__global__ void find_max_chunk(const uint32_t* __restrict__ chunk_v, uint32_t nchunks, unsigned int* out) {
  unsigned int mx = 0;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < nchunks; c += gridDim.x * blockDim.x) {
    mx = max(mx, chunk_v[c + 1] - chunk_v[c]);
  }
  mx = __reduce_max_sync(kAll, mx);
  if ((threadIdx.x & 31) == 0) atomicMax(out, mx);
}

// A value that `find` leaves in a zeroed word, kept in `known`; `unknown` on an error.
template <class Find>
int64_t found_once(std::atomic<int64_t>& known, int64_t unknown, cudaStream_t st, Find find) {
  int64_t v = known.load(std::memory_order_relaxed);
  if (v >= 0) return v;
  unsigned int* d = reinterpret_cast<unsigned int*>(ctx().ws.counters.as<uint64_t>() + 8);  // a free scratch word
  uint32_t h = 0;
  cudaError_t e = cudaMemsetAsync(d, 0, 4, st);
  if (e == cudaSuccess) {
    find(d);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess || read_small(d, &h, 4, st) != RG_OK) {
    cudaGetLastError();
    return unknown;
  }
  known.store(h, std::memory_order_relaxed);
  return h;
}

int64_t max_in_degree(const rg_graph* g, cudaStream_t st) {
  if (!g->directed) return g->max_deg;
  return found_once(g->max_in_deg, g->n, st, [&](unsigned int* d) {  // (n: too large a row for the one-launch path)
    find_max_degree<<<64, 256, 0, st>>>(g->in_view().off, (uint32_t)g->n, d);
  });
}

// The arrays of one launch, in the thread's one allocation: large ones on whole
// pages.  (Allocated one by one, their placement after earlier allocations of the
// process moved BFS on 2^24 vertices between 1.02 and 1.13 ms.)
// It is kept for the thread's next call.
struct Arena {
  DevBuf buf;
  int device = -1;
  bool in_use = false;  // a call's launches may be reading and writing it
};
thread_local Arena g_arena;

class Arrays {
 public:
  Arrays() = default;
  Arrays(const Arrays&) = delete;
  ~Arrays() { g_arena.in_use = false; }
  template <class T>
  void add(T** p, size_t count) {
    const size_t bytes = std::max<size_t>(count * sizeof(T), 16);
    const size_t align = bytes >= kPage ? kPage : 256;
    total_ = (total_ + align - 1) / align * align;
    at_.push_back({reinterpret_cast<void**>(p), total_});
    total_ += bytes;
  }
  size_t total() const { return total_; }
  // *fits: false where the memory is too small for them (the level-by-level runs need
  // a third of it)
  rg_status place(bool* fits) {
    const int device = ctx().device;
    if (g_arena.device != device) g_arena.buf.release();
    g_arena.device = device;
    const rg_status s = g_arena.buf.reserve(total_);
    *fits = s == RG_OK;
    if (s == RG_ENOMEM) {
      clear_error();
      return RG_OK;
    }
    RG_TRY(s);
    g_arena.in_use = true;
    for (const auto& a : at_) *a.first = g_arena.buf.as<char>() + a.second;
    return RG_OK;
  }

 private:
  static constexpr size_t kPage = 2 << 20;
  std::vector<std::pair<void**, size_t>> at_;
  size_t total_ = 0;
};

int fused_grid(int64_t work, int64_t per_cta) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(device_sms(), work / per_cta));
}

constexpr unsigned kMostGroups = 64;

// Words of the host's info block: what the launches write for their callers, 3 (or
// 3 of every source's four) once thread 0 is done, and kGaveUp.
constexpr int kDone = 3, kGaveUp = 7;

// Before a call's first launch.
volatile uint64_t* info_begin() {
  volatile uint64_t* info = ctx().ws.h_info;
  info[0] = info[1] = info[kDone] = info[kGaveUp] = 0;
  return info;
}
// Once the stream has passed the call's launches: whether every CTA of them ran to its end.
bool all_ran() { return ctx().ws.h_info[kGaveUp] == 0; }

template <auto kern, class Args>
rg_status launch_fused(Args& args, dim3 grid, size_t dyn, size_t most_dyn, cudaStream_t st) {
  static std::atomic<uint64_t> checked{0};  // of this kernel (two of one type are two)
  RG_TRY(once_per_device(checked, [&]() -> rg_status {
    // one CTA per SM must fit, with all the dynamic shared memory it may ask for
    if (most_dyn) {
      static std::atomic<uint64_t> limit_set{0};
      RG_TRY(allow_max_dyn_smem(limit_set, kern));
    }
    int per_sm = 0;
    RG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kFT, most_dyn));
    return per_sm > 0 ? RG_OK : fail(RG_ECUDA, "one-launch traversal does not fit an SM");
  }));
  Workspace& ws = ctx().ws;
  if (grid.y > kMostGroups) return fail(RG_EINVAL, "more groups than control blocks");
  if (!ws.one_launch.p) {
    RG_TRY(ws.one_launch.reserve(2 * kMostGroups * sizeof(Ctl)));
    ws.one_launch_used = 0;
    const cudaError_t e = cudaMemsetAsync(ws.one_launch.p, 0, 2 * kMostGroups * sizeof(Ctl), st);
    if (e != cudaSuccess) ws.one_launch.release();
    RG_CUDA(e);
  }
  Ctl* sets = ws.one_launch.as<Ctl>();
  args.ctl = sets + ws.one_launch_set * kMostGroups;
  args.stale = sets + (ws.one_launch_set ^ 1) * kMostGroups;
  args.nstale = ws.one_launch_used;
  args.polls = g_wait_polls >= 0 ? (unsigned)g_wait_polls : kPolls;
  args.from = g_wait_from;
  args.gave_up = ws.h_info_dev + kGaveUp;
  void* p[] = {&args};
  kt_begin(st);
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)kern, grid, dim3(kFT), p, dyn, st);
  if (e != cudaSuccess) ws.one_launch.release();  // cleared anew by the next launch
  RG_CUDA(e);
  kt_end(st);
  ws.one_launch_used = (int)grid.y;
  ws.one_launch_set ^= 1;
  g_timing.kernel_launches++;
  g_timing.edge_launches++;
  return RG_OK;
}

size_t small_entries(int64_t n) { return (size_t)(n + 32); }
// pieces: one per started kPiece edges of every vertex above kSmallDeg
size_t large_entries(int64_t n, int64_t m) {
  return (size_t)(std::min<int64_t>(n, m / (kSmallDeg + 1)) + m / kPiece + 64);
}
void add_queues(Arrays& X, Queues* q, int64_t n, int64_t m, int groups = 1) {
  X.add(&q->small, small_entries(n) * groups);
  X.add(&q->large, large_entries(n, m) * groups);
}

int64_t dense_threshold(const rg_graph* g) { return g->m / std::max<int64_t>(g_opts.dense_div, 1); }

// Where a launch may write its results by original id itself: page-locked memory of
// the caller (null: none, they are delivered afterwards).  The host link takes a
// kernel's stores at the rate of a copy (183 of 186 GB/s), so the reordering, a
// random read per vertex, and the result's way through memory hide behind it: BFS
// of 2^24 vertices 805 us, 927 with a copy.  (Rows of several sources are
// copied: stores to 64 rows at once took 2.7 ms in place of 2.0.)
template <class T>
T* direct_results(const rg_graph* g, const T* host_out, const T* dev_out) {
  if (!g->sorted || !host_out || dev_out || g_opts.async_results) return nullptr;
  return static_cast<T*>(device_alias(host_out, sizeof(T) * g->n, sizeof(T)));
}

// The results of a finished launch on their way to the caller: `dev_out`
// (device, original ids) and `host_out`.  `internal` holds them by internal
// id, `ordered` (when the launch wrote it) by original id.
template <class T>
rg_status deliver(rg_graph* g, const T* internal, const T* ordered, T* host_out, T* dev_out, cudaStream_t st) {
  const T* src = ordered ? ordered : internal;
  if (dev_out && dev_out != src) RG_CUDA(cudaMemcpyAsync(dev_out, src, sizeof(T) * g->n, cudaMemcpyDeviceToDevice, st));
  if (!host_out) return RG_OK;
  if (g_opts.async_results) {
    return download_async<T>(host_out, g->n, st, [&](T* stage) -> rg_status {
      RG_CUDA(cudaMemcpyAsync(stage, src, sizeof(T) * g->n, cudaMemcpyDeviceToDevice, st));
      return RG_OK;
    });
  }
  RG_CUDA(cudaMemcpyAsync(host_out, src, sizeof(T) * g->n, cudaMemcpyDeviceToHost, st));
  return RG_OK;
}

}  // namespace

bool short_chunks(const rg_graph* g, cudaStream_t st) {
  return found_once(g->max_chunk_rows, 0, st, [&](unsigned int* d) {
           find_max_chunk<<<64, 256, 0, st>>>(g->in_chunks(), (uint32_t)g->nchunks, d);
         }) <= kPullRows;
}

bool release_idle_arena() {
  if (g_arena.in_use || !g_arena.buf.p) return false;
  g_arena.buf.release();
  return true;
}

bool fused_fits(const rg_graph* g, int64_t max_edges) {
  return g->m <= max_edges && g->n <= max_edges && strides_fit(g->n, g->m) && !g_trace_on;
}

bool bc_rows_fit(const rg_graph* g, int k, bool direct) {
  return fused_fits(g, std::min(kFusedBcRowsEdges, kFusedBcRowsWork / k)) &&
         (direct || g->m >= g->n || k <= kFusedBcRowsFew || g->n * k <= kFusedBcRowsCells);
}

bool ms_fits(const rg_graph* g) {
  return fused_fits(g, kFusedMsEdges) && (2 * g->m >= g->n || g->n <= kFusedMsVertices);
}

namespace {

void bfs_arrays(const rg_graph* g, bool parents, bool ordered, BfsArgs* A, Arrays& X) {
  const int64_t n = g->n, m = g->m, nwords = (n + 31) / 32;
  A->parents = nullptr;
  A->depth_out = nullptr;
  X.add(&A->vis[0], nwords);
  X.add(&A->vis[1], nwords);
  X.add(&A->depth, n);
  if (parents) X.add(&A->parents, n);
  add_queues(X, &A->q[0], n, m);
  add_queues(X, &A->q[1], n, m);
  X.add(&A->rest, (size_t)(m / kRestPiece + m / (kRestList + 48) + 64));  // the last piece of a list may be short
  if (ordered) X.add(&A->depth_out, n);
}

}  // namespace

rg_status bfs_fused_run(rg_graph* g, uint32_t root, uint32_t* h_parents, int32_t* h_depth,
                        int64_t* rounds_out, int64_t* reached_out, int32_t* d_depth_out, bool* done) {
  Ctx& cx = ctx();
  cudaStream_t st = cx.stream;
  const int64_t n = g->n, m = g->m;
  BfsArgs A;
  const bool order = g->sorted && (h_depth || d_depth_out);
  int32_t* direct = direct_results(g, h_depth, d_depth_out);
  Arrays X;
  bfs_arrays(g, h_parents != nullptr, order && !d_depth_out && !direct, &A, X);
  bool fits = false;
  RG_TRY(X.place(&fits));
  if (!fits) return RG_OK;
  if (direct) A.depth_out = direct;
  if (order && d_depth_out) A.depth_out = d_depth_out;
  A.out = g->view();
  A.in = g->in_view();
  A.same = !g->directed;
  A.new_ids = g->sorted ? g->new_ids.as<uint32_t>() : nullptr;
  A.root = root;
  A.threshold = dense_threshold(g);
  A.info = cx.ws.h_info_dev;
  volatile uint64_t* info = info_begin();
  CallTimer timer(g);
  RG_TRY(launch_fused<bfs_fused>(A, fused_grid(m + n, kFusedEdgesPerCta), 0, 0, st));
  RG_TRY(timer.mark());
  if (!direct) RG_TRY(deliver<int32_t>(g, A.depth, A.depth_out, h_depth, d_depth_out, st));
  DevBuf tmp(true, st);  // parents by original id
  RG_TRY(download_orig<uint32_t>(g, A.parents, h_parents, tmp, st));
  RG_CUDA(cudaStreamSynchronize(st));
  RG_TRY(timer.finish());
  *done = info[kDone] == 1 && all_ran();
  if (!*done) return RG_OK;
  g_timing.edges_traversed = (int64_t)info[2];
  g_timing.algorithmic_bytes =
      4 * g_timing.edges_traversed + 4 * (n + 1) + 4 * n + 2 * ((n + 7) / 8) * (int64_t)info[0];
  if (rounds_out) *rounds_out = (int64_t)info[0];
  if (reached_out) *reached_out = (int64_t)info[1];
  return RG_OK;
}

namespace {

// The arrays of `groups` groups of bc_fused.
// *ordered (unless null): n results by original id.
void bc_arrays(const rg_graph* g, int groups, bool chain, bool long_lists, BcArgs* A, double** ordered, Arrays& X) {
  const size_t n = (size_t)g->n, m = (size_t)g->m;
  A->n_small = small_entries(g->n);
  A->n_large = large_entries(g->n, g->m);
  A->same = !g->directed;
  A->long_lists = long_lists;
  // pieces of lists above kLongList, two at least: at most 3/2 per kLongPiece edges
  A->n_heavy = A->long_lists ? m / kLongPiece + m / kLongList + 64 : 0;
  A->new_ids = g->sorted ? g->new_ids.as<uint32_t>() : nullptr;
  X.add(&A->vis, (n + 31) / 32 * groups);
  X.add(&A->lvl, n * groups);
  X.add(&A->sigma, n * groups);
  X.add(&A->even, n * groups);
  X.add(&A->odd, n * groups);
  X.add(&A->inv, n * groups);
  add_queues(X, &A->q, g->n, g->m, groups);
  X.add(&A->first_small, (n + 2) * groups);
  X.add(&A->first_large, (n + 2) * groups);
  X.add(&A->level_deg, (n + 2) * groups);
  X.add(&A->heavy, A->n_heavy * groups);
  if (chain) X.add(&A->deps, n);
  if (ordered) X.add(ordered, n);
}

bool has_long_lists(const rg_graph* g, cudaStream_t st) {
  return std::max(max_in_degree(g, st), (int64_t)g->max_deg) > kLongList;
}

// Groups for k sources and the CTAs of each.  Every source gets a group while there
// are SMs for it and the groups' arrays (44 bytes per vertex that a traversal keeps
// returning to) stay in L2; the SMs are shared out between the groups, up to what
// one traversal can use.
void bc_split(const rg_graph* g, int k, int* groups, int* width) {
  const int64_t in_l2 = std::max<int64_t>(1, kFusedBcRowsL2 / (44 * g->n));
  const int most = (int)std::min<int64_t>({(int64_t)k, (int64_t)device_sms(), in_l2, (int64_t)kMostGroups});
  *groups = (k + (k + most - 1) / most - 1) / ((k + most - 1) / most);  // as many rounds, evenly filled
  *width = std::min(fused_grid(g->m + g->n, kFusedEdgesPerCta), std::max(1, device_sms() / *groups));
}

}  // namespace

rg_status bc_fused_run(rg_graph* g, const uint32_t* src_orig, int nsrc, double* h_deps, int64_t* levels_out,
                       double* d_deps_out, bool* done) {
  Ctx& cx = ctx();
  cudaStream_t st = cx.stream;
  const int64_t n = g->n, m = g->m;
  BcArgs A;
  const bool order = g->sorted && (h_deps || d_deps_out);
  double* direct = direct_results(g, h_deps, d_deps_out);
  double* ordered = !order ? nullptr : direct ? direct : d_deps_out;
  int groups = 1, width = fused_grid(m + n, kFusedEdgesPerCta);
  if (m <= std::min(kFusedBcRowsEdges, kFusedBcRowsWork / std::max(nsrc, 1))) bc_split(g, std::min(nsrc, 64), &groups, &width);
  Arrays X;
  bool fits = false;
  bc_arrays(g, groups, true, has_long_lists(g, st), &A, order && !ordered ? &ordered : nullptr, X);
  RG_TRY(X.place(&fits));
  if (!fits) return RG_OK;
  A.info = cx.ws.h_info_dev;
  volatile uint64_t* info = info_begin();
  CallTimer timer(g);
  A.rows = false;
  A.g = g->view();
  A.gt = g->in_view();
  for (int it = 0; it < nsrc; it += 64) {
    A.k = std::min(nsrc - it, 64);
    for (int q = 0; q < A.k; q++) A.source[q] = src_orig[it + q];
    A.first_source = it == 0;
    A.deps_out = it + A.k == nsrc ? ordered : nullptr;
    RG_TRY(launch_fused<bc_fused>(A, dim3(width, groups), 0, 0, st));
  }
  RG_TRY(timer.mark());
  if (!direct) RG_TRY(deliver<double>(g, A.deps, ordered, h_deps, d_deps_out, st));
  RG_CUDA(cudaStreamSynchronize(st));
  RG_TRY(timer.finish());
  *done = info[kDone] == (uint64_t)nsrc && all_ran();
  if (!*done) return RG_OK;
  g_timing.edges_traversed = (int64_t)info[1];
  g_timing.algorithmic_bytes =
      4 * g_timing.edges_traversed + (int64_t)nsrc * (8 * (n + 1) + 8 * n + n + 16 * n + 8 * n);
  if (levels_out) *levels_out = (int64_t)info[0];
  return RG_OK;
}

// k independent sources, row q of `out` (device, original ids) from source q.
rg_status bc_rows_fused_run(rg_graph* g, const uint32_t* src_orig, int k, double* out, int64_t* levels_out,
                            bool* done) {
  Ctx& cx = ctx();
  cudaStream_t st = cx.stream;
  int groups, width;
  bc_split(g, k, &groups, &width);
  BcArgs A;
  Arrays X;
  bool fits = false;
  bc_arrays(g, groups, false, has_long_lists(g, st), &A, nullptr, X);
  RG_TRY(X.place(&fits));
  if (!fits) return RG_OK;
  A.g = g->view();
  A.gt = g->in_view();
  for (int q = 0; q < k; q++) A.source[q] = src_orig[q];
  A.k = k;
  A.rows = true;
  A.first_source = true;
  A.deps_out = out;
  A.info = reinterpret_cast<volatile uint64_t*>(cx.ws.h_small_dev);
  volatile uint64_t* info = reinterpret_cast<volatile uint64_t*>(cx.ws.h_small);
  for (int i = 0; i < 4 * k; i++) info[i] = 0;
  info_begin();
  RG_TRY(launch_fused<bc_fused>(A, dim3(width, groups), 0, 0, st));
  RG_CUDA(cudaStreamSynchronize(st));
  if (!all_ran()) return RG_OK;
  int64_t levels = 0;
  bool rounded = false, past_integers = false;
  for (int q = 0; q < k; q++) {
    if (info[4 * q + kDone] != 1) return RG_OK;
    const uint64_t counts = info[4 * q + 2];
    const unsigned char* c = reinterpret_cast<const unsigned char*>(&counts);
    rounded |= c[0] != 0;
    past_integers |= c[1] != 0;
    levels = std::max(levels, (int64_t)info[4 * q]);
    g_timing.edges_traversed += (int64_t)info[4 * q + 1];
  }
  // Counts that doubles round and 64-bit integers would not: the shared traversal
  // sums those.  (Past its integers it would answer with doubles itself.)
  if (rounded && !past_integers) return RG_OK;
  *done = true;
  *levels_out = levels;
  return RG_OK;
}

namespace {

// Bits of a depth: at most n - 1, and the round that finds nothing more counts.
int depth_planes(int64_t n) {
  int p = 1;
  while (n >> p) p++;
  return p;
}

// What Radii and multi-source BFS share.
// ordered: n radii by original id too; planes: the depth planes.
void radii_arrays(const rg_graph* g, bool ordered, bool planes, RadiiArgs* A, Arrays& X) {
  const int64_t n = g->n, m = g->m;
  A->radii_out = nullptr;
  A->planes = nullptr;
  X.add(&A->bits[0], (n + 31) / 32);
  X.add(&A->bits[1], (n + 31) / 32);
  X.add(&A->vis, n);
  X.add(&A->nvis, n);
  X.add(&A->radii, n);
  add_queues(X, &A->q[0], n, m);
  add_queues(X, &A->q[1], n, m);
  if (ordered) X.add(&A->radii_out, n);
  if (planes) X.add(&A->planes, (size_t)n * depth_planes(n));
}

// The rest of their arguments; seeds: original ids, each once.
void radii_args(const rg_graph* g, const uint32_t* seeds, const unsigned long long* masks, int k, RadiiArgs* A) {
  A->out = g->view();
  A->in = g->in_view();
  A->chunk_v = g->in_chunks();
  A->nchunks = (uint32_t)g->nchunks;
  A->new_ids = g->sorted ? g->new_ids.as<uint32_t>() : nullptr;
  A->k = k;
  for (int i = 0; i < k; i++) {
    A->seed[i] = seeds[i];
    A->mask[i] = masks[i];
  }
  // a push reads the frontier's edges alone, a pull all of them: where a level is
  // more than latencies, up to twice the share of edges is still pushed (64 sources,
  // R-MAT 2^20 561 -> 486 us, uniform 816 -> 761; uniform 2^10 would lose 8 of 52)
  A->threshold = dense_threshold(g) * (g->m >= 1 << 22 ? 2 : 1);
  A->depths = nullptr;
  A->sources = 0;
  A->info = ctx().ws.h_info_dev;
  info_begin();
}

}  // namespace

rg_status radii_fused_run(rg_graph* g, const uint32_t* seeds, const unsigned long long* masks, int k,
                          int32_t* h_radii, int64_t* rounds_out, int32_t* d_radii_out, bool* done) {
  Ctx& cx = ctx();
  cudaStream_t st = cx.stream;
  const int64_t n = g->n, m = g->m;
  RadiiArgs A;
  const bool order = g->sorted && (h_radii || d_radii_out);
  int32_t* direct = direct_results(g, h_radii, d_radii_out);
  Arrays X;
  bool fits = false;
  radii_arrays(g, order && !d_radii_out && !direct, false, &A, X);
  RG_TRY(X.place(&fits));
  if (!fits) return RG_OK;
  radii_args(g, seeds, masks, k, &A);
  if (direct) A.radii_out = direct;
  if (order && d_radii_out) A.radii_out = d_radii_out;
  volatile uint64_t* info = cx.ws.h_info;
  CallTimer timer(g);
  RG_TRY(launch_fused<radii_fused<false>>(A, fused_grid(m + n, kFusedEdgesPerCta), 0, 0, st));
  RG_TRY(timer.mark());
  if (!direct) RG_TRY(deliver<int32_t>(g, A.radii, A.radii_out, h_radii, d_radii_out, st));
  RG_CUDA(cudaStreamSynchronize(st));
  RG_TRY(timer.finish());
  *done = info[kDone] == 1 && all_ran();
  if (!*done) return RG_OK;
  g_timing.edges_traversed = (int64_t)info[1];
  g_timing.algorithmic_bytes = 4 * g_timing.edges_traversed + 16 * n + 4 * n;
  if (rounds_out) *rounds_out = (int64_t)info[0];
  return RG_OK;
}

rg_status ms_fused_run(rg_graph* g, const uint32_t* seeds, const unsigned long long* masks, int u, int k, int32_t* out,
                       int64_t* rounds_out, bool* done) {
  Ctx& cx = ctx();
  cudaStream_t st = cx.stream;
  const int64_t n = g->n, m = g->m;
  RadiiArgs A;
  Arrays X;
  bool fits = false;
  radii_arrays(g, false, true, &A, X);
  RG_TRY(X.place(&fits));
  if (!fits) return RG_OK;
  radii_args(g, seeds, masks, u, &A);
  A.depths = out;
  A.sources = k;
  volatile uint64_t* info = cx.ws.h_info;
  RG_TRY(launch_fused<radii_fused<true>>(A, fused_grid(m + n + n * (int64_t)k / 8, kFusedEdgesPerCta), 0, 0, st));
  RG_CUDA(cudaStreamSynchronize(st));
  *done = info[kDone] == 1 && all_ran();
  if (!*done) return RG_OK;
  g_timing.edges_traversed += (int64_t)info[1];
  *rounds_out = (int64_t)info[0];
  return RG_OK;
}

size_t one_launch_bytes(const rg_graph* g, int kind, int k) {
  Arrays X;
  if (kind == RG_QUERY_BC) {
    if (!(k > 1 ? bc_rows_fit(g, k, false) : fused_fits(g, kFusedBcEdges))) return 0;
    int groups = 1, width = 0;
    if (k > 1) bc_split(g, k, &groups, &width);
    BcArgs A;
    bc_arrays(g, groups, k == 1, true, &A, nullptr, X);
  } else if (kind == RG_QUERY_BFS && k == 1) {
    if (!fused_fits(g, kFusedBfsEdges)) return 0;
    BfsArgs A;
    bfs_arrays(g, false, false, &A, X);
  } else if (kind == RG_QUERY_BFS ? ms_fits(g)
                                  : k == 1 && fused_fits(g, g->sorted ? kFusedRadiiSortedEdges : kFusedRadiiEdges)) {
    RadiiArgs A;
    radii_arrays(g, false, kind == RG_QUERY_BFS, &A, X);
  }
  return X.total();
}

rg_status pagerank_fused_run(rg_graph* g, bool pull, int64_t max_iters, double* h_ranks, int64_t* iters_out, double* l1_out,
                             bool* done) {
  Ctx& cx = ctx();
  cudaStream_t st = cx.stream;
  const int64_t n = g->n, m = g->m;
  PrArgs A;
  const int grid = fused_grid(m + n, kFusedPrEdgesPerCta);
  // a row counts as `weight` edges: as few as keep a CTA's rows in its shared
  // memory (share / weight of them at most).  `share`: the edges of a CTA, but
  // for its last row
  const int64_t room = kFusedPrRows - 4 - n / grid;
  if (room <= 0) return RG_OK;
  const int64_t weight = m / grid / room + 1;
  // ... which lets a CTA hold more edges than its share by what the rows count for: in a
  // degree-sorted skewed graph some do.  (1.0e6 vertices, 6.7e6 edges, rows of 9: 1835 us,
  // 1658 pushed; 1.8e6 vertices, 8.2e6 edges, rows of 320: 26 ms and 2.2.)
  if (!pull && weight * n > (g->sorted ? 5 * m / 4 : 3 * m)) return RG_OK;
  const int64_t share = (m + weight * n + grid - 1) / grid;
  const int64_t rows = std::min<int64_t>(n, share / weight + 2);
  A.row_weight = (uint32_t)weight;
  // a row is not shared between CTAs: one with far more edges than a CTA's
  // share would hold the others up (one launch / swept, us: 4.7e5 vertices, 2.9e6 edges,
  // a row of 2.4 shares 1095 / 620; 8e4, 2.2e6, 1.75 445 / 337; 2.6e5, 6e5, 1.5 316 / 332)
  if (rows > kFusedPrRows || max_in_degree(g, st) > (pull && m > 1 << 20 ? 1 : 2) * share) return RG_OK;
  const bool order = g->sorted && h_ranks;
  const size_t steps = (size_t)(m / kPrStep + 2 * grid + 4);
  A.ranks_out = nullptr;
  Arrays X;
  X.add(&A.lane_row, (size_t)(m / 4 + 32 * (grid + 2) + 64));
  X.add(&A.opens, steps);
  X.add(&A.closes, steps);
  X.add(&A.p, n);
  X.add(&A.contrib[0], n);
  X.add(&A.contrib[1], n);
  X.add(&A.rmag, n);
  X.add(&A.l1, std::max<int64_t>(max_iters, 1));
  if (order) X.add(&A.ranks_out, n);
  bool fits = false;
  RG_TRY(X.place(&fits));
  if (!fits) return RG_OK;
  A.in = g->in_view();
  A.out_off = g->off.as<uint32_t>();
  A.chunk_v = g->in_chunks();
  A.new_ids = g->sorted ? g->new_ids.as<uint32_t>() : nullptr;
  A.max_iters = max_iters;
  A.p0 = 1 / (double)n;
  A.added = (1 - kPrDamp) * (1 / (double)n);
  A.info = cx.ws.h_info_dev;
  volatile uint64_t* info = info_begin();
  CallTimer timer(g);
  RG_TRY(launch_fused<pagerank_fused>(A, grid, sizeof(U128) * (size_t)rows, sizeof(U128) * kFusedPrRows, st));
  RG_TRY(timer.mark());
  RG_TRY(deliver<double>(g, A.p, A.ranks_out, h_ranks, nullptr, st));
  RG_CUDA(cudaStreamSynchronize(st));
  RG_TRY(timer.finish());
  *done = info[kDone] == 1 && all_ran();
  if (!*done) return RG_OK;
  const int64_t run = (int64_t)info[0];
  const bool broke = info[4] != 0;
  g_timing.edge_launches = run;
  g_timing.edges_traversed = m * run;
  g_timing.algorithmic_bytes = (4 * m + 4 * (n + 1) + 16 * n) * run;
  if (iters_out) *iters_out = broke ? run : max_iters + 1;
  if (l1_out) *l1_out = max_iters ? fx_to_double(U128{info[1], info[2]}) : 0.0;
  return RG_OK;
}

rg_status prd_fused_run(rg_graph* g, bool allow_pull, int64_t start, int64_t max_iters, double* p, double* ngh,
                        double* c, uint32_t* bits, double* ranks_out, int64_t* rounds, double* l1, bool* launched,
                        bool* done) {
  Ctx& cx = ctx();
  cudaStream_t st = cx.stream;
  const int64_t n = g->n, m = g->m;
  PrdArgs A;
  A.rows = Queues{};
  Arrays X;
  add_queues(X, &A.q[0], n, m);
  add_queues(X, &A.q[1], n, m);
  if (start == 0) add_queues(X, &A.rows, n, m);
  X.add(&A.touched, (n + 31) / 32);
  bool fits = false;
  RG_TRY(X.place(&fits));
  if (!fits) return RG_OK;
  A.out = g->view();
  A.in = g->in_view();
  A.new_ids = g->sorted ? g->new_ids.as<uint32_t>() : nullptr;
  A.p = p;
  A.ngh = ngh;
  A.c = c;
  A.bits = bits;
  A.start = start;
  A.max_iters = max_iters;
  A.threshold = dense_threshold(g);
  A.short_push = n / 64;
  A.allow_pull = allow_pull;
  A.one_over_n = 1 / (double)n;
  A.added = (1 - kPrDamp) * A.one_over_n;
  A.ranks_out = ranks_out;
  A.info = cx.ws.h_info_dev;
  volatile uint64_t* info = info_begin();
  RG_TRY(launch_fused<prd_fused>(A, fused_grid(m + n, kFusedEdgesPerCta), 0, 0, st));
  *launched = true;
  RG_CUDA(cudaStreamSynchronize(st));
  *done = info[kDone] == 1 && all_ran();
  if (!*done) return RG_OK;
  *rounds = (int64_t)info[0];
  *l1 = double_of(info[1]);
  g_timing.edges_traversed += (int64_t)info[2];
  return RG_OK;
}

}  // namespace rg
