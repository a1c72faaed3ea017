// Whole traversals in one launch (fused.cu), and the PageRank device helpers
// that its kernels share with the sweeps of pagerank.cu.
#pragma once

#include "app_common.cuh"
#include "pr_exact.cuh"

namespace rg {

// A CTA of a one-launch traversal is given at least this many edges (and
// vertices): 2048 and 8192 measured within 3 % at 2^14 vertices and 10-20 %
// apart at 2^10, the smaller the better for BC and Radii, the same for BFS.
constexpr int64_t kFusedEdgesPerCta = 4096;

// The one-launch PageRank is a chain of dependent loads per step, so smaller
// CTAs pay for longer (2^14 vertices, 4.4e5 edges, 20 iterations: 236 us a
// call with 8192 edges per CTA, 189 with 4096, 153 with 2048, 148 with 1024).
constexpr int64_t kFusedPrEdgesPerCta = 1024;

// Rows of a CTA of the one-launch PageRank (16 bytes of shared memory each).
constexpr int64_t kFusedPrRows = 12000;

// Largest graphs (edges, and vertices) that take the one-launch path, by app.
// Device time against the level-by-level run, R-MAT edge factor 16, degree
// sorted (in brackets: uniform, unsorted), us:
//   BFS       2^10 vertices 27 / 182, 2^16 43 / 298, 2^20 87 / 415 (104 / 402),
//             2^24 450 / 973 (1680 / 2972): every size
//   BC        2^10 51 / 246 (72 / 240), 2^18 125 / 506 (125 / 496), 2^22
//             703 / 1573 (970 / 1975), 2^24 3150 / 5520 (5560 / 9983): every size
//   Radii     2^10 63 / 309, 2^18 231 / 583 (257 / 515), 2^20 462 / 789 (718 /
//             963), 2^20.5 631 / 913 (997 / 1012), 2^21 749 / 988 (1293 / 1249), 2^22
//             1658 / 1866 (2623 / 2355), 2^22.5 2609 / 2739, 2^23 2970 / 2758: sorted
//             1.7e8 edges, others 5e7 (their pulls want more warps than one CTA per
//             SM holds)
//   multi-source BFS  64 sources: 2^10 74 / 295, 2^18 226 / 615 (330 / 628), 2^21
//             943 / 1760 (1535 / 2633), 2^22 1800 / 2992 (3076 / 4666); 2 sources:
//             2^20 331 / 584 (539 / 746), 2^21 481 / 726 (918 / 988), 2^22 1050 / 1364
//             (1768 / 1736): 1.3e8 edges
//   PageRank  20 iterations, against pulls: 2^10 97 / 217, 2^14 154 / 247 (93 /
//             160), 2^16 308 / 308 (183 / 245), 2^17 565 / 473 (297 / 365): 3e6
//             edges; against pushes: 2^16 309 / 730, 2^18 1331 / 1559, 2^19 2737 /
//             2332: 8e6 edges.  Few edges a vertex: 2^20 vertices, one each 735 / 794
//             (skewed 809 / 811), 1.36e6 1069 / 834: 2^20 vertices
//   PageRankDelta  whole, against dense rounds swept and the rest handed over:
//             2^14 167 / 173 (85 / 102), 2^17 374 / 369 (164 / 175), 2^18 411 / 343
//             (258 / 239), 2^19 619 / 495 (462 / 381), 2^20 1086 / 829 (842 / 646):
//             6e6 edges; where dense rounds would push level by level, 3.3e7.  Its
//             vertices cost a warp of few per SM more than its edges do: uniform, 2
//             edges a vertex, 2^19 772 / 680, 2^20 1961 / 1370, 2^21 3637 / 2224, a star
//             of 3e6 11718 / 3858 (pushed level by level: 781 / 1290, 1954 / 2477, 3637 /
//             3149, 11714 / 152065): 2^18 vertices; against pushes 2^21, pulled above
constexpr int64_t kFusedBfsEdges = INT64_MAX;
constexpr int64_t kFusedBcEdges = INT64_MAX;
constexpr int64_t kFusedRadiiEdges = 6 << 23, kFusedRadiiSortedEdges = 5 << 25;
constexpr int64_t kFusedPagerankEdges = 3 << 20;
constexpr int64_t kFusedPagerankPushEdges = 8 << 20;
constexpr int64_t kFusedPagerankVertices = 1 << 20;
constexpr int64_t kFusedPrdEdges = 6 << 20;
constexpr int64_t kFusedPrdPushEdges = 1 << 25;
constexpr int64_t kFusedPrdVertices = 1 << 18, kFusedPrdPushVertices = 1 << 21;
//   multi-source BC  16 sources: 2^14 116 / 1023 (147 / 864), 2^18 850 / 2055
//             (900 / 2193), 2^19 1800 / 3010 (3000 / 4154), 2^20 4564 / 5299 (8250 /
//             6911); 64 sources: 2^16 921 / 1498 (1426 / 1464), 2^17 1764 / 1961
//             (2016 / 1933), 2^18 3280 / 2978; 5 sources: 2^19 650 / 1613 (770 /
//             1400), 2^20 1444 / 2468 (2637 / 2436): 2.7e8 edges times sources and
//             2.5e7 edges
constexpr int64_t kFusedBcRowsEdges = 24 << 20;
constexpr int64_t kFusedBcRowsWork = 256 << 20;  // edges times sources
// Groups' arrays at once: 64 sources on 2^17 vertices 2079 us with all of them
// (370 MB), 2016 in 80 MB; 16 sources on 2^18 808 us with all (184 MB), 1008 in 80 MB.
constexpr int64_t kFusedBcRowsL2 = 192 << 20;
constexpr int64_t kFusedMsEdges = 1 << 27;
// Graphs of fewer edges than vertices, where a source costs passes over the vertices
// alone (device us, one launch / shared): 2^20 vertices, 1000 edges, 2 sources 51 / 127,
// 16 269 / 196, 64 1022 / 449; 2^24 vertices 2 sources 463 / 707, 10 2147 / 1361; 2^16
// vertices, 64 sources 97 / 2239.  (Page-locked rows are written by the launch: 2992 /
// 3312 a whole call for 64 sources on 2^20.)
constexpr int64_t kFusedBcRowsFew = 3, kFusedBcRowsCells = 8 << 20;  // sources; vertices times sources
// Multi-source BFS, half as many edges as vertices: 2^24 vertices, 2 sources 194 / 157,
// 10 284 / 246; 2^20 vertices 31 / 75 and 44 / 89.
constexpr int64_t kFusedMsVertices = 6 << 20;
bool bc_rows_fit(const rg_graph* g, int k, bool direct);
bool ms_fits(const rg_graph* g);

// Whether a call on g may take the one-launch path: small enough, and no
// per-level records (rg_set_trace) are asked for.
bool fused_fits(const rg_graph* g, int64_t max_edges);

// Rows of a chunk up to which a sweep pulls: a lane walks from row to row, and over
// those without edges too (4e6 of them in one place: 0.8 s a sweep).
constexpr uint32_t kPullRows = 2048;
// Whether g's pull lists have no chunk of more (found once per graph).
bool short_chunks(const rg_graph* g, cudaStream_t st);

// Each sets *done when the launch answered the call; otherwise (its bounded
// waits ran out, or its arrays do not fit the memory) the caller answers level by
// level.
rg_status bfs_fused_run(rg_graph* g, uint32_t root, uint32_t* h_parents, int32_t* h_depth,
                        int64_t* rounds_out, int64_t* reached_out, int32_t* d_depth_out, bool* done);
rg_status bc_fused_run(rg_graph* g, const uint32_t* src_orig, int nsrc, double* h_deps, int64_t* levels_out,
                       double* d_deps_out, bool* done);
// k <= 64 independent sources; out: k rows of n (device, original ids); *levels_out:
// the most levels of any source.  Synchronises.
rg_status bc_rows_fused_run(rg_graph* g, const uint32_t* src_orig, int k, double* out, int64_t* levels_out,
                            bool* done);
// seeds: original ids, each once, with its mask
rg_status radii_fused_run(rg_graph* g, const uint32_t* seeds, const unsigned long long* masks, int k,
                          int32_t* h_radii, int64_t* rounds_out, int32_t* d_radii_out, bool* done);
// pull: the call would be answered by pulls otherwise.
rg_status pagerank_fused_run(rg_graph* g, bool pull, int64_t max_iters, double* h_ranks, int64_t* iters_out, double* l1_out,
                             bool* done);
// BFS depths from k <= 64 sources; seeds: the distinct ones (original ids) with
// the mask of the sources at each.  out: k rows of n (device, original ids).
// Synchronises.
rg_status ms_fused_run(rg_graph* g, const uint32_t* seeds, const unsigned long long* masks, int u, int k, int32_t* out,
                       int64_t* rounds_out, bool* done);

// PageRankDelta from round `start` on (0: a whole run, which initialises p, ngh
// and c itself; else p, c and the frontier's bits as the filter of round `start`
// left them, ngh 0).  Synchronises; *rounds as the reference counts them.  *launched:
// p, ngh and c have changed, whether the launch ran to its end or not.
// ranks_out (device, original ids) may be null.
rg_status prd_fused_run(rg_graph* g, bool allow_pull, int64_t start, int64_t max_iters, double* p, double* ngh,
                        double* c, uint32_t* bits, double* ranks_out, int64_t* rounds, double* l1, bool* launched,
                        bool* done);

// Device memory of the arrays that a served query (RG_QUERY_*) of k sources takes in one
// launch, its result beside them; 0 where it does not.
size_t one_launch_bytes(const rg_graph* g, int kind, int k);

constexpr double kPrDamp = 0.85;  // PageRank.C:126
constexpr double kPrdEps = 0.0000001, kPrdEps2 = 0.01;  // PageRankDelta.C:103-104

// The exact pull of pagerank.cu over signed contributions (PageRankDelta's):
// acc[v] = sum of c over v's in-neighbours as a 128-bit two's complement fixed
// point number.  acc must be 0 in the rows that cross a step of kExactStep edges.
// The sweep does nothing if the gate is closed; it follows the kernel before it
// (launch_following).
constexpr uint32_t kExactStep = 512;

// What a PageRankDelta filter found, and the gate it is to the next round: that
// pulls if the frontier is dense and the run goes on (a round that did nothing
// leaves zeros, which close the gates after it).
struct PrdTotals {
  unsigned long long count, degsum;
  double l1;
  unsigned long long unused;
};
struct PrdGate {
  const PrdTotals* prev;  // null: open
  int64_t threshold;
  __device__ __forceinline__ bool open() const {
    return !prev || ((int64_t)(prev->count + prev->degsum) > threshold && !(prev->l1 < kPrdEps));
  }
};
rg_status exact_pull_signed(rg_graph* g, const double* c, U128* acc, const PrdGate& gate, cudaStream_t st);

// acc[v] += x for a 128-bit sum shared with other warps: the low word's
// atomic returns the old value, so the carry out of it is known and goes into
// the high word.  Every carry is counted once, so the final sum is exact.
__device__ __forceinline__ void atomic_add128(U128* p, const U128& x) {
  const unsigned long long old = atomicAdd(&p->lo, x.lo);
  const unsigned long long hi = x.hi + (old + x.lo < old ? 1ull : 0ull);
  if (hi) atomicAdd(&p->hi, hi);
}

__device__ __forceinline__ void store128(U128* p, const U128& x) {
  asm volatile("st.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x.lo), "l"(x.hi) : "memory");
}

__device__ __forceinline__ U128 shfl_up128(const U128& x, int o) {
  return U128{__shfl_up_sync(0xffffffffu, x.lo, o), __shfl_up_sync(0xffffffffu, x.hi, o)};
}

__device__ __forceinline__ U128 block_sum128(U128 v) {
  __shared__ U128 ws[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    add128(v, U128{__shfl_xor_sync(0xffffffffu, v.lo, o), __shfl_xor_sync(0xffffffffu, v.hi, o)});
  }
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
  __syncthreads();
  U128 t{0ull, 0ull};
  if (threadIdx.x < 32) {
    if (threadIdx.x < (blockDim.x >> 5)) t = ws[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      add128(t, U128{__shfl_xor_sync(0xffffffffu, t.lo, o), __shfl_xor_sync(0xffffffffu, t.hi, o)});
    }
  }
  return t;  // valid in thread 0
}

// p'/deg, the IEEE quotient of PR_F (PageRank.C:48), by degree class (the
// deg_quotient classes): the integer reciprocal is read only for degrees
// that need it, and degree-sorted graphs keep whole warps in one class.
__device__ __forceinline__ double pr_quotient(double pn, uint32_t d, const unsigned long long* __restrict__ rmag,
                                              int64_t v) {
  if (d == 0) return 0.0;
  if ((d & (d - 1)) == 0) return double_of(bits_of(pn) - ((unsigned long long)(31 - __clz(d)) << 52));
  return div_by_magic(pn, d, rmag[v]);
}

}  // namespace rg
