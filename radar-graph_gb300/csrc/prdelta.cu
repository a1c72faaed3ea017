// PageRankDelta (PageRankDelta.C:98-155) on the device.
//
// Each round pushes (or, in push-pull, pulls) the frontier's deltas --
// nghSum[d] += Delta[s]/deg(s) -- and then one vertex kernel applies the round's
// filter (PR_Vertex_F_FirstRound in round 1, PR_Vertex_F after), resets nghSum,
// forms the next frontier's contributions and bitmap, and sums |Delta| for the L1
// stop (< 1e-7).  The arithmetic is FP64 like the reference; a pulled sum is
// formed exactly and rounded once (pr_exact.cuh).
//
// Small graphs run whole in one launch (fused.cu).  Larger ones run their dense
// first rounds here, a launch each over the whole chip, and hand the rest, rounds
// that reach few vertices, to the same launch: 14 of the 19 rounds of a 2e6-vertex
// R-MAT graph, each of which cost a filter over every vertex, a compaction and a
// host round trip (1.4 of 3.1 ms).

#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "app_common.cuh"
#include "fused.cuh"

namespace rg {

namespace {

__global__ void prd_init(uint32_t n, const uint32_t* __restrict__ off, double* p, double* ngh, double* c,
                         double one_over_n) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    p[v] = 0.0;
    ngh[v] = 0.0;
    const uint32_t d = off[v + 1] - off[v];
    c[v] = d ? one_over_n / d : 0.0;
  }
}

// vertexFilter over all vertices with the round's functor, fused with the
// L1 terms, the nghSum reset (PR_Vertex_Reset) and the next contributions.
// Each warp owns 32 consecutive vertices = one bitmap word (grid stride in
// whole warps), so the active set is written with a ballot, no atomics; a word
// that nothing reached and that held no member stays as it is.  kExact: the sums
// are the pull's (acc, zeroed where the next one adds); else the push's (ngh).
template <bool kFirst, bool kExact>
__global__ void __launch_bounds__(256) prd_filter(uint32_t n, const uint32_t* __restrict__ off,
                                                  const uint32_t* __restrict__ pull_off, double* p, double* ngh,
                                                  U128* acc, double* c, double one_over_n, double added,
                                                  const uint32_t* __restrict__ bits, uint32_t* next_bits,
                                                  double* l1_out) {
  const int lane = threadIdx.x & 31;
  double local = 0.0;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * 32 < n; w += warps) {
    const uint64_t v = w * 32 + lane;
    bool act = false;
    U128 a{0ull, 0ull};
    double g = 0.0;
    if (v < n) {
      if (kExact) a = acc[v];
      else g = ngh[v];
    }
    const bool some = kExact ? (a.lo | a.hi) != 0ull : g != 0.0;
    if (!kFirst && !bits[w] && !__any_sync(0xffffffffu, some)) {
      if (lane == 0) next_bits[w] = 0u;
      continue;
    }
    if (v < n) {
      if (kExact && some) {
        g = fx_to_signed(a);
        const uint32_t b = pull_off[v], e = pull_off[v + 1];
        if (b / kExactStep != (e - 1) / kExactStep) acc[v] = U128{0ull, 0ull};
      }
      double pv = p[v], d;
      if (kFirst) {  // PageRankDelta.C:46-61
        d = __dadd_rn(__dmul_rn(kPrDamp, g), added);
        pv = __dadd_rn(pv, d);
        d = __dsub_rn(d, one_over_n);
        act = fabs(d) > __dmul_rn(kPrdEps2, pv);
        p[v] = pv;
      } else {  // PageRankDelta.C:63-76
        d = __dmul_rn(g, kPrDamp);
        act = fabs(d) > __dmul_rn(kPrdEps2, pv);
        if (act) p[v] = __dadd_rn(pv, d);
      }
      if (!kExact && some) ngh[v] = 0.0;
      const uint32_t deg = off[v + 1] - off[v];
      c[v] = (act && deg) ? __ddiv_rn(d, (double)deg) : 0.0;
      local += fabs(d);
    }
    const unsigned now = __ballot_sync(0xffffffffu, act);
    if (lane == 0) next_bits[w] = now;
  }
  local = warp_sum(local);
  __shared__ double ws[8];
  if (lane == 0) ws[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = threadIdx.x < 8 ? ws[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0 && t != 0.0) atomicAdd(l1_out, t);
  }
}

struct PrdState {
  DevBuf p, ngh, c, acc, l1, tmp;
  Frontier f[2];
};

}  // namespace

rg_status pagerank_delta_run(rg_graph* g, int variant, int64_t max_iters, double* h_ranks, int64_t* iters_out,
                             double* l1_out) {
  if (!g) return fail(RG_EINVAL, "null graph");
  if (variant < 0 || variant > 4) return fail(RG_EINVAL, "bad variant %d", variant);
  if (max_iters < 0) return fail(RG_EINVAL, "max_iters < 0");
  OptScope opt_scope(g, kAppPagerank);  // the PageRank schedule: same kind of sweep
  Ctx* cx = nullptr;
  RG_TRY(get_ctx(&cx));
  cudaStream_t st = cx->stream;
  const int64_t n = g->n;
  static thread_local PrdState S;
  RG_TRY(S.p.reserve(8 * n));
  RG_TRY(S.ngh.reserve(8 * n));
  RG_TRY(S.c.reserve(8 * n));
  RG_TRY(S.l1.reserve(8));
  RG_TRY(frontier_alloc(g, S.f[0]));
  RG_TRY(frontier_alloc(g, S.f[1]));
  const double one_over_n = 1 / (double)n;
  const double added = (1 - kPrDamp) * one_over_n;  // PageRankDelta.C:55
  double* p = S.p.as<double>();
  double* ngh = S.ngh.as<double>();
  double* c = S.c.as<double>();
  double* d_l1 = S.l1.as<double>();
  const int vblocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)device_sms() * 16);
  const bool pulls = variant == RG_PUSH_PULL || g_opts.direction == 1;
  int64_t round = 0;
  double l1 = 0.0;
  CallTimer timer(g);
  bool whole = false;  // answered by one launch
  if (fused_fits(g, kFusedPrdEdges)) {
    RG_TRY(prd_fused_run(g, true, 0, max_iters, p, ngh, c, S.f[0].bits.as<uint32_t>(), nullptr, &round, &l1, &whole));
  }
  if (!whole) {
    prd_init<<<vblocks, 256, 0, st>>>((uint32_t)n, g->off.as<uint32_t>(), p, ngh, c, one_over_n);
    g_timing.kernel_launches++;
    U128* acc = nullptr;
    if (pulls) {
      RG_TRY(S.acc.reserve(sizeof(U128) * n));
      acc = S.acc.as<U128>();
      RG_CUDA(cudaMemsetAsync(acc, 0, sizeof(U128) * n, st));
    }
    RG_TRY(frontier_set_all(g, S.f[0], st));  // every vertex starts in the frontier
    FView cur = view_of(S.f[0]), nxt = view_of(S.f[1]);
    EmOpts o;
    o.variant = variant;
    o.dense_forward = variant != RG_PUSH_PULL;  // no_output | dense_forward; push-pull pulls
    Workspace& ws = cx->ws;
    bool hand_over = !g_trace_on;  // sparse rounds go to one launch (once)
    round = 0;
    while (round++ < max_iters) {
      const bool dense = cur.count + cur.degsum > g->m / std::max<int64_t>(g_opts.dense_div, 1);
      if (!dense && round > 1 && hand_over) {
        bool done = false;
        // (a launch that gives up has changed p, ngh and c: the run starts again, level by level)
        RG_TRY(prd_fused_run(g, false, round - 1, max_iters, p, ngh, c, cur.bits, nullptr, &round, &l1, &done));
        if (done) break;
        hand_over = false;
        prd_init<<<vblocks, 256, 0, st>>>((uint32_t)n, g->off.as<uint32_t>(), p, ngh, c, one_over_n);
        if (acc) RG_CUDA(cudaMemsetAsync(acc, 0, sizeof(U128) * n, st));
        RG_TRY(frontier_set_all(g, S.f[0], st));
        cur = view_of(S.f[0]);
        nxt = view_of(S.f[1]);
        round = 0;
        continue;
      }
      const bool pull = dense && g->m > 0 && pulls;
      if (pull) {
        g_timing.edges_traversed += cur.degsum;
        RG_TRY(exact_pull_signed(g, c, acc, st));
      } else {
        RG_TRY(edge_map(g, cur, OpPrDelta{c, ngh}, nullptr, o, st));
      }
      RG_CUDA(cudaMemsetAsync(d_l1, 0, 8, st));
      auto filter = round == 1 ? (pull ? prd_filter<true, true> : prd_filter<true, false>)
                               : (pull ? prd_filter<false, true> : prd_filter<false, false>);
      filter<<<vblocks, 256, 0, st>>>((uint32_t)n, g->off.as<uint32_t>(), g->in_view().off, p, ngh, acc, c, one_over_n,
                                      added, cur.bits, nxt.bits, d_l1);
      RG_CUDA(cudaGetLastError());
      g_timing.kernel_launches++;
      RG_CUDA(cudaMemcpyAsync(&ws.h_info[4], d_l1, 8, cudaMemcpyDeviceToHost, st));
      Frontier shell;  // non-owning view of nxt for the compaction (which syncs)
      shell.bits.p = nxt.bits;
      RG_TRY(compact_bits(g, shell, st, true, nullptr, 0, nullptr, nxt.queue, nxt.qoff));
      shell.bits.p = nullptr;
      nxt.count = shell.count;
      nxt.degsum = shell.degsum;
      g_timing.kernel_launches += 3;
      memcpy(&l1, &ws.h_info[4], 8);
      if (l1 < kPrdEps) break;  // PageRankDelta.C:144
      std::swap(cur, nxt);
    }
  }
  RG_TRY(timer.stop());
  RG_TRY(download_orig<double>(g, p, h_ranks, S.tmp, st));
  RG_CUDA(cudaStreamSynchronize(st));
  // edge array + contribution per frontier edge; p, Delta, nghSum, c, the
  // degree and the bitmap per vertex per round
  g_timing.algorithmic_bytes = 12 * g_timing.edges_traversed + (int64_t)(44 * n + n / 8) * std::min(round, max_iters);
  if (iters_out) *iters_out = round;
  if (l1_out) *l1_out = l1;
  return RG_OK;
}

}  // namespace rg

extern "C" rg_status rg_pagerank_delta(rg_graph* g, rg_variant variant, int64_t max_iters, double* h_ranks,
                                       int64_t* iters_out, double* l1_out) {
  return rg::pagerank_delta_run(g, variant, max_iters, h_ranks, iters_out, l1_out);
}
