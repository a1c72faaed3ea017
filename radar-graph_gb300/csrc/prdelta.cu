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
#include "pr_exact.cuh"

namespace rg {

namespace {

// Every vertex starts in the frontier.  rmag: the integer reciprocals of the
// degrees (pr_exact.cuh), for this quotient and the later ones.
__global__ void __launch_bounds__(256) prd_init(uint32_t n, const uint32_t* __restrict__ off, double* p, double* ngh,
                                                double* c, unsigned long long* rmag, uint32_t* bits,
                                                double one_over_n) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    p[v] = 0.0;
    ngh[v] = 0.0;
    const uint32_t d = off[v + 1] - off[v];
    const unsigned long long R = (d & (d - 1)) ? recip_magic(d) : 0ull;
    c[v] = deg_quotient(one_over_n, d, R);
    rmag[v] = R;
    if ((threadIdx.x & 31) == 0) bits[v >> 5] = n - v >= 32 ? 0xffffffffu : (1u << (n - v)) - 1u;
  }
}

// vertexFilter over all vertices with the round's functor, fused with the
// L1 terms, the nghSum reset (PR_Vertex_Reset) and the next contributions.
// Each warp owns 32 consecutive vertices = one bitmap word (grid stride in
// whole warps), so the active set is written with a ballot, no atomics; a word
// that nothing reached and that held no member stays as it is.  kExact: the sums
// are the pull's (acc, zeroed where the next one adds); else the push's (ngh).
//
// Bound by memory at 52 bytes a vertex; the FP64 pipe (a warp instruction in 16
// clocks) comes next, so the quotient is an integer one: with FP64 divisions the
// filter of 2^21 vertices took 70 us.
template <bool kFirst, bool kExact>
__global__ void __launch_bounds__(256) prd_filter(uint32_t n, const uint32_t* __restrict__ off,
                                                  const uint32_t* __restrict__ pull_off, double* p, double* ngh,
                                                  U128* acc, double* c, const unsigned long long* __restrict__ rmag,
                                                  double one_over_n, double added, const uint32_t* __restrict__ bits,
                                                  uint32_t* next_bits, PrdGate gate, PrdTotals* totals) {
  follow();
  if (!gate.open()) return;
  const int lane = threadIdx.x & 31;
  double local = 0.0;
  uint32_t count = 0;
  unsigned long long degsum = 0;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * 32 < n; w += warps) {
    const uint64_t v = w * 32 + lane;
    bool act = false;
    U128 a{0ull, 0ull};
    double g = 0.0, pv = 0.0;
    uint32_t deg = 0, b = 0, e = 1;
    unsigned long long R = 0;
    if (v < n) {  // a dense round changes nearly every vertex: all that it needs is loaded together
      if (kExact) {
        a = acc[v];
        b = pull_off[v];
        e = pull_off[v + 1];
      } else {
        g = ngh[v];
      }
      pv = p[v];
      deg = off[v + 1] - off[v];
      R = rmag[v];
    }
    const bool some = kExact ? (a.lo | a.hi) != 0ull : g != 0.0;
    if (!kFirst && !bits[w] && !__any_sync(0xffffffffu, some)) {
      if (lane == 0) next_bits[w] = 0u;
      continue;
    }
    if (v < n) {
      if (kExact && some) {
        g = fx_to_signed(a);
        if (b / kExactStep != (e - 1) / kExactStep) acc[v] = U128{0ull, 0ull};
      }
      double d;
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
      c[v] = act ? deg_quotient_signed(d, deg, R) : 0.0;
      if (act) degsum += deg;
      local += fabs(d);
    }
    const unsigned now = __ballot_sync(0xffffffffu, act);
    if (lane == 0) {
      next_bits[w] = now;
      count += __popc(now);
    }
  }
  local = warp_sum(local);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) degsum += __shfl_xor_sync(0xffffffffu, degsum, o);
  __shared__ double ws[8];
  __shared__ unsigned long long wd[8], wc[8];
  if (lane == 0) {
    ws[threadIdx.x >> 5] = local;
    wd[threadIdx.x >> 5] = degsum;
    wc[threadIdx.x >> 5] = count;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = threadIdx.x < 8 ? ws[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0) {
      unsigned long long dg = 0, ct = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        dg += wd[i];
        ct += wc[i];
      }
      if (t != 0.0) atomicAdd(&totals->l1, t);
      if (ct) {
        atomicAdd(&totals->count, ct);
        atomicAdd(&totals->degsum, dg);
      }
    }
  }
}

// Pulled rounds enqueued at a time: each is gated on the totals of the one before,
// so the host waits once for all of them; a closed one costs two empty launches.
constexpr int kPulledRounds = 6;

struct PrdState {
  DevBuf arrays, totals, tmp;
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
  bool pulls = variant == RG_PUSH_PULL || g_opts.direction == 1;
  // a whole run in one launch; push variants on graphs with more vertices than that is
  // good for are pulled, as they would be there
  const bool fits = fused_fits(g, pulls ? kFusedPrdEdges : kFusedPrdPushEdges);
  const bool small = fits && n <= (pulls ? kFusedPrdVertices : kFusedPrdPushVertices);
  if (fits && !small) pulls = true;
  // (2^20 vertices with 4e6 empty rows among them: 1120 ms pulled, 2.7 pushed)
  if (pulls && !small && !short_chunks(g, st)) {
    pulls = false;
    g_opts.direction = 0;  // (until the call returns)
  }
  // the per-vertex arrays in one allocation, whole 2 MiB pages each (apart, their
  // placement moves the gathers' speed)
  const size_t page = 2u << 20, row = ((size_t)n * 8 + page - 1) / page * page;
  auto reserve_rows = [&](int rows) { return S.arrays.reserve(rows * row); };
  auto reserve_levels = [&]() -> rg_status {
    if (pulls && reserve_rows(6) != RG_OK) {  // pushed, without the exact sums' 16 bytes a vertex
      clear_error();
      pulls = false;
      g_opts.direction = 0;
    }
    return reserve_rows(pulls ? 6 : 4);
  };
  RG_TRY(small ? reserve_rows(3) : reserve_levels());
  RG_TRY(S.totals.reserve(sizeof(PrdTotals) * (kPulledRounds + 1)));
  RG_TRY(frontier_alloc(g, S.f[0]));
  RG_TRY(frontier_alloc(g, S.f[1]));
  const double one_over_n = 1 / (double)n;
  const double added = (1 - kPrDamp) * one_over_n;  // PageRankDelta.C:55
  auto array = [&](int i) { return reinterpret_cast<double*>(S.arrays.as<unsigned char>() + i * row); };
  double *p = array(0), *ngh = array(1), *c = array(2);
  PrdTotals* totals = S.totals.as<PrdTotals>();
  const int vblocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)device_sms() * 16);
  int64_t round = 0;
  double l1 = 0.0;
  CallTimer timer(g);
  bool whole = false, launched = false;  // answered by one launch
  if (small) {
    RG_TRY(prd_fused_run(g, true, 0, max_iters, p, ngh, c, S.f[0].bits.as<uint32_t>(), nullptr, &round, &l1, &launched,
                         &whole));
  }
  if (!whole) {
    if (small) {
      RG_TRY(reserve_levels());
      p = array(0), ngh = array(1), c = array(2);
    }
    unsigned long long* rmag = reinterpret_cast<unsigned long long*>(array(3));
    U128* acc = pulls ? reinterpret_cast<U128*>(array(4)) : nullptr;
    FView cur = view_of(S.f[0]), nxt = view_of(S.f[1]);
    bool queued = false;  // cur's queue is that of its bits
    auto start = [&]() -> rg_status {
      prd_init<<<vblocks, 256, 0, st>>>((uint32_t)n, g->off.as<uint32_t>(), p, ngh, c, rmag, S.f[0].bits.as<uint32_t>(),
                                        one_over_n);
      RG_CUDA(cudaGetLastError());
      g_timing.kernel_launches++;
      if (acc) RG_CUDA(cudaMemsetAsync(acc, 0, sizeof(U128) * n, st));
      cur = view_of(S.f[0]);
      nxt = view_of(S.f[1]);
      cur.count = n;
      cur.degsum = g->m;
      queued = false;
      return RG_OK;
    };
    RG_TRY(start());
    EmOpts o;
    o.variant = variant;
    o.dense_forward = true;  // no_output | dense_forward; what pulls is swept below
    Workspace& ws = cx->ws;
    const int64_t threshold = g->m / std::max<int64_t>(g_opts.dense_div, 1);
    auto filter_args = [&](auto filter, const PrdGate& gate, PrdTotals* t) {
      g_timing.kernel_launches++;
      return launch_following(filter, vblocks, 256, 0, st, (uint32_t)n, g->off.as<uint32_t>(), g->in_view().off, p, ngh,
                              acc, c, rmag, one_over_n, added, cur.bits, nxt.bits, gate, t);
    };
    bool hand_over = !g_trace_on && strides_fit(n, g->m);  // sparse rounds go to one launch (once)
    while (round++ < max_iters) {
      const bool dense = cur.count + cur.degsum > threshold;
      if (!dense && round > 1 && hand_over) {
        bool done = false;
        launched = false;
        RG_TRY(prd_fused_run(g, false, round - 1, max_iters, p, ngh, c, cur.bits, nullptr, &round, &l1, &launched,
                             &done));
        if (done) break;
        hand_over = false;
        if (launched) {  // gave up, having changed p, ngh and c: the run starts again, level by level
          RG_TRY(start());
          round = 0;
          continue;
        }
      }
      if (dense && g->m > 0 && pulls) {
        const int k = (int)std::min<int64_t>(kPulledRounds, max_iters - round + 1);
        RG_CUDA(cudaMemsetAsync(totals, 0, sizeof(PrdTotals) * k, st));
        for (int i = 0; i < k; i++) {
          const PrdGate gate{i ? totals + i - 1 : nullptr, threshold};
          RG_TRY(exact_pull_signed(g, c, acc, gate, st));
          RG_CUDA(filter_args(round + i == 1 ? prd_filter<true, true> : prd_filter<false, true>, gate, totals + i));
          std::swap(cur, nxt);
        }
        PrdTotals t[kPulledRounds];
        RG_TRY(read_small(totals, t, sizeof(PrdTotals) * k, st));
        if (k % 2) std::swap(cur, nxt);  // back to where the first of them began
        for (int i = 0;; i++) {
          g_timing.edges_traversed += cur.degsum;
          g_timing.edge_launches++;
          std::swap(cur, nxt);
          cur.count = (int64_t)t[i].count;
          cur.degsum = (int64_t)t[i].degsum;
          l1 = t[i].l1;
          if (l1 < kPrdEps || i + 1 == k || !((int64_t)(t[i].count + t[i].degsum) > threshold)) break;
          round++;
        }
        queued = false;
      } else {
        if (!queued) {
          Frontier shell;  // non-owning view of cur for the compaction (which syncs)
          shell.bits.p = cur.bits;
          RG_TRY(compact_bits(g, shell, st, true, nullptr, 0, nullptr, cur.queue, cur.qoff));
          shell.bits.p = nullptr;
          g_timing.kernel_launches += 3;
          queued = true;
        }
        RG_TRY(edge_map(g, cur, OpPrDelta{c, ngh}, nullptr, o, st));
        RG_CUDA(cudaMemsetAsync(totals, 0, sizeof(PrdTotals), st));
        RG_CUDA(filter_args(round == 1 ? prd_filter<true, false> : prd_filter<false, false>, PrdGate{nullptr, 0}, totals));
        std::swap(cur, nxt);
        RG_CUDA(cudaMemcpyAsync(&ws.h_info[4], &totals->l1, 8, cudaMemcpyDeviceToHost, st));
        Frontier shell;
        shell.bits.p = cur.bits;
        RG_TRY(compact_bits(g, shell, st, true, nullptr, 0, nullptr, cur.queue, cur.qoff));
        shell.bits.p = nullptr;
        cur.count = shell.count;
        cur.degsum = shell.degsum;
        queued = true;
        g_timing.kernel_launches += 3;
        memcpy(&l1, &ws.h_info[4], 8);
      }
      if (l1 < kPrdEps) break;  // PageRankDelta.C:144
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
