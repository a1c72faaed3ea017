// Triangle counting (GAP tc_local, src/*/GAP/src/tc_local.cc:49-157) on the
// device.
//
// In degree order (descending, ties by descending id, the order of
// builder.h:247-282 and of the degree sort) every vertex u keeps its lower list
// L(u): its neighbours below u, ascending.  A triangle is counted once, as
// u > v > w: for every v in L(u) the common members of L(u) and L(v) (all of
// them below v).  Lower lists hold only higher-degree neighbours, so they stay
// short on skewed graphs.  Per-vertex counts (triangles containing each vertex)
// are returned by original id; counts of the w's among the first ids are kept
// per CTA in shared memory and merged once per CTA -- the RADAR variant's
// per-thread copies of triangles[u] for u < numHubs (tc_local.cc:54-96).
//
// The lower lists come from one stable sort: walking the rows v in order and
// keeping the neighbours u > v yields the pairs (u, v) ordered by v, so sorting
// them by u alone leaves every list ascending.  That holds for a cleaned symmetric
// graph; one with repeats, or with edges in one direction alone, is cleaned first.

#include <cuda_runtime.h>

#include <algorithm>

#include "app_common.cuh"
#include "sort.cuh"

namespace rg {

namespace {

constexpr unsigned kAll = 0xffffffffu;

// An edge's share of a sum that is 0 over both directions of every edge (and, but for
// chance in 2^64, over nothing else that is not balanced): negative from the lower id.
__device__ __forceinline__ unsigned long long edge_share(uint32_t u, uint32_t v) {
  unsigned long long x = ((unsigned long long)max(u, v) << 32 | min(u, v)) * 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 29)) * 0xD6E8FEB86659FD93ull;
  x ^= x >> 32;
  return u > v ? x : u < v ? 0ull - x : 0ull;
}

// The pairs (u, v), u > v, of a symmetric graph, ordered by v: counted per
// kSweepChunk edges (a warp each; rows from the chunk starts) with the sum of the
// edges' shares (balance), then written as u << bits | v at the chunk's place with the
// digit counts of the sort by u.
// Bound by the row searches' latency: four edges per lane share one (7.3e6 entries:
// 42 and 47 us with a search each, 19 and 30 now).
template <bool kEmit>
__global__ void __launch_bounds__(256) upper_pairs(DevGraph g, const uint32_t* __restrict__ chunk_v, uint32_t nchunks,
                                                   uint32_t* __restrict__ count, const uint32_t* __restrict__ place,
                                                   int bits, uint64_t* __restrict__ key, int passes, uint32_t* hist,
                                                   unsigned long long* balance) {
  __shared__ uint32_t sh[kEmit ? kMaxSortPasses * 256 : 1];
  if (kEmit) sort_zero(sh, passes);
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long sum = 0;
  for (uint32_t c = warp; c < nchunks; c += nwarps) {
    const uint32_t vlo = chunk_v[c], vhi = chunk_v[c + 1];
    uint32_t n = 0, at = kEmit ? place[c] : 0;
    // four edges per lane: one row search for them
    for (int r = 0; r < kSweepChunk / 128; r++) {
      const uint32_t e = c * kSweepChunk + r * 128 + lane * 4;
      uint32_t u[4] = {}, v[4] = {}, own = 0;
      if (e < g.m) {
        const uint4 x = __ldg(reinterpret_cast<const uint4*>(g.adj + e));  // adj is padded past m
        u[0] = x.x, u[1] = x.y, u[2] = x.z, u[3] = x.w;
        uint32_t row = upper_index(g.off, vlo, vhi, e), next = g.off[row + 1];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          while (e + k < g.m && e + k >= next) next = g.off[++row + 1];
          v[k] = row;
          if (e + k >= g.m) u[k] = v[k];
          own += u[k] > v[k];
          if (!kEmit) sum += edge_share(u[k], v[k]);
        }
      }
      if (!kEmit) {
        n += own;
        continue;
      }
      uint32_t inc = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kAll, inc, o);
        if (lane >= o) inc += t;
      }
      uint32_t to = at + inc - own;
      at += __shfl_sync(kAll, inc, 31);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (u[k] <= v[k]) continue;
        const uint64_t x = ((uint64_t)u[k] << bits) | v[k];
        key[to++] = x;
        sort_count_key(sh, x, bits, 2 * bits, passes);
      }
    }
    if (!kEmit) {
      n = __reduce_add_sync(kAll, n);
      if (lane == 0) count[c] = n;
    }
  }
  if (kEmit) {
    sort_flush(sh, hist, passes);
  } else {
    sum = warp_sum(sum);
    if (lane == 0 && sum) atomicAdd(balance, sum);
  }
}

constexpr int kTcThreads = 512;
constexpr int kTcWarps = kTcThreads / 32;
constexpr uint32_t kMarkIds = 16384;  // ids with a bit in a warp's marks (2 KiB)
constexpr uint32_t kHubIds = 4096;    // ids with a counter per CTA (16 KiB)

constexpr uint32_t kTake = 4;

struct TcShared {
  uint32_t mark[kTcWarps][kMarkIds / 32];
  uint32_t hub[kHubIds];
  uint32_t found[kTcWarps][32];  // per edge of a warp's group
};

// A warp takes 32 edges at a time, one per lane, in the order of the graph's rows
// v; the neighbours u > v count.
//  * Where one of L(v) and L(u) is far shorter than the other (or v is past the
//    ids that a bitmap covers), its members are searched in the other; the searches of all such edges are
//    dealt out to the lanes together, so a tail vertex with two or three lower
//    neighbours does not idle a warp.
//  * Otherwise, v being a high-degree vertex, L(v) is marked in the warp's bitmap,
//    once for all of a row's edges, and L(u) streamed against it as far as v: 32
//    members per load where a search step gathers 32 lines.  (Marking L(u) and
//    streaming L(v) reads 2.7 times as much on R-MAT s18: the members of L(u)
//    below v are few where v is a hub, all of L(v) are not.)
// What bounds it is the streamed members: a bitmap lookup each and a shared-memory
// add per triangle.  R-MAT, 2e5 vertices, 3.6e6 edges, 8e7 triangles: 4061 us by
// a merge or search per lane, 880 us streaming L(v) at half the occupancy.
// A w meets a given edge at most once, so a CTA adds at most 32 per group to a
// hub counter: fewer than 2^32 over the fewer than 2^27 groups of any graph.
__global__ void __launch_bounds__(kTcThreads, 4) count_triangles(DevGraph g, const uint32_t* __restrict__ chunk_v,
                                                                const uint32_t* __restrict__ off,
                                                                const uint32_t* __restrict__ adj, unsigned int* next,
                                                                unsigned long long* tri, unsigned long long* total) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TcShared& S = *reinterpret_cast<TcShared*>(smem_raw);
  for (uint32_t i = threadIdx.x; i < kTcWarps * (kMarkIds / 32); i += kTcThreads) (&S.mark[0][0])[i] = 0u;
  for (uint32_t i = threadIdx.x; i < kHubIds; i += kTcThreads) S.hub[i] = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t* mark = S.mark[w];
  uint32_t* found = S.found[w];
  const uint32_t groups = (g.m + 31) / 32;
  unsigned long long sum = 0;
  auto hit = [&](uint32_t x) {
    if (x < kHubIds) atomicAdd(S.hub + x, 1u);
    else atomicAdd(tri + x, 1ull);
  };
  uint32_t t = 0, end = 0;
  for (;; t++) {
    if (t >= end) {  // groups are taken kTake at a time: one counter serves every warp
      if (lane == 0) t = atomicAdd(next, (unsigned)kTake);
      t = __shfl_sync(kAll, t, 0);
      if (t >= groups) break;
      end = min(t + kTake, groups);
    }
    const uint32_t e = t * 32 + lane, ch = t / (kSweepChunk / 32);
    uint32_t u = 0, v = 0, a = 0, la = 0, b = 0, lb = 0;
    if (e < g.m) {
      u = g.adj[e];
      v = upper_index(g.off, chunk_v[ch], chunk_v[ch + 1], e);
      if (u > v) {
        b = off[v];
        lb = off[v + 1] - b;
        a = off[u];
        la = lb ? min(off[u + 1] - a, v) : 0u;  // at least L(u)'s members below v
      }
    }
    const uint32_t lo = min(la, lb), hi = max(la, lb);
    if (!__any_sync(kAll, lo > 0)) continue;
    found[lane] = 0u;
    const bool search = lo > 0 && (lo <= 8 || lo * 32 <= hi || v >= kMarkIds);
    // searches: item t of the group's concatenated short lists
    uint32_t inc = search ? lo : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(kAll, inc, o);
      if (lane >= o) inc += x;
    }
    const uint32_t items = __shfl_sync(kAll, inc, 31);
    const uint32_t sp = la <= lb ? a : b, lp = la <= lb ? b : a;  // where the short and the long list begin
    __syncwarp();
    for (uint32_t i0 = 0; i0 < items; i0 += 32) {
      const uint32_t i = i0 + lane;
      int j = 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        if (__shfl_sync(kAll, inc, j + o - 1) <= i) j += o;
      }
      j &= 31;
      const uint32_t js = __shfl_sync(kAll, sp, j), jl = __shfl_sync(kAll, lp, j), jh = __shfl_sync(kAll, hi, j);
      const uint32_t jn = __shfl_sync(kAll, lo, j), first = __shfl_sync(kAll, inc, j) - jn;
      if (i < items) {
        const uint32_t x = adj[js + (i - first)];
        uint32_t l = 0, h = jh;
        while (l < h) {
          const uint32_t mid = (l + h) >> 1;
          if (adj[jl + mid] < x) l = mid + 1;
          else h = mid;
        }
        if (l < jh && adj[jl + l] == x) {
          atomicAdd(found + j, 1u);
          hit(x);
        }
      }
    }
    __syncwarp();
    uint32_t marked = kNone, mb = 0, mn = 0;  // the v whose list is marked
    auto unmark = [&] {
      __syncwarp();
      for (uint32_t i = lane; i < mn; i += 32) mark[adj[mb + i] >> 5] = 0u;
      __syncwarp();
    };
    for (unsigned todo = __ballot_sync(kAll, lo > 0 && !search); todo; todo &= todo - 1) {
      const int j = __ffs(todo) - 1;
      const uint32_t jv = __shfl_sync(kAll, v, j), ja = __shfl_sync(kAll, a, j), jn = __shfl_sync(kAll, la, j);
      if (jv != marked) {
        unmark();
        marked = jv;
        mb = __shfl_sync(kAll, b, j);
        mn = __shfl_sync(kAll, lb, j);
        for (uint32_t i = lane; i < mn; i += 32) {  // v < kMarkIds, so every member has a bit
          const uint32_t x = adj[mb + i];
          atomicOr(mark + (x >> 5), 1u << (x & 31));
        }
        __syncwarp();
      }
      uint32_t c = 0;
      for (uint32_t i0 = 0; i0 < jn; i0 += 128) {
        uint32_t x[4];
#pragma unroll
        for (int k = 0; k < 4; k++) x[k] = i0 + 32 * k + lane < jn ? adj[ja + i0 + 32 * k + lane] : kNone;
        if (__shfl_sync(kAll, x[0], 0) >= jv) break;  // the rest lies above v
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (x[k] < jv && ((mark[x[k] >> 5] >> (x[k] & 31)) & 1u)) {
            c++;
            hit(x[k]);
          }
        }
      }
      c = __reduce_add_sync(kAll, c);
      if (lane == j) found[lane] += c;
    }
    unmark();
    const uint32_t c = found[lane];
    const uint32_t v0 = __shfl_sync(kAll, v, 0);
    if (c) atomicAdd(tri + u, (unsigned long long)c);
    if (__all_sync(kAll, v == v0 || c == 0)) {  // one row: one add for it
      const uint32_t cs = __reduce_add_sync(kAll, c);
      if (lane == 0 && cs) atomicAdd(tri + v0, (unsigned long long)cs);
    } else if (c) {
      atomicAdd(tri + v, (unsigned long long)c);
    }
    sum += c;
    __syncwarp();
  }
  sum = warp_sum(sum);
  if (lane == 0 && sum) atomicAdd(total, sum);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < min(kHubIds, g.n); i += kTcThreads) {
    if (S.hub[i]) atomicAdd(tri + i, (unsigned long long)S.hub[i]);
  }
}

struct TcState {
  DevBuf tri, total, out;
};

// The entries of a graph, one by one.
__global__ void __launch_bounds__(256) entry_ends(DevGraph g, const uint32_t* __restrict__ chunk_v, uint32_t* src,
                                                  uint32_t* dst) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < g.m; e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t c = (uint32_t)(e / kSweepChunk);
    src[e] = upper_index(g.off, chunk_v[c], chunk_v[c + 1], (uint32_t)e);
    dst[e] = g.adj[e];
  }
}

// The graph with both directions of every edge of g, each once.
rg_status cleaned(rg_graph* g, rg_graph** out, cudaStream_t st) {
  DevBuf ends(true, st);
  RG_TRY(ends.reserve(8 * (size_t)g->m));
  uint32_t *src = ends.as<uint32_t>(), *dst = src + g->m;
  entry_ends<<<(unsigned)(device_sms() * 16), 256, 0, st>>>(g->view(), g->chunk_v.as<uint32_t>(), src, dst);
  RG_CUDA(cudaGetLastError());
  return rg_graph_create_from_edges(g->n, g->m, src, dst, 1, out);
}

// Lower lists of the degree-ordered graph rs, and their members' count.  *clean:
// whether every edge of rs is there once in either direction (else the lists are not
// rs's).
rg_status lower_lists(rg_graph* rs, DevBuf& off, DevBuf& adj, int64_t* entries, bool* clean, cudaStream_t st) {
  const int64_t n = rs->n;
  const uint32_t nchunks = (uint32_t)rs->nchunks;
  int bits = 1;
  while (bits < 32 && ((uint64_t)(n - 1) >> bits) != 0) bits++;
  const int passes = sort_passes(bits, 2 * bits);
  DevBuf place(true, st), k0(true, st), k1(true, st);
  SortScratch sort(st);
  const uint32_t sum_at = (nchunks + 2) & ~1u;  // the balance, behind the scan's total
  RG_TRY(place.reserve(4 * ((size_t)sum_at + 2)));
  uint32_t* pl = place.as<uint32_t>();
  RG_CUDA(cudaMemsetAsync(pl + sum_at, 0, 8, st));
  const unsigned blocks =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>((rs->nchunks * 32 + 255) / 256, (int64_t)device_sms() * 8));
  upper_pairs<false><<<blocks, 256, 0, st>>>(rs->view(), rs->chunk_v.as<uint32_t>(), nchunks, pl, nullptr, bits,
                                             nullptr, passes, nullptr,
                                             reinterpret_cast<unsigned long long*>(pl + sum_at));
  RG_CUDA(cudaGetLastError());
  RG_TRY(scan_u32(ctx().ws, pl, pl, nchunks, st));
  uint32_t read[4];  // the total, the balance in the last two
  RG_TRY(read_small(pl + nchunks, read, 4 * (sum_at + 2 - nchunks), st));
  const uint32_t k = read[0];
  *entries = k;
  *clean = (read[sum_at - nchunks] | read[sum_at + 1 - nchunks]) == 0;
  if (k == 0 || !*clean) return RG_OK;
  RG_TRY(k0.reserve(8 * (size_t)k));
  RG_TRY(k1.reserve(8 * (size_t)k));
  RG_TRY(sort_begin(sort, k, passes, st));
  upper_pairs<true><<<blocks, 256, 0, st>>>(rs->view(), rs->chunk_v.as<uint32_t>(), nchunks, nullptr, pl, bits,
                                            k0.as<uint64_t>(), passes, sort_counts(sort), nullptr);
  RG_CUDA(cudaGetLastError());
  uint64_t *key = k0.as<uint64_t>(), *other = k1.as<uint64_t>();
  RG_TRY(sort_run(sort, &key, &other, k, bits, 2 * bits, st));
  g_timing.kernel_launches += 3 + passes;
  RG_TRY(csr_from_sorted_rows(ctx().ws, key, k, bits, n, true, off, adj, entries, sort, "lower lists", st));
  *clean = *entries == k;
  return RG_OK;
}

}  // namespace

rg_status triangle_run(rg_graph* g, uint64_t* h_counts, uint64_t* total_out) {
  if (!g) return fail(RG_EINVAL, "null graph");
  if (g->directed) return fail(RG_EUNSUPPORTED, "triangle counting needs an undirected graph (tc_local.cc:21-25)");
  Ctx* cx = nullptr;
  RG_TRY(get_ctx(&cx));
  cudaStream_t st = cx->stream;
  const int64_t n = g->n, m = g->m;
  static thread_local TcState S;
  CallTimer timer(g);
  RG_TRY(S.tri.reserve(8 * (size_t)n));
  RG_TRY(S.total.reserve(16));
  RG_TRY(S.out.reserve(8 * (size_t)n));
  unsigned long long* tri = S.tri.as<unsigned long long>();
  unsigned long long* total = S.total.as<unsigned long long>();
  // degree order (the relabelled graph of the sort, or g itself when sorted)
  rg_graph* rs = g;
  rg_graph* tmp = nullptr;
  if (!g->sorted) {
    RG_TRY(rg_graph_degree_sort(g, &tmp, nullptr));
    rs = tmp;
  }
  uint64_t t = 0;
  rg_graph* gt = nullptr;  // rs cleaned, where it needs that
  auto count = [&]() -> rg_status {
    RG_CUDA(cudaMemsetAsync(tri, 0, 8 * n, st));
    RG_CUDA(cudaMemsetAsync(total, 0, 16, st));
    DevBuf off(true, st), adj(true, st);
    int64_t k = 0;
    bool clean = true;
    if (m > 0) RG_TRY(lower_lists(rs, off, adj, &k, &clean, st));
    if (!clean) {
      RG_TRY(cleaned(rs, &gt, st));
      RG_TRY(lower_lists(gt, off, adj, &k, &clean, st));
    }
    rg_graph* const lists = gt ? gt : rs;
    if (k > 0) {
      static std::atomic<uint64_t> limit_set{0};
      RG_TRY(allow_max_dyn_smem(limit_set, count_triangles));
      const int64_t grid = std::min<int64_t>((lists->m + 32 * kTcWarps - 1) / (32 * kTcWarps), (int64_t)device_sms() * 4);
      kt_begin(st);
      count_triangles<<<(unsigned)grid, kTcThreads, sizeof(TcShared), st>>>(
          lists->view(), lists->chunk_v.as<uint32_t>(), off.as<uint32_t>(), adj.as<uint32_t>(),
          (unsigned int*)(total + 1), tri, total);
      kt_end(st);
      RG_CUDA(cudaGetLastError());
      g_timing.kernel_launches++;
      g_timing.edge_launches++;
    }
    if (h_counts) {  // by original id: rs's permutation maps g's ids to the order's
      const int64_t blocks = std::min<int64_t>((n + 255) / 256, (int64_t)device_sms() * 32);
      gather_kernel<unsigned long long><<<(unsigned)blocks, 256, 0, st>>>(tri, rs->new_ids.as<uint32_t>(), n,
                                                                          S.out.as<unsigned long long>());
      RG_CUDA(cudaGetLastError());
      RG_CUDA(cudaMemcpyAsync(h_counts, S.out.p, 8 * n, cudaMemcpyDeviceToHost, st));
    }
    return read_small(total, &t, 8, st);
  };
  const rg_status s = count();
  if (gt) rg_graph_free(gt);
  if (tmp) rg_graph_free(tmp);
  RG_TRY(s);
  RG_TRY(timer.stop());
  g_timing.edges_traversed = m;
  if (total_out) *total_out = t;
  return RG_OK;
}

}  // namespace rg

extern "C" rg_status rg_triangle_count(rg_graph* g, uint64_t* h_counts, uint64_t* total_out) {
  return rg::triangle_run(g, h_counts, total_out);
}
