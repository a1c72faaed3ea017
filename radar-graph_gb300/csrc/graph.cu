// Device graph image, scans, frontier compaction and the degree-sort relabel.
//
// Degree sort (preprocessGraph, IO.h:843-895): the reference sorts
// pair<degree, id> with std::greater, i.e. degree descending and ties by
// DEScending original id, and gives rank r to the r-th pair.  Here a stable
// LSD radix sort on the 32-bit key ~degree runs over ids laid out in
// descending order, which yields exactly that order (the sort is stable, so
// equal degrees keep the descending-id input order).  Neighbour lists are then
// relabelled in place order (IO.h:877-895 keeps the order, it does not
// re-sort).

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#include "app_common.cuh"
#include "rg_device.cuh"
#include "sort.cuh"

namespace rg {

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------
static thread_local char g_err[512] = "";

rg_status fail(rg_status s, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
  return s;
}
void clear_error() { g_err[0] = 0; }
const char* last_error() { return g_err; }

rg_status cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
  const char* f = strrchr(file, '/');
  fail(e == cudaErrorMemoryAllocation ? RG_ENOMEM : RG_ECUDA, "%s: %s (%s:%d)",
       cudaGetErrorString(e), what, f ? f + 1 : file, line);
  cudaGetLastError();  // clear a sticky-free error so the context stays usable
  return e == cudaErrorMemoryAllocation ? RG_ENOMEM : RG_ECUDA;
}

rg_status DevBuf::reserve(size_t b) {
  if (b <= bytes && p) return RG_OK;
  release();
  const rg_status s = allocate(b);
  if (s != RG_ENOMEM || !release_idle_arena()) return s;
  clear_error();
  return allocate(b);
}

rg_status DevBuf::allocate(size_t b) {
  size_t want = b < 256 ? 256 : b;
  if (pooled && on_stream) {  // used and released in its stream's order
    RG_CUDA(cudaMallocAsync(&p, want, free_stream));
  } else if (pooled) {  // usable from every stream once the allocating stream has it
    RG_CUDA(cudaMallocAsync(&p, want, 0));
    RG_CUDA(cudaStreamSynchronize(0));
  } else {
    RG_CUDA(cudaMalloc(&p, want));
  }
  bytes = want;
  return RG_OK;
}

Workspace::~Workspace() {
  if (h_info) cudaFreeHost(h_info);
  if (h_small) cudaFreeHost(h_small);
}

__global__ void read_small_kernel(const unsigned char* __restrict__ src, volatile unsigned char* dst, size_t bytes) {
  for (size_t i = threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
  __threadfence_system();
}

rg_status read_small(const void* d_src, void* h_dst, size_t bytes, cudaStream_t st) {
  if (bytes == 0) return RG_OK;
  Ctx* c = nullptr;
  RG_TRY(get_ctx(&c));
  Workspace& ws = c->ws;
  if (bytes > kSmallRead || !ws.h_small_dev) {
    RG_CUDA(cudaMemcpyAsync(h_dst, d_src, bytes, cudaMemcpyDeviceToHost, st));
    RG_CUDA(cudaStreamSynchronize(st));
    return RG_OK;
  }
  read_small_kernel<<<1, 256, 0, st>>>(static_cast<const unsigned char*>(d_src), ws.h_small_dev, bytes);
  RG_CUDA(cudaGetLastError());
  RG_CUDA(cudaStreamSynchronize(st));
  memcpy(h_dst, ws.h_small, bytes);
  return RG_OK;
}

void* device_alias(const void* p, size_t bytes, size_t align) {
  typedef CUresult (*GetAttributes)(unsigned int, CUpointer_attribute*, void**, CUdeviceptr);
  static const GetAttributes get = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<GetAttributes>(f);
  }();
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  if (!p || !get || at % align) return nullptr;
  unsigned int type = 0, managed = 0;
  CUdeviceptr dev = 0, start = 0;
  size_t size = 0;
  CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void* into[] = {&type, &managed, &dev, &start, &size};
  if (get(5, what, into, (CUdeviceptr)at) != CUDA_SUCCESS) return nullptr;
  if (type != CU_MEMORYTYPE_HOST || managed || !dev || !start || dev < start || dev - start > size) return nullptr;
  return size - (dev - start) >= bytes ? reinterpret_cast<void*>(dev) : nullptr;
}

static thread_local Ctx* t_ctx = nullptr;

rg_status get_ctx(Ctx** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(RG_ENODEV, "no CUDA device: %s", cudaGetErrorString(e));
  }
  if (t_ctx && t_ctx->device == dev) {
    *out = t_ctx;
    return RG_OK;
  }
  // a thread that switches devices keeps one context per process lifetime of
  // the last device used; the old one is released
  delete t_ctx;
  t_ctx = nullptr;
  Ctx* c = new (std::nothrow) Ctx();
  if (!c) return fail(RG_ENOMEM, "host allocation failed");
  c->device = dev;
  {  // freed pool blocks stay mapped for reuse (graph images are large)
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
      uint64_t keep = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    cudaGetLastError();
  }
  if (cudaStreamCreateWithFlags(&c->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess ||
      cudaHostAlloc((void**)&c->ws.h_info, 64, cudaHostAllocMapped) != cudaSuccess ||
      cudaHostGetDevicePointer((void**)&c->ws.h_info_dev, c->ws.h_info, 0) != cudaSuccess ||
      cudaHostAlloc((void**)&c->ws.h_small, kSmallRead, cudaHostAllocMapped) != cudaSuccess ||
      cudaHostGetDevicePointer((void**)&c->ws.h_small_dev, c->ws.h_small, 0) != cudaSuccess ||
      c->ws.counters.reserve(4096) != RG_OK) {
    cudaGetLastError();
    delete c;
    return fail(RG_ECUDA, "stream/event/pinned allocation failed");
  }
  cudaMemset(c->ws.counters.p, 0, 4096);
  c->stream = c->own_stream;
  t_ctx = c;
  *out = c;
  return RG_OK;
}

Ctx& ctx() { return *t_ctx; }

// Binary search, degrees non-increasing: the first v with at most t entries.
__global__ void find_pull_split(const uint32_t* __restrict__ off, uint32_t n, uint32_t t, uint32_t* out) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (off[mid + 1] - off[mid] <= t) hi = mid;
    else lo = mid + 1;
  }
  *out = lo;
}

uint32_t pull_split(const rg_graph* g, const DevGraph& pull_g, cudaStream_t st) {
  int64_t v = g->pull_split.load(std::memory_order_relaxed);
  if (v >= 0) return (uint32_t)v;
  Ctx* c = nullptr;
  if (get_ctx(&c) != RG_OK) return pull_g.n;  // a hint only: one group size for every vertex
  Workspace& ws = c->ws;
  uint32_t* d = reinterpret_cast<uint32_t*>(ws.counters.as<uint64_t>() + 8);  // a free scratch word
  find_pull_split<<<1, 1, 0, st>>>(pull_g.off, pull_g.n, 8u, d);
  uint32_t h = pull_g.n;
  if (cudaGetLastError() != cudaSuccess || read_small(d, &h, 4, st) != RG_OK) {
    cudaGetLastError();
    return pull_g.n;  // a hint only: one group size for every vertex
  }
  g->pull_split.store(h, std::memory_order_relaxed);
  return h;
}

rg_status copy_stream(cudaStream_t* out) {
  Ctx* c = nullptr;
  RG_TRY(get_ctx(&c));
  if (!c->copy_stream) RG_CUDA(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
  *out = c->copy_stream;
  return RG_OK;
}

}  // namespace rg

extern "C" rg_status rg_set_stream(void* stream) {
  rg::Ctx* c = nullptr;
  RG_TRY(rg::get_ctx(&c));
  c->stream = stream ? (cudaStream_t)stream : c->own_stream;
  return RG_OK;
}

namespace rg {

// ---------------------------------------------------------------------------
// exclusive scan of uint32 (three kernels: tile sums, scan of sums, apply)
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

template <int kThreads>
__device__ __forceinline__ uint32_t block_exclusive_sum(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_tot[kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) warp_tot[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t t = lane < kThreads / 32 ? warp_tot[lane] : 0;
    uint32_t ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t u = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= o) ti += u;
    }
    if (lane < kThreads / 32) warp_tot[lane] = ti - t;
    if (lane == kThreads / 32 - 1) *total = ti;
  }
  __syncthreads();
  uint32_t r = warp_tot[w] + inc - v;
  __syncthreads();
  return r;
}

__global__ void scan_tile_sums(const uint32_t* __restrict__ in, int64_t n, uint32_t* __restrict__ sums) {
  int64_t base = (int64_t)blockIdx.x * kScanTile;
  uint32_t s = 0;
  for (int i = 0; i < kScanItems; i++) {
    int64_t idx = base + (int64_t)i * kScanThreads + threadIdx.x;
    if (idx < n) s += in[idx];
  }
  __shared__ uint32_t tot;
  block_exclusive_sum<kScanThreads>(s, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// One block scans `nt` tile sums in place (exclusive) and writes the total.
__global__ void scan_sums(uint32_t* sums, int64_t nt, uint32_t* total_out) {
  __shared__ uint32_t carry_s, tot;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int64_t base = 0; base < nt; base += kScanThreads) {
    int64_t i = base + threadIdx.x;
    uint32_t v = i < nt ? sums[i] : 0;
    uint32_t ex = block_exclusive_sum<kScanThreads>(v, &tot);
    uint32_t c = carry_s;
    if (i < nt) sums[i] = c + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry_s = c + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total_out = carry_s;
}

__global__ void scan_apply(const uint32_t* __restrict__ in, int64_t n, const uint32_t* __restrict__ sums,
                           uint32_t* __restrict__ out) {
  // each thread scans kScanItems consecutive elements
  int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    int64_t idx = base + i;
    v[i] = idx < n ? in[idx] : 0;
    s += v[i];
  }
  __shared__ uint32_t tot;
  uint32_t ex = block_exclusive_sum<kScanThreads>(s, &tot) + sums[blockIdx.x];
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    int64_t idx = base + i;
    if (idx < n) out[idx] = ex;
    ex += v[i];
  }
}

rg_status scan_u32(Workspace& ws, const uint32_t* in, uint32_t* out, int64_t n, cudaStream_t st) {
  int64_t nt = (n + kScanTile - 1) / kScanTile;
  if (nt == 0) nt = 1;
  RG_TRY(ws.scan_tmp.reserve(sizeof(uint32_t) * (nt + 1)));
  uint32_t* sums = ws.scan_tmp.as<uint32_t>();
  if (n > 0) scan_tile_sums<<<(unsigned)nt, kScanThreads, 0, st>>>(in, n, sums);
  else RG_CUDA(cudaMemsetAsync(sums, 0, 4, st));
  scan_sums<<<1, kScanThreads, 0, st>>>(sums, nt, out + n);
  if (n > 0) scan_apply<<<(unsigned)nt, kScanThreads, 0, st>>>(in, n, sums, out);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

// ---------------------------------------------------------------------------
// bitmap -> ascending queue + degree scan (ligra.h:161-192 compaction,
// vertexSubset.h:196-211 toSparse)
// ---------------------------------------------------------------------------
constexpr int kCompThreads = 256;
// Words per lane: a warp emits its non-zero words one after another, each
// step waiting on its offsets, so fewer words per warp means more warps to
// hide that latency (RMAT s24 four-app step: 8 words 50.2 ms, 2 words
// 49.1 ms, 1 word 49.5 ms).
constexpr int kCompWords = 2;
constexpr int kCompTile = kCompThreads * kCompWords;  // words per block
constexpr int kCompWarps = kCompThreads / 32;
constexpr int kWarpWords = kCompWords * 32;  // consecutive words per warp

// Count and degree sum of the set bits of word x (vertices vb .. vb+31).  The
// degrees of a run of consecutive set bits [a, e) telescope to
// off[vb+e] - off[vb+a], so a dense word costs two loads, not 64.  Bits at
// or above n are never set, so vb + e <= n.
__device__ __forceinline__ void word_count_deg(uint32_t x, uint32_t vb, const uint32_t* __restrict__ off,
                                               uint32_t& c, uint32_t& d) {
  c += __popc(x);
  uint32_t starts = x & ~(x << 1);
  while (starts) {
    const int a = __ffs(starts) - 1;
    starts &= starts - 1;
    const uint32_t rest = ~x >> a;  // bit 0 is clear: bit a of x is set
    const int e = rest ? a + __ffs(rest) - 1 : 32;
    d += off[vb + e] - off[vb + a];
  }
}

// A warp owns kWarpWords consecutive words, lane l the words l, l+32, ...
// (coalesced loads of the bitmap).
__device__ __forceinline__ void warp_words(const uint32_t* __restrict__ bits, int64_t nwords, int64_t wbase,
                                           uint32_t (&xs)[kCompWords]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < kCompWords; i++) {
    const int64_t w = wbase + i * 32 + lane;
    xs[i] = w < nwords ? bits[w] : 0u;
  }
}

__global__ void comp_count(const uint32_t* __restrict__ bits, int64_t nwords, const uint32_t* __restrict__ off,
                           uint32_t* __restrict__ part_c, uint32_t* __restrict__ part_d) {
  const int lane = threadIdx.x & 31;
  const int64_t wbase = (int64_t)blockIdx.x * kCompTile + (int64_t)(threadIdx.x >> 5) * kWarpWords;
  uint32_t xs[kCompWords];
  warp_words(bits, nwords, wbase, xs);
  uint32_t c = 0, d = 0;
#pragma unroll
  for (int i = 0; i < kCompWords; i++) {
    if (xs[i]) word_count_deg(xs[i], (uint32_t)((wbase + i * 32 + lane) * 32), off, c, d);
  }
  __shared__ uint32_t tc, td;
  block_exclusive_sum<kCompThreads>(c, &tc);
  block_exclusive_sum<kCompThreads>(d, &td);
  if (threadIdx.x == 0) {
    part_c[blockIdx.x] = tc;
    part_d[blockIdx.x] = td;
  }
}

// Also writes (count, degsum) straight into the caller's mapped host words
// `host_info`, so a level's host sync needs no copy (none on a copy engine
// another stream may be using).
__global__ void comp_scan(uint32_t* part_c, uint32_t* part_d, int64_t nt, uint64_t* info,
                          uint32_t* qoff_total_slot_base, volatile uint64_t* host_info) {
  __shared__ uint32_t cc, cd, tc, td;
  if (threadIdx.x == 0) { cc = 0; cd = 0; }
  __syncthreads();
  for (int64_t base = 0; base < nt; base += kCompThreads) {
    int64_t i = base + threadIdx.x;
    uint32_t vc = i < nt ? part_c[i] : 0, vd = i < nt ? part_d[i] : 0;
    uint32_t ec = block_exclusive_sum<kCompThreads>(vc, &tc);
    uint32_t ed = block_exclusive_sum<kCompThreads>(vd, &td);
    uint32_t c0 = cc, d0 = cd;
    if (i < nt) { part_c[i] = c0 + ec; part_d[i] = d0 + ed; }
    __syncthreads();
    if (threadIdx.x == 0) { cc = c0 + tc; cd = d0 + td; }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    info[0] = cc;
    info[1] = cd;
    // qoff[count] = degsum: the slot sits right after the last queue entry
    if (qoff_total_slot_base) qoff_total_slot_base[cc] = cd;
    host_info[0] = cc;
    host_info[1] = cd;
    __threadfence_system();
  }
}

// Emission: the warp walks its non-zero words in order, one word per step
// with lane b on bit b, so the queue, qoff and depth stores of a word are
// consecutive (coalesced) and its degrees come from 33 consecutive offsets.
__global__ void comp_emit(const uint32_t* __restrict__ bits, int64_t nwords, const uint32_t* __restrict__ off,
                          const uint32_t* __restrict__ part_c, const uint32_t* __restrict__ part_d,
                          uint32_t* __restrict__ queue, uint32_t* __restrict__ qoff, int32_t* depth,
                          int32_t level, uint32_t* or_into) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t wbase = (int64_t)blockIdx.x * kCompTile + (int64_t)warp * kWarpWords;
  uint32_t xs[kCompWords];
  warp_words(bits, nwords, wbase, xs);
  uint32_t c = 0, d = 0;
#pragma unroll
  for (int i = 0; i < kCompWords; i++) {
    if (xs[i]) {
      const int64_t w = wbase + i * 32 + lane;
      word_count_deg(xs[i], (uint32_t)(w * 32), off, c, d);
      if (or_into) or_into[w] |= xs[i];
    }
  }
  // the warp's place in the block, after the block's place in the frontier
  __shared__ uint32_t wc[kCompWarps], wd[kCompWarps];
  c = __reduce_add_sync(0xffffffffu, c);
  d = __reduce_add_sync(0xffffffffu, d);
  if (lane == 0) {
    wc[warp] = c;
    wd[warp] = d;
  }
  __syncthreads();
  uint32_t pc = part_c[blockIdx.x], pd = part_d[blockIdx.x];
  for (int j = 0; j < warp; j++) {
    pc += wc[j];
    pd += wd[j];
  }
  const uint32_t below_mask = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < kCompWords; i++) {
    unsigned nz = __ballot_sync(0xffffffffu, xs[i] != 0u);
    while (nz) {
      const int j = __ffs(nz) - 1;
      nz &= nz - 1;
      const uint32_t x = __shfl_sync(0xffffffffu, xs[i], j);
      const uint32_t v = (uint32_t)((wbase + i * 32 + j) * 32) + (uint32_t)lane;
      const bool set = (x >> lane) & 1u;
      const uint32_t dg = set ? off[v + 1] - off[v] : 0u;
      uint32_t inc = dg;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (set) {
        const uint32_t at = pc + (uint32_t)__popc(x & below_mask);
        queue[at] = v;
        qoff[at] = pd + inc - dg;
        if (depth) depth[v] = level;
      }
      pc += (uint32_t)__popc(x);
      pd += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

rg_status compact_bits(const rg_graph* g, Frontier& f, cudaStream_t st, bool sync, int32_t* depth,
                       int32_t level, uint32_t* or_into, uint32_t* queue_out, uint32_t* qoff_out,
                       const uint32_t* deg_off) {
  Workspace& ws = ctx().ws;
  const uint32_t* doff = deg_off ? deg_off : g->off.as<uint32_t>();
  const int64_t nwords = (g->n + 31) / 32;
  const int64_t nt = (nwords + kCompTile - 1) / kCompTile;
  RG_TRY(ws.scan_partials.reserve(sizeof(uint32_t) * 2 * (nt + 1)));
  uint32_t* pc = ws.scan_partials.as<uint32_t>();
  uint32_t* pd = pc + nt + 1;
  uint32_t* q = queue_out ? queue_out : f.queue.as<uint32_t>();
  uint32_t* qo = qoff_out ? qoff_out : f.qoff.as<uint32_t>();
  uint64_t* info = ws.counters.as<uint64_t>();
  comp_count<<<(unsigned)nt, kCompThreads, 0, st>>>(f.bits.as<uint32_t>(), nwords, doff, pc, pd);
  comp_scan<<<1, kCompThreads, 0, st>>>(pc, pd, nt, info, qo, ws.h_info_dev);
  comp_emit<<<(unsigned)nt, kCompThreads, 0, st>>>(f.bits.as<uint32_t>(), nwords, doff, pc, pd, q, qo, depth,
                                                   level, or_into);
  RG_CUDA(cudaGetLastError());
  f.queue_valid = (queue_out == nullptr);
  f.bits_valid = true;
  if (sync) {
    RG_CUDA(cudaStreamSynchronize(st));
    f.count = (int64_t)ws.h_info[0];
    f.degsum = (int64_t)ws.h_info[1];
  }
  return RG_OK;
}

rg_status frontier_alloc(const rg_graph* g, Frontier& f) {
  const int64_t nwords = (g->n + 31) / 32;
  RG_TRY(f.queue.reserve(sizeof(uint32_t) * (g->n + 64)));
  RG_TRY(f.qoff.reserve(sizeof(uint32_t) * (g->n + 65)));
  RG_TRY(f.bits.reserve(sizeof(uint32_t) * (nwords + 8)));
  return RG_OK;
}

__global__ void set_bits_from_queue(const uint32_t* __restrict__ q, int64_t k, uint32_t* bits) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < k) atomicOr(bits + (q[i] >> 5), 1u << (q[i] & 31));
}

rg_status frontier_bits_from_queue(const rg_graph* g, Frontier& f, cudaStream_t st) {
  const int64_t nwords = (g->n + 31) / 32;
  RG_CUDA(cudaMemsetAsync(f.bits.p, 0, sizeof(uint32_t) * nwords, st));
  if (f.count > 0) {
    set_bits_from_queue<<<(unsigned)((f.count + 255) / 256), 256, 0, st>>>(f.queue.as<uint32_t>(), f.count,
                                                                          f.bits.as<uint32_t>());
  }
  RG_CUDA(cudaGetLastError());
  f.bits_valid = true;
  return RG_OK;
}

__global__ void lookup_kernel(const uint32_t* __restrict__ new_ids, const uint32_t* __restrict__ off,
                              const uint32_t* __restrict__ ids, int64_t k, uint32_t* __restrict__ out_id,
                              uint32_t* __restrict__ out_deg) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < k) {
    const uint32_t v = new_ids ? new_ids[ids[i]] : ids[i];
    out_id[i] = v;
    out_deg[i] = off[v + 1] - off[v];
  }
}

rg_status host_arrays(const rg_graph* g) {
  std::lock_guard<std::mutex> lk(g->host_mu);
  if (g->host_ready) return RG_OK;
  const int64_t n = g->n;
  HostU32 off(n + 1);
  RG_CUDA(cudaMemcpy(off.data(), g->off.p, 4 * (n + 1), cudaMemcpyDeviceToHost));
  g->h_deg.resize(n);
#pragma omp parallel for
  for (int64_t v = 0; v < n; v++) g->h_deg[v] = off[v + 1] - off[v];
  if (g->sorted) {
    g->h_new_ids.resize(n);
    RG_CUDA(cudaMemcpy(g->h_new_ids.data(), g->new_ids.p, 4 * n, cudaMemcpyDeviceToHost));
  }
  if (g->directed) {
    RG_CUDA(cudaMemcpy(off.data(), g->in_off.p, 4 * (n + 1), cudaMemcpyDeviceToHost));
    g->h_in_deg.resize(n);
#pragma omp parallel for
    for (int64_t v = 0; v < n; v++) g->h_in_deg[v] = off[v + 1] - off[v];
  }
  g->host_ready = true;
  return RG_OK;
}

rg_status lookup_ids(const rg_graph* g, const uint32_t* ids, int64_t k, bool orig, uint32_t* internal_out,
                     uint32_t* deg_out, bool in_degree) {
  in_degree = in_degree && g->directed;
  for (int64_t i = 0; i < k; i++) {
    if (ids[i] >= (uint64_t)g->n) return fail(RG_EINVAL, "vertex id %u >= n", ids[i]);
  }
  const bool map = orig && g->sorted;
  bool ready;
  {
    std::lock_guard<std::mutex> lk(g->host_mu);
    ready = g->host_ready;
  }
  if (ready || k > 4096) {
    RG_TRY(host_arrays(g));
    if ((in_degree ? g->h_in_deg : g->h_deg).size() != (size_t)g->n || (map && g->h_new_ids.size() != (size_t)g->n))
      return fail(RG_EUNSUPPORTED, "host degree arrays missing");
    for (int64_t i = 0; i < k; i++) {
      const uint32_t v = map ? g->h_new_ids[ids[i]] : ids[i];
      if (internal_out) internal_out[i] = v;
      if (deg_out) deg_out[i] = in_degree ? g->h_in_deg[v] : g->h_deg[v];
    }
    return RG_OK;
  }
  if (k == 0) return RG_OK;
  Ctx* cx = nullptr;
  RG_TRY(get_ctx(&cx));
  cudaStream_t st = cx->stream;
  RG_TRY(cx->ws.lookup.reserve(12 * (size_t)k));
  uint32_t* d = cx->ws.lookup.as<uint32_t>();
  std::vector<uint32_t> back(2 * k);
  RG_CUDA(cudaMemcpyAsync(d, ids, 4 * k, cudaMemcpyHostToDevice, st));
  lookup_kernel<<<(unsigned)((k + 255) / 256), 256, 0, st>>>(map ? g->new_ids.as<uint32_t>() : nullptr,
                                                             (in_degree ? g->in_off : g->off).as<uint32_t>(), d, k,
                                                             d + k, d + 2 * k);
  RG_CUDA(cudaGetLastError());
  RG_TRY(read_small(d + k, back.data(), 8 * (size_t)k, st));
  for (int64_t i = 0; i < k; i++) {
    if (internal_out) internal_out[i] = back[i];
    if (deg_out) deg_out[i] = back[k + i];
  }
  return RG_OK;
}

rg_status frontier_from_host(const rg_graph* g, Frontier& f, const uint32_t* ids, int64_t k,
                             cudaStream_t st) {
  RG_TRY(frontier_alloc(g, f));
  if (k > g->n + 64) return fail(RG_EINVAL, "frontier larger than n+64 entries");
  std::vector<uint32_t> qo(k + 1), deg(k);
  RG_TRY(lookup_ids(g, ids, k, false, nullptr, deg.data()));
  uint64_t acc = 0;
  for (int64_t i = 0; i < k; i++) {
    qo[i] = (uint32_t)acc;
    acc += deg[i];
  }
  qo[k] = (uint32_t)acc;
  if (k) RG_CUDA(cudaMemcpyAsync(f.queue.p, ids, 4 * k, cudaMemcpyHostToDevice, st));
  RG_CUDA(cudaMemcpyAsync(f.qoff.p, qo.data(), 4 * (k + 1), cudaMemcpyHostToDevice, st));
  f.count = k;
  f.degsum = (int64_t)acc;
  f.queue_valid = true;
  RG_TRY(frontier_bits_from_queue(g, f, st));
  // the host vector must outlive the async copy
  RG_CUDA(cudaStreamSynchronize(st));
  return RG_OK;
}

__global__ void fill_all_bits(uint32_t* bits, int64_t n) {
  int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t nwords = (n + 31) / 32;
  if (w < nwords) {
    int64_t rem = n - w * 32;
    bits[w] = rem >= 32 ? 0xffffffffu : ((1u << rem) - 1u);
  }
}

rg_status frontier_set_all(const rg_graph* g, Frontier& f, cudaStream_t st) {
  RG_TRY(frontier_alloc(g, f));
  const int64_t nwords = (g->n + 31) / 32;
  fill_all_bits<<<(unsigned)((nwords + 255) / 256), 256, 0, st>>>(f.bits.as<uint32_t>(), g->n);
  RG_CUDA(cudaGetLastError());
  f.bits_valid = true;
  return compact_bits(g, f, st, true);
}

// ---------------------------------------------------------------------------
// graph image
// ---------------------------------------------------------------------------

// chunk_v[c] = source vertex of edge min(c*kSweepChunk, m-1), c = 0..nchunks.
__global__ void build_chunk_starts(const uint32_t* __restrict__ off, uint32_t n, uint32_t m, int64_t nchunks,
                                   uint32_t* __restrict__ chunk_v) {
  int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c > nchunks) return;
  uint64_t e = (uint64_t)c * kSweepChunk;
  if (e >= m) e = m - 1;
  chunk_v[c] = upper_index(off, 0u, n - 1, (uint32_t)e);
}

static rg_status finish_graph(rg_graph* g) {
  cudaStream_t st = ctx().stream;
  if (g->m > 0) {
    g->nchunks = (g->m + kSweepChunk - 1) / kSweepChunk;
    RG_TRY(g->chunk_v.reserve(sizeof(uint32_t) * (g->nchunks + 1)));
    build_chunk_starts<<<(unsigned)((g->nchunks + 1 + 255) / 256), 256, 0, st>>>(
        g->off.as<uint32_t>(), (uint32_t)g->n, (uint32_t)g->m, g->nchunks, g->chunk_v.as<uint32_t>());
    RG_CUDA(cudaGetLastError());
    if (g->directed) {
      RG_TRY(g->in_chunk_v.reserve(sizeof(uint32_t) * (g->nchunks + 1)));
      build_chunk_starts<<<(unsigned)((g->nchunks + 1 + 255) / 256), 256, 0, st>>>(
          g->in_off.as<uint32_t>(), (uint32_t)g->n, (uint32_t)g->m, g->nchunks, g->in_chunk_v.as<uint32_t>());
      RG_CUDA(cudaGetLastError());
    }
  }
  RG_CUDA(cudaStreamSynchronize(st));
  return RG_OK;
}

static rg_status new_graph(rg_graph** out) {
  Ctx* c = nullptr;
  RG_TRY(get_ctx(&c));
  rg_graph* g = new (std::nothrow) rg_graph();
  if (!g) return fail(RG_ENOMEM, "host allocation failed");
  g->device = c->device;
  *out = g;
  return RG_OK;
}

}  // namespace rg

rg_graph::~rg_graph() {}

using namespace rg;

static rg_status graph_create_common(int64_t n, int64_t m, const uint32_t* off, const uint32_t* adj,
                                     cudaMemcpyKind kind, rg_graph** out) {
  if (!out || n <= 0 || m < 0 || !off || (m > 0 && !adj)) {
    return fail(RG_EINVAL, "rg_graph_create: bad arguments");
  }
  if (m >= 0xFFFFFFFFll || n >= 0xFFFFFFFFll) {
    return fail(RG_EUNSUPPORTED, "rg_graph_create: >= 2^32 edges or vertices");
  }
  HostU32 dev_off_copy;  // a host copy of the offsets only when they live on the device
  const uint32_t* h_off = off;
  if (kind != cudaMemcpyHostToDevice) {
    dev_off_copy.resize(n + 1);
    RG_CUDA(cudaMemcpy(dev_off_copy.data(), off, 4 * (n + 1), cudaMemcpyDeviceToHost));
    h_off = dev_off_copy.data();
  }
  if (h_off[0] != 0 || h_off[n] != (uint32_t)m) return fail(RG_EINVAL, "offsets must start at 0 and end at m");
  rg_graph* g = nullptr;
  RG_TRY(new_graph(&g));
  g->n = n;
  g->m = m;
  g->h_deg.resize(n);
  rg_status s;
  if ((s = g->off.reserve(4 * (n + 1))) != RG_OK || (s = g->adj.reserve(4 * (m + 8))) != RG_OK) {
    delete g;
    return s;
  }
  // host degrees and the monotonicity check run on a helper thread (all
  // cores) while this thread uploads the CSR
  int64_t bad_at = -1;
  uint32_t mx = 0;
  std::thread degrees([&] {
    int64_t bad = INT64_MAX;
    uint32_t m_loc = 0;
#pragma omp parallel for reduction(max : m_loc) reduction(min : bad)
    for (int64_t v = 0; v < n; v++) {
      if (h_off[v + 1] < h_off[v]) bad = std::min(bad, v);
      const uint32_t d = h_off[v + 1] - h_off[v];
      g->h_deg[v] = d;
      m_loc = std::max(m_loc, d);
    }
    mx = m_loc;
    bad_at = bad == INT64_MAX ? -1 : bad;
  });
  cudaStream_t st = ctx().stream;
  cudaError_t e = cudaMemcpyAsync(g->off.p, off, 4 * (n + 1), kind, st);
  if (e == cudaSuccess && m > 0) e = cudaMemcpyAsync(g->adj.p, adj, 4 * m, kind, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(g->adj.as<uint32_t>() + m, 0, 32, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  degrees.join();
  if (e != cudaSuccess) {
    delete g;
    return cuda_fail(e, "graph upload", __FILE__, __LINE__);
  }
  if (bad_at >= 0) {
    delete g;
    return fail(RG_EINVAL, "offsets not monotone at %lld", (long long)bad_at);
  }
  g->max_deg = mx;
  g->host_ready = true;  // an uploaded graph's host degrees are complete (it has no permutation)
  if ((s = finish_graph(g)) != RG_OK) { delete g; return s; }
  *out = g;
  return RG_OK;
}

extern "C" rg_status rg_graph_create(int64_t n, int64_t m, const uint32_t* h_off, const uint32_t* h_adj,
                                     rg_graph** out) {
  return graph_create_common(n, m, h_off, h_adj, cudaMemcpyHostToDevice, out);
}

extern "C" rg_status rg_graph_create_device(int64_t n, int64_t m, const uint32_t* d_off,
                                            const uint32_t* d_adj, rg_graph** out) {
  return graph_create_common(n, m, d_off, d_adj, cudaMemcpyDeviceToDevice, out);
}

namespace rg {
void drop_hub_cache(const rg_graph* g);
}

extern "C" rg_status rg_graph_free(rg_graph* g) {
  if (!g) return RG_OK;
  rg::drop_hub_cache(g);
  // no work may still read the graph when its pooled buffers go back
  // (cudaFree would synchronize the device the same way)
  cudaDeviceSynchronize();
  delete g;
  return RG_OK;
}

extern "C" rg_status rg_graph_info(const rg_graph* g, int64_t* n, int64_t* m, int* sorted) {
  if (!g) return fail(RG_EINVAL, "null graph");
  if (n) *n = g->n;
  if (m) *m = g->m;
  if (sorted) *sorted = g->sorted ? 1 : 0;
  return RG_OK;
}

extern "C" rg_status rg_graph_download(const rg_graph* g, uint32_t* h_off, uint32_t* h_adj, uint32_t* h_new_ids) {
  if (!g) return fail(RG_EINVAL, "null graph");
  if (h_off) RG_CUDA(cudaMemcpy(h_off, g->off.p, 4 * (g->n + 1), cudaMemcpyDeviceToHost));
  if (h_adj && g->m) RG_CUDA(cudaMemcpy(h_adj, g->adj.p, 4 * g->m, cudaMemcpyDeviceToHost));
  if (h_new_ids) {
    if (g->sorted) RG_CUDA(cudaMemcpy(h_new_ids, g->new_ids.p, 4 * g->n, cudaMemcpyDeviceToHost));
    else for (int64_t i = 0; i < g->n; i++) h_new_ids[i] = (uint32_t)i;
  }
  return RG_OK;
}

// ---------------------------------------------------------------------------
// degree sort
// ---------------------------------------------------------------------------
namespace rg {

// (~deg(id), id) with ids laid out in DESCENDING order.
__global__ void sort_init(const uint32_t* __restrict__ off, uint32_t n, uint64_t* __restrict__ key) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const uint32_t v = n - 1 - (uint32_t)i;
    key[i] = ((uint64_t)~(off[v + 1] - off[v]) << 32) | v;
  }
}

// failed: nonzero when the sort gave up, whose output then has holes (nothing is done)
__global__ void rank_to_ids(const uint64_t* __restrict__ sorted, const uint32_t* __restrict__ off, uint32_t n,
                            uint32_t* __restrict__ new_ids, uint32_t* __restrict__ new_deg,
                            const unsigned int* failed) {
  if (*failed) return;
  int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) {
    const uint32_t v = (uint32_t)sorted[r];
    new_ids[v] = (uint32_t)r;
    new_deg[r] = off[v + 1] - off[v];
  }
}

// Edge-balanced relabel: every warp owns kSweepChunk consecutive edges of the
// original CSR (16-byte loads), finds each edge's source from the chunk
// partition, and writes new_ids[neighbour] at the source's new position.
// The neighbour array may be pinned host memory read over the host link
// (rg_graph_create_sorted); it then has no padding, so the last partial
// group of four is read entry by entry.  failed: as for rank_to_ids (there are no
// new ids then).
__global__ void __launch_bounds__(256) relabel_sweep(DevGraph g, const uint32_t* __restrict__ chunk_v,
                                                     uint32_t nchunks, const uint32_t* __restrict__ new_ids,
                                                     const uint32_t* __restrict__ new_off,
                                                     uint32_t* __restrict__ new_adj, unsigned int* bad_id,
                                                     const unsigned int* failed) {
  if (*failed) return;
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t c = warp; c < nchunks; c += nwarps) {
    const uint32_t vlo = chunk_v[c], vhi = chunk_v[c + 1];
#pragma unroll
    for (int r = 0; r < kSweepChunk / 128; r++) {
      const uint32_t e = c * kSweepChunk + r * 128 + lane * 4;
      if (e >= g.m) continue;
      uint32_t dd[4];
      if (e + 4 <= g.m) {
        const uint4 d4 = __ldg(reinterpret_cast<const uint4*>(g.adj + e));
        dd[0] = d4.x;
        dd[1] = d4.y;
        dd[2] = d4.z;
        dd[3] = d4.w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) dd[i] = e + i < g.m ? __ldg(g.adj + e + i) : 0u;
      }
      uint32_t s = upper_index(g.off, vlo, vhi, e);
      uint32_t nxt = g.off[s + 1];
      uint32_t base = new_off[new_ids[s]] - g.off[s];  // modulo 2^32; base + e is the new slot
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t ee = e + i;
        if (ee >= g.m) break;
        if (ee >= nxt) {
          do { s++; nxt = g.off[s + 1]; } while (ee >= nxt);
          base = new_off[new_ids[s]] - g.off[s];
        }
        if (dd[i] < g.n) {
          new_adj[base + ee] = new_ids[dd[i]];
        } else {  // a neighbour id out of range: reported, never used as an index
          new_adj[base + ee] = 0u;
          atomicOr(bad_id, 1u);
        }
      }
    }
  }
}

}  // namespace rg

// in-degree of each rank's vertex (a directed graph's new in-lists)
__global__ void rank_in_deg(const uint64_t* __restrict__ sorted, const uint32_t* __restrict__ in_off, uint32_t n,
                            uint32_t* __restrict__ new_in_deg, const unsigned int* failed) {
  if (*failed) return;
  int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) {
    const uint32_t v = (uint32_t)sorted[r];
    new_in_deg[r] = in_off[v + 1] - in_off[v];
  }
}

// Degree sort (IO.h:728-903): ranks by out-degree, or for a directed graph by
// in-degree unless by_out (-preprocess 1 / 0, IO.h:739-750); both lists of a
// directed graph are relabelled, their order kept.
static rg_status degree_sort_impl(const rg_graph* g, bool by_out, rg_graph** out, uint32_t* h_new_ids) {
  if (!g || !out) return fail(RG_EINVAL, "rg_graph_degree_sort: null argument");
  const int64_t n = g->n, m = g->m;
  const bool by_in = g->directed && !by_out;
  Ctx* c = nullptr;
  RG_TRY(get_ctx(&c));
  cudaStream_t st = c->stream;
  Workspace& ws = c->ws;
  // temporaries from the stream-ordered pool, released in order on `st`
  DevBuf k0{true, st}, k1{true, st}, new_deg{true, st}, bad{true, st};
  RG_TRY(bad.reserve(16));
  RG_CUDA(cudaMemsetAsync(bad.p, 0, 8, st));
  unsigned int* failed = bad.as<unsigned int>() + 1;
  RG_TRY(k0.reserve(8 * n));
  RG_TRY(k1.reserve(8 * n));
  sort_init<<<(unsigned)((n + 255) / 256), 256, 0, st>>>((by_in ? g->in_off : g->off).as<uint32_t>(), (uint32_t)n,
                                                        k0.as<uint64_t>());
  // ~deg differs from 0xFFFFFFFF only in the low bits that max_deg spans
  // (in-degrees: all 32 bits, their maximum is not kept)
  int bits = 0;
  while (bits < 32 && (g->max_deg >> bits) != 0) bits++;
  if (by_in) bits = 32;
  uint64_t *order = k0.as<uint64_t>(), *other = k1.as<uint64_t>();
  SortScratch sort(st);
  if (bits > 0) {
    RG_TRY(sort_begin(sort, n, sort_passes(32, 32 + bits), st));
    RG_TRY(sort_count(sort, order, n, 32, 32 + bits, st));
    RG_TRY(sort_run(sort, &order, &other, n, 32, 32 + bits, st));
    RG_CUDA(cudaMemcpyAsync(failed, sort_failed(sort), 4, cudaMemcpyDeviceToDevice, st));
  }
  RG_CUDA(cudaGetLastError());
  rg_graph* ng = nullptr;
  RG_TRY(new_graph(&ng));
  ng->n = n;
  ng->m = m;
  rg_status s;
  if ((s = ng->off.reserve(4 * (n + 1))) != RG_OK || (s = ng->adj.reserve(4 * (m + 8))) != RG_OK ||
      (s = ng->new_ids.reserve(4 * n)) != RG_OK || (s = new_deg.reserve(4 * n)) != RG_OK) {
    delete ng;
    return s;
  }
  rank_to_ids<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(order, g->off.as<uint32_t>(), (uint32_t)n,
                                                          ng->new_ids.as<uint32_t>(), new_deg.as<uint32_t>(), failed);
  if ((s = scan_u32(ws, new_deg.as<uint32_t>(), ng->off.as<uint32_t>(), n, st)) != RG_OK) {
    delete ng;
    return s;
  }
  ng->directed = g->directed;
  if (g->directed) {  // in-lists: offsets from the ranks' in-degrees (new_deg is free again after the scan)
    if ((s = ng->in_off.reserve(4 * (n + 1))) != RG_OK || (s = ng->in_adj.reserve(4 * (m + 8))) != RG_OK) {
      delete ng;
      return s;
    }
    rank_in_deg<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(order, g->in_off.as<uint32_t>(), (uint32_t)n,
                                                            new_deg.as<uint32_t>(), failed);
    if ((s = scan_u32(ws, new_deg.as<uint32_t>(), ng->in_off.as<uint32_t>(), n, st)) != RG_OK) {
      delete ng;
      return s;
    }
  }
  if (m > 0) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device);
    const int64_t blocks = std::min<int64_t>((g->nchunks * 32 + 255) / 256, (int64_t)std::max(sms, 1) * 8);
    relabel_sweep<<<(unsigned)blocks, 256, 0, st>>>(g->view(), g->chunk_v.as<uint32_t>(), (uint32_t)g->nchunks,
                                                    ng->new_ids.as<uint32_t>(), ng->off.as<uint32_t>(),
                                                    ng->adj.as<uint32_t>(), bad.as<unsigned int>(), failed);
    if (g->directed) {
      relabel_sweep<<<(unsigned)blocks, 256, 0, st>>>(g->in_view(), g->in_chunks(), (uint32_t)g->nchunks,
                                                      ng->new_ids.as<uint32_t>(), ng->in_off.as<uint32_t>(),
                                                      ng->in_adj.as<uint32_t>(), bad.as<unsigned int>(), failed);
    }
  }
  cudaError_t e = cudaMemsetAsync(ng->adj.as<uint32_t>() + m, 0, 32, st);
  if (e == cudaSuccess && g->directed) e = cudaMemsetAsync(ng->in_adj.as<uint32_t>() + m, 0, 32, st);
  unsigned int h_bad[2] = {0, 0};
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h_bad, bad.p, 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    delete ng;
    return cuda_fail(e, "degree sort", __FILE__, __LINE__);
  }
  if (h_bad[1]) {
    delete ng;
    return fail(RG_ECUDA, "rg_graph_degree_sort: the sort did not finish");
  }
  if (h_bad[0]) {
    delete ng;
    return fail(RG_EINVAL, "rg_graph_degree_sort: a neighbour id is >= n");
  }
  ng->sorted = true;
  ng->max_deg = g->max_deg;  // host arrays: on first full use (host_arrays)
  if (h_new_ids) {
    e = cudaMemcpy(h_new_ids, ng->new_ids.p, 4 * n, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) { delete ng; return cuda_fail(e, "new_ids download", __FILE__, __LINE__); }
  }
  if ((s = finish_graph(ng)) != RG_OK) { delete ng; return s; }
  *out = ng;
  return RG_OK;
}

extern "C" rg_status rg_graph_degree_sort(const rg_graph* g, rg_graph** out, uint32_t* h_new_ids) {
  return degree_sort_impl(g, false, out, h_new_ids);
}

extern "C" rg_status rg_graph_degree_sort_by(const rg_graph* g, int by_out_degree, rg_graph** out,
                                             uint32_t* h_new_ids) {
  return degree_sort_impl(g, by_out_degree != 0, out, h_new_ids);
}

// ---------------------------------------------------------------------------
// CSR construction on the device (the symmetric loader's clean-up, IO.h:429-474,
// for an edge list): both directions of every edge become 64-bit entries
// a << bits | b (ids < 2^bits), a radix sort orders them by (a, b), self loops and
// repeats are dropped while the survivors are written to the neighbour array, and each
// vertex's offset is the place of its first entry; large inputs sort every edge once
// with a < b and then the survivors by b.  The result is bit-identical to
// rg_csr_from_edges.
// ---------------------------------------------------------------------------
namespace rg {

// Entries from an edge list, their digit counts (passes of the sort on `hi`
// bits) and the largest id: the edge as it is, both ways round, or with its smaller
// end first and, in hist2, the digits of its larger end counted for the sort by that
// alone.  src and dst may be page-locked host memory, read once over the host link
// (which bounds it: 268 MB in 1.3 ms).  kWide: both are 16-byte aligned.
enum PackMode { kPackEdge, kPackBoth, kPackSmaller };

template <bool kWide, PackMode mode>
__global__ void __launch_bounds__(256) csr_pack(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst,
                                                int64_t ne, int bits, uint64_t* __restrict__ key, int hi,
                                                int passes, uint32_t* hist, uint32_t* hist2, unsigned int* max_id) {
  __shared__ uint32_t sh[kMaxSortPasses * 256], sh2[mode == kPackSmaller ? kMaxSortPasses / 2 * 256 : 1];
  const int passes2 = mode == kPackSmaller ? sort_passes(0, bits) : 0;
  sort_zero(sh, passes);
  if (mode == kPackSmaller) sort_zero(sh2, passes2);
  unsigned int mx = 0;
  auto one = [&](int64_t i, uint32_t a, uint32_t b) {
    mx = max(mx, max(a, b));
    const bool swap = mode == kPackSmaller && b < a;
    const uint64_t k = ((uint64_t)(swap ? b : a) << bits) | (swap ? a : b);
    key[i] = k;
    sort_count_key(sh, k, 0, hi, passes);
    if (mode == kPackSmaller) sort_count_key(sh2, k, 0, bits, passes2);
    if (mode == kPackBoth) {
      const uint64_t k1 = ((uint64_t)b << bits) | a;
      key[ne + i] = k1;
      sort_count_key(sh, k1, 0, hi, passes);
    }
  };
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
  if (kWide) {
    for (int64_t q = t; q * 4 < ne; q += nt) {
      if (q * 4 + 4 <= ne) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(src) + q), b = __ldg(reinterpret_cast<const uint4*>(dst) + q);
        one(q * 4, a.x, b.x);
        one(q * 4 + 1, a.y, b.y);
        one(q * 4 + 2, a.z, b.z);
        one(q * 4 + 3, a.w, b.w);
      } else {
        for (int64_t i = q * 4; i < ne; i++) one(i, src[i], dst[i]);
      }
    }
  } else {
    for (int64_t i = t; i < ne; i += nt) one(i, src[i], dst[i]);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) atomicMax(max_id, mx);
  sort_flush(sh, hist, passes);
  if (mode == kPackSmaller) sort_flush(sh2, hist2, passes2);
}

// Sorted entries -> neighbour array and offsets.  kClean drops self loops and
// repeats (the first of equal entries stays): csr_count gives the kept entries of
// each tile, and csr_emit, from their scan (whose last word is their total), writes
// them and the offsets.
constexpr int kCsrThreads = 256, kCsrItems = 8, kCsrTile = kCsrThreads * kCsrItems;

static int csr_sms() {
  int sms = 0;
  return cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx().device) == cudaSuccess ? sms : 1;
}

template <bool kClean>
__device__ __forceinline__ bool csr_keep(uint64_t x, uint64_t prev, bool has_prev, int bits) {
  const uint64_t mask = (1ull << bits) - 1;
  return !kClean || ((x >> bits) != (x & mask) && (!has_prev || x != prev));
}

__global__ void __launch_bounds__(kCsrThreads) csr_count(const uint64_t* __restrict__ key, int64_t k, int bits,
                                                         uint32_t* __restrict__ tile_count) {
  const int64_t t0 = (int64_t)blockIdx.x * kCsrTile;
  uint32_t c = 0;
#pragma unroll 4
  for (int s = 0; s < kCsrItems; s++) {
    const int64_t i = t0 + s * kCsrThreads + threadIdx.x;
    if (i < k) c += csr_keep<true>(key[i], i ? key[i - 1] : 0ull, i > 0, bits);
  }
  __shared__ uint32_t tot;
  block_exclusive_sum<kCsrThreads>(c, &tot);
  if (threadIdx.x == 0) tile_count[blockIdx.x] = tot;
}

// The same for long inputs; hist holds the digit counts of the values, and those of
// dropped entries are taken out.
__global__ void __launch_bounds__(kCsrThreads) csr_count_digits(const uint64_t* __restrict__ key, int64_t k, int bits,
                                                         uint32_t* __restrict__ tile_count, uint32_t* hist) {
  __shared__ uint32_t sh[kMaxSortPasses / 2 * 256];
  const int passes = sort_passes(0, bits);
  sort_zero(sh, passes);
  // a warp takes a tile; dropped entries are collected until they fill a warp (one
  // here and there would have every step wait for its three counts)
  __shared__ uint32_t dropped[kCsrThreads / 32][64];
  const int lane = threadIdx.x & 31;
  uint32_t* mine = dropped[threadIdx.x >> 5];
  int nd = 0;
  const int64_t tiles = (k + kCsrTile - 1) / kCsrTile, nwarps = (int64_t)gridDim.x * (kCsrThreads / 32);
  for (int64_t t = (int64_t)blockIdx.x * (kCsrThreads / 32) + (threadIdx.x >> 5); t < tiles; t += nwarps) {
    const int64_t t0 = t * kCsrTile;
    uint32_t c = 0;
    uint64_t before = lane == 0 && t0 > 0 ? key[t0 - 1] : 0ull;
    for (int s0 = 0; s0 < kCsrTile / 32; s0 += kCsrItems) {
      uint64_t x[kCsrItems];
#pragma unroll
      for (int s = 0; s < kCsrItems; s++) {
        const int64_t i = t0 + (s0 + s) * 32 + lane;
        x[s] = i < k ? key[i] : 0ull;
      }
#pragma unroll
      for (int s = 0; s < kCsrItems; s++) {
        const int64_t i = t0 + (s0 + s) * 32 + lane;
        const uint64_t up = __shfl_up_sync(0xffffffffu, x[s], 1);
        const bool keep = i < k && csr_keep<true>(x[s], lane ? up : before, i > 0, bits);
        before = __shfl_sync(0xffffffffu, x[s], 31);
        c += keep;
        const unsigned drop = __ballot_sync(0xffffffffu, i < k && !keep);
        if (!drop) continue;
        if ((drop >> lane) & 1u) mine[nd + __popc(drop & ((1u << lane) - 1u))] = (uint32_t)(x[s] & ((1ull << bits) - 1));
        nd += __popc(drop);
        if (nd >= 32) {
          nd -= 32;
          __syncwarp();
          sort_count_key(sh, mine[nd + lane], 0, bits, passes);
          __syncwarp();
        }
      }
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) tile_count[t] = c;
  }
  __syncwarp();
  if (lane < nd) sort_count_key(sh, mine[lane], 0, bits, passes);
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += kCsrThreads) {
    if (sh[i]) atomicSub(hist + i, sh[i]);
  }
}

// What csr_emit makes of the kept entries (row, value), the i-th of them at `pos`.
// Alone: adj[pos] = value and the rows' offsets.  The lists of a symmetric graph come
// from two sorts of half the entries each: those to larger ids (kUpper: their offsets,
// and the entries the other way round) and, from the sort of these, those to smaller
// ids (kLower); row v is its smaller neighbours
// and then its larger ones, so a half's entry lies at pos + the other half's entries
// before it (kLower writes its own, kPlace the larger ones when both offsets are
// there).
enum CsrPart { kAlone, kUpper, kLower, kPlace };

struct CsrOut {
  uint32_t* off;          // kAlone, kUpper, kLower: the rows' offsets, n + 1
  uint32_t* adj;          // not kUpper
  const uint32_t* other;  // kLower: the offsets of kUpper; kPlace: those of kLower
  uint64_t* back;         // kUpper: value << bits | row
  const uint32_t* failed;  // kLower, kPlace: the second sort's flag, which the host has not seen yet (its output,
                           // and the offsets made of it, are no indices then)
};

template <bool kClean, CsrPart kPart>
__global__ void __launch_bounds__(kCsrThreads) csr_emit(const uint64_t* __restrict__ key, int64_t k, int bits,
                                                        const uint32_t* __restrict__ tile_first, uint32_t n,
                                                        CsrOut out) {
  if ((kPart == kLower || kPart == kPlace) && *out.failed) return;
  // a warp's sub-tile of kCsrItems x 32 entries, 32 at a time: writes stay coalesced
  __shared__ uint32_t wsum[kCsrThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const int64_t tiles = (k + kCsrTile - 1) / kCsrTile;
  const uint64_t mask = (1ull << bits) - 1;
  {
    const int64_t tile = blockIdx.x, t0 = tile * kCsrTile + (int64_t)w * kCsrItems * 32;
    uint64_t x[kCsrItems];
    uint64_t before = 0;  // the entry before the sub-tile
    if (lane == 0 && t0 > 0 && t0 <= k) before = key[t0 - 1];
#pragma unroll
    for (int s = 0; s < kCsrItems; s++) {
      const int64_t i = t0 + s * 32 + lane;
      x[s] = i < k ? key[i] : 0ull;
    }
    uint32_t at = 0;
    if (kClean) {
      uint32_t c = 0;
      uint64_t b = before;
#pragma unroll
      for (int s = 0; s < kCsrItems; s++) {
        const int64_t i = t0 + s * 32 + lane;
        const uint64_t up = __shfl_up_sync(0xffffffffu, x[s], 1);
        c += __popc(__ballot_sync(0xffffffffu, i < k && csr_keep<true>(x[s], lane ? up : b, i > 0, bits)));
        b = __shfl_sync(0xffffffffu, x[s], 31);
      }
      __syncthreads();
      if (lane == 0) wsum[w] = c;
      __syncthreads();
      at = tile_first[tile];
      for (int j = 0; j < w; j++) at += wsum[j];
    } else {
      at = (uint32_t)min(t0, k);
    }
#pragma unroll
    for (int s = 0; s < kCsrItems; s++) {
      const int64_t i = t0 + s * 32 + lane;
      const uint64_t up = __shfl_up_sync(0xffffffffu, x[s], 1);
      const uint64_t prev = lane ? up : before;
      before = __shfl_sync(0xffffffffu, x[s], 31);
      const bool in = i < k;
      const bool keep = in && csr_keep<kClean>(x[s], prev, i > 0, bits);
      const unsigned kept = __ballot_sync(0xffffffffu, keep);
      const uint32_t pos = at + __popc(kept & lt);
      at += __popc(kept);
      const uint32_t row = (uint32_t)(x[s] >> bits), value = (uint32_t)(x[s] & mask);
      if (keep) {
        if (kPart == kAlone) out.adj[pos] = value;
        if (kPart == kLower || kPart == kPlace) out.adj[pos + out.other[row + (kPart == kPlace)]] = value;
        if (kPart == kUpper) out.back[pos] = ((uint64_t)value << bits) | row;
      }
      if (kPart == kPlace) continue;
      // offsets of the rows that begin at this entry: its own and the empty ones
      // before it; runs of more than a few by the whole warp
      const uint32_t from = i > 0 ? (uint32_t)(prev >> bits) + 1 : 0;
      uint32_t many = 0;  // rows
      if (in && row < n && from <= row) {  // (ids are < n)
        many = row - from + 1;
        if (many < 8) {
          for (uint32_t v = from; v <= row; v++) out.off[v] = pos;
          many = 0;
        }
      }
      for (unsigned runs = __ballot_sync(0xffffffffu, many > 0); runs; runs &= runs - 1) {
        const int j = __ffs(runs) - 1;
        const uint32_t f = __shfl_sync(0xffffffffu, from, j), c = __shfl_sync(0xffffffffu, many, j);
        const uint32_t p = __shfl_sync(0xffffffffu, pos, j);
        for (uint32_t v = lane; v < c; v += 32) out.off[f + v] = p;
      }
    }
  }
  // rows past the last entry's
  if (kPart != kPlace) {
    const uint64_t last = min(key[k - 1] >> bits, (uint64_t)n);
    const uint32_t end = kClean ? tile_first[tiles] : (uint32_t)k;
    for (uint64_t v = last + 1 + (uint64_t)blockIdx.x * kCsrThreads + threadIdx.x; v <= n;
         v += (uint64_t)gridDim.x * kCsrThreads) {
      out.off[v] = end;
    }
  }
}

template <bool kClean, CsrPart kPart>
static rg_status csr_emit_run(const uint64_t* key, int64_t k, int bits, const uint32_t* first, int64_t n,
                              const CsrOut& out, cudaStream_t st) {
  const int64_t tiles = (k + kCsrTile - 1) / kCsrTile;
  csr_emit<kClean, kPart><<<(unsigned)tiles, kCsrThreads, 0, st>>>(key, k, bits, first, (uint32_t)n, out);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

// How many of the sorted entries stay (*kept) and where each tile's begin (`first`,
// their scan).  One host sync, which also reads the sort's failure flag and, unless
// null, the largest id.
template <bool kClean>
static rg_status csr_kept(Workspace& ws, const uint64_t* key, int64_t k, int bits, int64_t n, DevBuf& first,
                          int64_t* kept, uint32_t* hist, const uint32_t* failed, const unsigned int* max_id,
                          const char* who, cudaStream_t st) {
  const int64_t tiles = (k + kCsrTile - 1) / kCsrTile;
  DevBuf back(true, st);
  RG_TRY(first.reserve(4 * (size_t)(tiles + 1)));
  RG_TRY(back.reserve(16));
  if (kClean) {
    if (hist) {  // (digit counts are flushed once per CTA: as many as run at once)
      const int64_t blocks = std::min<int64_t>((tiles * 32 + kCsrThreads - 1) / kCsrThreads, (int64_t)csr_sms() * 8);
      csr_count_digits<<<(unsigned)blocks, kCsrThreads, 0, st>>>(key, k, bits, first.as<uint32_t>(), hist);
    } else {
      csr_count<<<(unsigned)tiles, kCsrThreads, 0, st>>>(key, k, bits, first.as<uint32_t>());
    }
    RG_TRY(scan_u32(ws, first.as<uint32_t>(), first.as<uint32_t>(), tiles, st));
  }
  uint32_t h[3] = {0, 0, 0};  // entries, sort failure, largest id
  uint32_t* b = back.as<uint32_t>();
  RG_CUDA(cudaMemcpyAsync(b, first.as<uint32_t>() + tiles, 4, cudaMemcpyDeviceToDevice, st));
  RG_CUDA(cudaMemcpyAsync(b + 1, failed, 4, cudaMemcpyDeviceToDevice, st));
  if (max_id) RG_CUDA(cudaMemcpyAsync(b + 2, max_id, 4, cudaMemcpyDeviceToDevice, st));
  RG_TRY(read_small(b, h, max_id ? 12 : 8, st));
  if (max_id && h[2] >= (uint64_t)n) return fail(RG_EINVAL, "edge endpoint %u >= n", h[2]);
  if (h[1]) return fail(RG_ECUDA, "%s: the sort did not finish", who);
  *kept = kClean ? (int64_t)h[0] : k;
  return RG_OK;
}

// off and adj, sized here, of the sorted entries; *m_out entries survive.
template <bool kClean>
static rg_status csr_from_sorted(Workspace& ws, const uint64_t* key, int64_t k, int bits, int64_t n, DevBuf& off,
                                 DevBuf& adj, int64_t* m_out, const uint32_t* failed, const unsigned int* max_id,
                                 const char* who, cudaStream_t st) {
  DevBuf first(true, st);
  RG_TRY(csr_kept<kClean>(ws, key, k, bits, n, first, m_out, nullptr, failed, max_id, who, st));
  RG_TRY(off.reserve(4 * (size_t)(n + 1)));
  RG_TRY(adj.reserve(4 * (size_t)(*m_out + 8)));
  const CsrOut out{off.as<uint32_t>(), adj.as<uint32_t>(), nullptr, nullptr, nullptr};
  RG_TRY((csr_emit_run<kClean, kAlone>(key, k, bits, first.as<uint32_t>(), n, out, st)));
  RG_CUDA(cudaMemsetAsync(adj.as<uint32_t>() + *m_out, 0, 32, st));
  return RG_OK;
}

__global__ void add_offsets(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, int64_t n, uint32_t* off) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += (int64_t)gridDim.x * blockDim.x) {
    off[v] = a[v] + b[v];
  }
}

// The lists of a symmetric graph from its edges, each once with the smaller end as
// row, sorted with repeats in `key` (k entries; `other` holds as many); `sort`: begun
// for them by the larger end, whose digits it has counted.  Sorting the
// edges by both ends and then the kept ones by the larger end alone is three quarters
// of sorting every entry by both: 6.7e7 entries, with the clean-up, in 2.0 ms, 2.5 as
// entries.
static rg_status csr_from_edges_sorted(Workspace& ws, const uint64_t* key, uint64_t* other, int64_t k, int bits,
                                       int64_t n, SortScratch& sort, DevBuf& off, DevBuf& adj, int64_t* m_out,
                                       const uint32_t* failed, const unsigned int* max_id, const char* who,
                                       cudaStream_t st) {
  DevBuf first(true, st), upper(true, st), lower(true, st), back(true, st);
  int64_t kept = 0;
  RG_TRY(csr_kept<true>(ws, key, k, bits, n, first, &kept, sort_counts(sort), failed, max_id, who, st));
  *m_out = 2 * kept;
  RG_TRY(off.reserve(4 * (size_t)(n + 1)));
  RG_TRY(adj.reserve(4 * (size_t)(*m_out + 8)));
  RG_TRY(upper.reserve(4 * (size_t)(n + 1)));
  RG_TRY(lower.reserve(4 * (size_t)(n + 1)));
  RG_TRY(back.reserve(8 * (size_t)std::max<int64_t>(kept, 1)));
  CsrOut out{upper.as<uint32_t>(), nullptr, nullptr, back.as<uint64_t>(), nullptr};
  RG_TRY((csr_emit_run<true, kUpper>(key, k, bits, first.as<uint32_t>(), n, out, st)));
  uint32_t gave_up = 0;
  if (kept > 0) {
    uint64_t *a = back.as<uint64_t>(), *b = other;
    RG_TRY(sort_run(sort, &a, &b, kept, bits, 2 * bits, st));
    out = CsrOut{lower.as<uint32_t>(), adj.as<uint32_t>(), upper.as<uint32_t>(), nullptr, sort_failed(sort)};
    RG_TRY((csr_emit_run<false, kLower>(a, kept, bits, nullptr, n, out, st)));
    out = CsrOut{nullptr, adj.as<uint32_t>(), lower.as<uint32_t>(), nullptr, sort_failed(sort)};
    RG_TRY((csr_emit_run<true, kPlace>(key, k, bits, first.as<uint32_t>(), n, out, st)));
  } else {
    RG_CUDA(cudaMemsetAsync(lower.p, 0, 4 * (size_t)(n + 1), st));
  }
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + 256) / 256, (int64_t)csr_sms() * 16));
  add_offsets<<<blocks, 256, 0, st>>>(upper.as<uint32_t>(), lower.as<uint32_t>(), n, off.as<uint32_t>());
  RG_CUDA(cudaGetLastError());
  RG_CUDA(cudaMemsetAsync(adj.as<uint32_t>() + *m_out, 0, 32, st));
  if (kept > 0) RG_TRY(read_small(sort_failed(sort), &gave_up, 4, st));
  return gave_up ? fail(RG_ECUDA, "%s: the sort did not finish", who) : RG_OK;
}

rg_status csr_from_sorted_rows(Workspace& ws, const uint64_t* key, int64_t k, int bits, int64_t n, bool clean,
                               DevBuf& off, DevBuf& adj, int64_t* kept, const SortScratch& sort, const char* who,
                               cudaStream_t st) {
  auto fn = clean ? csr_from_sorted<true> : csr_from_sorted<false>;
  return fn(ws, key, k, bits, n, off, adj, kept, sort_failed(sort), nullptr, who, st);
}

__global__ void max_degree(const uint32_t* __restrict__ off, int64_t n, unsigned int* out) {
  unsigned int mx = 0;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    mx = max(mx, off[v + 1] - off[v]);
  }
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, mx);
}

}  // namespace rg

namespace rg {
rg_status build_in_lists(rg_graph* g, cudaStream_t st);
}

// Shared by the symmetric and directed builders.  Directed: the entries are the
// edges as they are, and the in-lists are built afterwards; symmetric: both directions
// of every edge or, from kHalvesFrom edges on, each edge once (csr_from_edges_sorted):
// that sorts a quarter less in more launches.  from_edges, us, halves against both:
// 1e4 edges 235 / 147, 1e6 340 / 250, 3e6 560 / 485, 1e7 1240 / 1245, 3e7 3200 / 3550.
constexpr int64_t kHalvesFrom = 12 << 20;

static rg_status create_from_edges(const char* who, int64_t n, int64_t num_edges, const uint32_t* src,
                                   const uint32_t* dst, int on_device, bool directed, rg_graph** out) {
  if (!out || n <= 0 || num_edges < 0 || (num_edges > 0 && (!src || !dst))) {
    return fail(RG_EINVAL, "%s: bad arguments", who);
  }
  if (n >= 0xFFFFFFFFll || (directed ? num_edges : 2 * num_edges) >= 0xFFFFFFFFll) {
    return fail(RG_EUNSUPPORTED, "%s: >= 2^32 vertices or directed entries", who);
  }
  const PackMode mode = directed ? kPackEdge : num_edges >= kHalvesFrom ? kPackSmaller : kPackBoth;
  const int64_t k = mode == kPackBoth ? 2 * num_edges : num_edges;
  Ctx* c = nullptr;
  RG_TRY(get_ctx(&c));
  cudaStream_t st = c->stream;
  int sms = 0;
  RG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  int bits = 1;
  while (bits < 32 && ((uint64_t)(n - 1) >> bits) != 0) bits++;
  rg_graph* g = nullptr;
  RG_TRY(new_graph(&g));
  g->n = n;
  rg_status s = RG_OK;
  uint32_t mx = 0;
  {
    // temporaries from the pool
    DevBuf k0{true, st}, k1{true, st}, info{true, st};
    SortScratch sort(st), by_end(st);
    const int hi = 2 * bits, passes = sort_passes(0, hi);
    auto fill = [&]() -> rg_status {
      RG_TRY(info.reserve(8));
      RG_CUDA(cudaMemsetAsync(info.p, 0, 8, st));
      if (k == 0) {
        RG_TRY(g->off.reserve(4 * (n + 1)));
        RG_TRY(g->adj.reserve(32));
        RG_CUDA(cudaMemsetAsync(g->off.p, 0, 4 * (n + 1), st));
        RG_CUDA(cudaMemsetAsync(g->adj.p, 0, 32, st));
        return RG_OK;
      }
      RG_TRY(k0.reserve(8 * (size_t)k));
      RG_TRY(k1.reserve(8 * (size_t)k + 16));
      RG_TRY(sort_begin(sort, k, passes, st));
      if (mode == kPackSmaller) RG_TRY(sort_begin(by_end, k, sort_passes(bits, hi), st));
      const uint32_t *d_src = src, *d_dst = dst;
      if (!on_device) {
        d_src = static_cast<const uint32_t*>(device_alias(src, 4 * num_edges, 4));
        d_dst = static_cast<const uint32_t*>(device_alias(dst, 4 * num_edges, 4));
      }
      if (!d_src || !d_dst) {
        // pageable: copied (into the sort's second buffer, free until its first pass)
        uint32_t* c2 = k1.as<uint32_t>();
        RG_CUDA(cudaMemcpyAsync(c2, src, 4 * num_edges, cudaMemcpyHostToDevice, st));
        RG_CUDA(cudaMemcpyAsync(c2 + ((num_edges + 3) & ~3ll), dst, 4 * num_edges, cudaMemcpyHostToDevice, st));
        d_src = c2;
        d_dst = c2 + ((num_edges + 3) & ~3ll);
      }
      const bool wide = (((uintptr_t)d_src | (uintptr_t)d_dst) & 15u) == 0;
      const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((num_edges + 1023) / 1024, (int64_t)sms * 8));
      auto pack = mode == kPackEdge   ? (wide ? csr_pack<true, kPackEdge> : csr_pack<false, kPackEdge>)
                  : mode == kPackBoth ? (wide ? csr_pack<true, kPackBoth> : csr_pack<false, kPackBoth>)
                                      : (wide ? csr_pack<true, kPackSmaller> : csr_pack<false, kPackSmaller>);
      pack<<<(unsigned)blocks, 256, 0, st>>>(d_src, d_dst, num_edges, bits, k0.as<uint64_t>(), hi, passes,
                                             sort_counts(sort), mode == kPackSmaller ? sort_counts(by_end) : nullptr,
                                             info.as<unsigned int>());
      RG_CUDA(cudaGetLastError());
      uint64_t *key = k0.as<uint64_t>(), *other = k1.as<uint64_t>();
      RG_TRY(sort_run(sort, &key, &other, k, 0, hi, st));
      if (mode != kPackSmaller) {
        return csr_from_sorted<true>(c->ws, key, k, bits, n, g->off, g->adj, &g->m, sort_failed(sort),
                                     info.as<unsigned int>(), who, st);
      }
      return csr_from_edges_sorted(c->ws, key, other, k, bits, n, by_end, g->off, g->adj, &g->m, sort_failed(sort),
                                   info.as<unsigned int>(), who, st);
    };
    s = fill();
    if (s == RG_OK) {
      const int dblocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)sms * 16));
      max_degree<<<dblocks, 256, 0, st>>>(g->off.as<uint32_t>(), n, info.as<unsigned int>() + 1);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) s = cuda_fail(e, "device CSR build", __FILE__, __LINE__);
      else s = read_small(info.as<unsigned int>() + 1, &mx, 4, st);
    }
  }
  if (s != RG_OK) {
    delete g;
    return s;
  }
  g->max_deg = mx;  // host degree array: on first full use (host_arrays)
  if ((s = finish_graph(g)) != RG_OK) { delete g; return s; }
  if (directed) {
    g->directed = true;
    s = build_in_lists(g, st);          // uses the out-list partition
    if (s == RG_OK) s = finish_graph(g);  // partitions of both lists
    if (s != RG_OK) {
      rg_graph_free(g);
      return s;
    }
  }
  *out = g;
  return RG_OK;
}

extern "C" rg_status rg_graph_create_from_edges(int64_t n, int64_t num_edges, const uint32_t* src, const uint32_t* dst,
                                                int on_device, rg_graph** out) {
  return create_from_edges("rg_graph_create_from_edges", n, num_edges, src, dst, on_device, false, out);
}

extern "C" rg_status rg_graph_create_directed_from_edges(int64_t n, int64_t num_edges, const uint32_t* src,
                                                         const uint32_t* dst, int on_device, rg_graph** out) {
  return create_from_edges("rg_graph_create_directed_from_edges", n, num_edges, src, dst, on_device, true, out);
}

// ---------------------------------------------------------------------------
// directed graphs: the in-lists (the reference's CSC, IO.h:287-345) built on
// the device.  The out-list entries are already ordered by source, so one
// stable radix sort by target leaves every in-list's sources ascending.
// ---------------------------------------------------------------------------
namespace rg {

// Entries target << bits | source in list order, and their digit counts.
__global__ void __launch_bounds__(256) in_entries(DevGraph g, const uint32_t* __restrict__ chunk_v, uint32_t nchunks,
                                                  int bits, uint64_t* __restrict__ key, int passes, uint32_t* hist) {
  __shared__ uint32_t sh[kMaxSortPasses * 256];
  sort_zero(sh, passes);
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t c = warp; c < nchunks; c += nwarps) {
    const uint32_t vlo = chunk_v[c], vhi = chunk_v[c + 1];
    for (int r = 0; r < kSweepChunk / 32; r++) {
      const uint32_t e = c * kSweepChunk + r * 32 + lane;
      if (e >= g.m) break;
      const uint64_t k = ((uint64_t)g.adj[e] << bits) | upper_index(g.off, vlo, vhi, e);
      key[e] = k;
      sort_count_key(sh, k, bits, 2 * bits, passes);
    }
  }
  sort_flush(sh, hist, passes);
}

rg_status build_in_lists(rg_graph* g, cudaStream_t st) {
  const int64_t n = g->n, m = g->m;
  if (m == 0) {
    RG_TRY(g->in_off.reserve(4 * (n + 1)));
    RG_TRY(g->in_adj.reserve(32));
    RG_CUDA(cudaMemsetAsync(g->in_off.p, 0, 4 * (n + 1), st));
    RG_CUDA(cudaMemsetAsync(g->in_adj.p, 0, 32, st));
    return RG_OK;
  }
  int sms = 0;
  RG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device));
  int bits = 1;
  while (bits < 32 && ((uint64_t)(n - 1) >> bits) != 0) bits++;
  const int passes = sort_passes(bits, 2 * bits);
  DevBuf k0{true, st}, k1{true, st};
  SortScratch sort(st);
  RG_TRY(k0.reserve(8 * (size_t)m));
  RG_TRY(k1.reserve(8 * (size_t)m));
  RG_TRY(sort_begin(sort, m, passes, st));
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((g->nchunks * 32 + 255) / 256, (int64_t)sms * 8));
  in_entries<<<(unsigned)blocks, 256, 0, st>>>(g->view(), g->chunk_v.as<uint32_t>(), (uint32_t)g->nchunks, bits,
                                               k0.as<uint64_t>(), passes, sort_counts(sort));
  RG_CUDA(cudaGetLastError());
  uint64_t *key = k0.as<uint64_t>(), *other = k1.as<uint64_t>();
  RG_TRY(sort_run(sort, &key, &other, m, bits, 2 * bits, st));
  int64_t kept = 0;
  RG_TRY(csr_from_sorted_rows(ctx().ws, key, m, bits, n, false, g->in_off, g->in_adj, &kept, sort, "in-lists", st));
  RG_CUDA(cudaStreamSynchronize(st));
  return RG_OK;
}

}  // namespace rg

extern "C" rg_status rg_graph_create_directed(int64_t n, int64_t m, const uint32_t* h_off, const uint32_t* h_adj,
                                              rg_graph** out) {
  rg_graph* g = nullptr;
  RG_TRY(rg_graph_create(n, m, h_off, h_adj, &g));
  g->directed = true;
  g->host_ready = false;  // host in-degrees come with the in-lists (host_arrays)
  rg_status s = build_in_lists(g, ctx().stream);
  if (s == RG_OK) s = finish_graph(g);  // partitions of both lists
  if (s != RG_OK) {
    rg_graph_free(g);
    return s;
  }
  *out = g;
  return RG_OK;
}

extern "C" rg_status rg_graph_is_directed(const rg_graph* g, int* directed) {
  if (!g || !directed) return fail(RG_EINVAL, "null argument");
  *directed = g->directed ? 1 : 0;
  return RG_OK;
}

// ---------------------------------------------------------------------------
// readGraph + preprocessGraph in one call (symmetric graphs): only the
// offsets are uploaded; the ranking runs on them while nothing else waits,
// and the relabel reads the neighbour array straight from page-locked host
// memory over the host link, writing the relabelled array into HBM.  The
// unsorted neighbour array never lands on the device, which saves one full
// pass over it.  Host memory the device cannot read in place (pageable, or
// not 16-byte aligned) takes the copy-then-sort path.
// ---------------------------------------------------------------------------
namespace rg {

__global__ void check_offsets(const uint32_t* __restrict__ off, int64_t n, uint32_t m, unsigned int* bad) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += (int64_t)gridDim.x * blockDim.x) {
    const bool ok = (v == 0 ? off[0] == 0u : off[v - 1] <= off[v]) && (v < n || off[n] == m);
    if (!ok) atomicOr(bad, 1u);
  }
}

}  // namespace rg

extern "C" rg_status rg_graph_create_sorted(int64_t n, int64_t m, const uint32_t* h_off, const uint32_t* h_adj,
                                            rg_graph** out, uint32_t* h_new_ids) {
  if (!out || n <= 0 || m < 0 || !h_off || (m > 0 && !h_adj)) return fail(RG_EINVAL, "rg_graph_create_sorted: bad arguments");
  if (n >= 0xFFFFFFFFll || m >= 0xFFFFFFFFll) return fail(RG_EUNSUPPORTED, ">= 2^32 vertices or edges");
  Ctx* c = nullptr;
  RG_TRY(get_ctx(&c));
  cudaStream_t st = c->stream;
  const uint32_t* d_adj = nullptr;
  if (m > 0) {
    cudaPointerAttributes pa;
    if (cudaPointerGetAttributes(&pa, h_adj) == cudaSuccess && pa.type == cudaMemoryTypeHost && pa.devicePointer &&
        ((uintptr_t)pa.devicePointer & 15u) == 0) {
      d_adj = static_cast<const uint32_t*>(pa.devicePointer);
    }
    cudaGetLastError();  // an unregistered pointer is not an error here
  }
  if (m > 0 && !d_adj) {  // copy, then sort
    rg_graph* g0 = nullptr;
    RG_TRY(rg_graph_create(n, m, h_off, h_adj, &g0));
    const rg_status s = rg_graph_degree_sort(g0, out, h_new_ids);
    rg_graph_free(g0);
    return s;
  }
  rg_graph* g0 = nullptr;
  RG_TRY(new_graph(&g0));
  g0->n = n;
  g0->m = m;
  DevBuf info(true, st);
  rg_status s = g0->off.reserve(4 * (n + 1));
  if (s == RG_OK) s = info.reserve(16);
  unsigned int h_info[2] = {0, 0};
  if (s == RG_OK) {
    cudaError_t e = cudaMemcpyAsync(g0->off.p, h_off, 4 * (n + 1), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(info.p, 0, 8, st);
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    const int64_t blocks = std::min<int64_t>((n + 256) / 256, (int64_t)std::max(sms, 1) * 16);
    if (e == cudaSuccess) {
      check_offsets<<<(unsigned)blocks, 256, 0, st>>>(g0->off.as<uint32_t>(), n, (uint32_t)m, info.as<unsigned int>());
      max_degree<<<(unsigned)blocks, 256, 0, st>>>(g0->off.as<uint32_t>(), n, info.as<unsigned int>() + 1);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_info, info.p, 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) s = cuda_fail(e, "graph offsets", __FILE__, __LINE__);
  }
  if (s == RG_OK && h_info[0]) s = fail(RG_EINVAL, "rg_graph_create_sorted: offsets not monotone or not ending at m");
  if (s == RG_OK) {
    g0->max_deg = h_info[1];
    g0->adj.p = const_cast<uint32_t*>(d_adj);  // borrowed: released below without freeing
    s = finish_graph(g0);                       // the chunk partition of the old CSR
    if (s == RG_OK) s = degree_sort_impl(g0, false, out, h_new_ids);
  }
  g0->adj.p = nullptr;
  g0->adj.bytes = 0;
  delete g0;
  return s;
}
