// One-sweep radix sort (Adinets and Merrill 2022; the look-back is Merrill and
// Garland's single-pass scan, 2016): the digit counts of every pass are taken in one read of
// the keys; each pass then reads and writes every key once.  A tile of kTile
// keys ranks its keys per warp, publishes its digit counts, learns how many
// equal digits lie in earlier tiles by looking back over what those published,
// orders the tile in shared memory and writes runs of equal digits.
//
// Bound by memory: 16 bytes per key and pass.  The sort it replaces counted,
// scanned and scattered key and value arrays in three launches per pass, its
// writes scattered one by one: 67e6 pairs on 42 bits took 7.3 ms.
//
// Tiles take their numbers in the order they start, so whatever a tile waits
// for is already running; the wait is bounded all the same, and a pass that
// gives up raises `fail`, which the caller reads with its own results.

#include <cuda_runtime.h>

#include <algorithm>

#include "app_common.cuh"
#include "sort.cuh"

namespace rg {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 12;
constexpr int kTile = kThreads * kItems;  // 48 KiB of keys: three CTAs per SM
constexpr int kMatchOf = 3;  // one item in this many finds its equals by a match, the others by votes
constexpr unsigned kAll = 0xffffffffu;
constexpr int kBack = 4;  // earlier tiles looked at together
constexpr unsigned kPolls = 1u << 20;  // of the look-back before it gives up
constexpr size_t kHead = 64;  // words of hist before the counts: tickets (0..7) and the failure flag (8)

// base[p][d] = keys of pass p with a digit below d (in place of the counts)
__global__ void sort_bases(uint32_t* hist) {
  __shared__ uint32_t w[8];
  uint32_t* h = hist + blockIdx.x * 256;
  const int lane = threadIdx.x & 31;
  const uint32_t v = h[threadIdx.x];
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kAll, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) w[threadIdx.x >> 5] = inc;
  __syncthreads();
  uint32_t before = 0;
  for (int i = 0; i < (int)(threadIdx.x >> 5); i++) before += w[i];
  h[threadIdx.x] = before + inc - v;
}

__global__ void __launch_bounds__(256) sort_hist_all(const uint64_t* __restrict__ keys, int64_t k, int lo, int hi,
                                                     int passes, uint32_t* hist) {
  __shared__ uint32_t sh[kMaxSortPasses * 256];
  sort_zero(sh, passes);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
    sort_count_key(sh, keys[i], lo, hi, passes);
  }
  sort_flush(sh, hist, passes);
}

// A tile's published count of a digit: its own (kOwn) or with all before it
// (kWhole), tagged with the pass so that one clearing serves every pass.
constexpr uint64_t kOwn = 1, kWhole = 2;
__device__ __forceinline__ uint64_t status_word(uint32_t pass, uint64_t kind, uint32_t count) {
  return ((uint64_t)(pass + 1) << 34) | (kind << 32) | count;
}

// The digit of a key at `shift`.
__device__ __forceinline__ uint32_t digit_of(uint64_t key, int shift, uint32_t digits) {
  const uint32_t lo = (uint32_t)key, hi = (uint32_t)(key >> 32);
  return (shift < 32 ? __funnelshift_r(lo, hi, shift) : hi >> (shift - 32)) & digits;
}

// What a tile shares.
struct Tile {
  uint16_t count[kWarps][257];  // per warp and digit (256: past the end): first counts, then ranks
  uint32_t first[256];          // place of a digit's first key in the ordered tile
  uint32_t to[256];             // its place in the output, less `first`
  uint32_t wsum[8];
  uint32_t tile;
};

// kFull: the tile has kTile keys.  kBits: the most that a digit has.
template <int kBits, bool kFull>
__device__ __forceinline__ void sort_tile(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, int64_t k,
                                          int here, int shift, uint32_t digits, uint32_t pass,
                                          const uint32_t* __restrict__ base, uint64_t* status, uint32_t* head, Tile& T,
                                          uint64_t* keys, unsigned polls) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j0 = w * 32 * kItems + lane;
  const unsigned lt = (1u << lane) - 1u;
  uint64_t key[kItems];
  uint32_t place[kItems];  // rank among the warp's equal digits, then the place in the ordered tile
#pragma unroll
  for (int i = 0; i < kItems; i++) key[i] = kFull || j0 + i * 32 < here ? in[j0 + i * 32] : 0ull;
  uint16_t* mine = T.count[w];
#pragma unroll
  for (int i = 0; i < kItems; i++) {
    const uint32_t d = kFull || j0 + i * 32 < here ? digit_of(key[i], shift, digits) : 256u;
    unsigned peers;
    if (kFull && (i % kMatchOf)) {
      // equal digits by a vote per bit ...
      peers = kAll;
#pragma unroll
      for (int b = 0; b < kBits; b++) {
        const int bit = ((int)(d << (31 - b))) >> 31;
        peers &= ~(__ballot_sync(kAll, bit) ^ (unsigned)bit);
      }
    } else {
      // ... or by one match: the two go through different pipes
      peers = __match_any_sync(kAll, d);
    }
    const uint32_t c = mine[d];
    __syncwarp();
    if (!(peers & lt)) mine[d] = (uint16_t)(c + __popc(peers));
    __syncwarp();
    place[i] = c + __popc(peers & lt);
  }
  __syncthreads();
  uint32_t total = 0, inc = 0;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int x = 0; x < kWarps; x++) {
      const uint16_t c = T.count[x][threadIdx.x];
      T.count[x][threadIdx.x] = (uint16_t)total;
      total += c;
    }
    volatile uint64_t* p = status + (int64_t)T.tile * 256 + threadIdx.x;
    *p = status_word(pass, T.tile == 0 ? kWhole : kOwn, total);
    inc = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kAll, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) T.wsum[w] = inc;
  }
  __syncthreads();
  uint32_t f = 0;
  if (threadIdx.x < 256) {
    f = inc - total;
    for (int x = 0; x < w; x++) f += T.wsum[x];
    T.first[threadIdx.x] = f;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; i++) {
    if (kFull || j0 + i * 32 < here) {
      const uint32_t d = digit_of(key[i], shift, digits);
      keys[T.first[d] + mine[d] + place[i]] = key[i];
    }
  }
  // look back while the others order the tile
  if (threadIdx.x < 256) {
    uint32_t before = 0;
    unsigned spins = 0;
    bool whole = T.tile == 0;
    for (int64_t t = (int64_t)T.tile - 1; !whole;) {
      // kBack tiles at a time, so that their loads overlap; those up to the
      // first that has published nothing yet are taken
      uint64_t x[kBack];
#pragma unroll
      for (int i = 0; i < kBack; i++) {
        const volatile uint64_t* p = status + (t - i) * 256 + threadIdx.x;
        x[i] = t - i >= 0 ? *p : 0ull;
      }
      bool open = true;
#pragma unroll
      for (int i = 0; i < kBack; i++) {
        open = open && !whole && (x[i] >> 34) == pass + 1;
        if (open) {
          before += (uint32_t)x[i];
          whole = (x[i] >> 32) & kWhole;
          t--;
        }
      }
      if (!whole && ++spins > polls) {
        atomicExch(head + 8, 1u);
        break;
      }
    }
    if (T.tile > 0) {
      volatile uint64_t* p = status + (int64_t)T.tile * 256 + threadIdx.x;
      *p = status_word(pass, kWhole, before + total);
    }
    T.to[threadIdx.x] = base[threadIdx.x] + before - f;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; i++) {
    const int j = threadIdx.x + i * kThreads;
    if (kFull || j < here) {
      const uint64_t x = keys[j];
      const uint32_t at = T.to[digit_of(x, shift, digits)] + (uint32_t)j;  // modulo 2^32
      if (at < k) out[at] = x;  // (past the end only when a wait gave up)
    }
  }
}

template <int kBits>
__global__ void __launch_bounds__(kThreads, 3) sort_sweep(const uint64_t* __restrict__ in, uint64_t* __restrict__ out,
                                                          int64_t k, int shift, uint32_t digits, uint32_t pass,
                                                          const uint32_t* __restrict__ base, uint64_t* status,
                                                          uint32_t* head, unsigned polls) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* keys = reinterpret_cast<uint64_t*>(smem_raw);
  __shared__ Tile T;
  if (threadIdx.x == 0) T.tile = atomicAdd(head + pass, 1u);
  for (int i = threadIdx.x; i < kWarps * 257; i += kThreads) (&T.count[0][0])[i] = 0;
  __syncthreads();
  const int64_t t0 = (int64_t)T.tile * kTile;
  const int here = (int)min((int64_t)kTile, k - t0);
  if (here == kTile) sort_tile<kBits, true>(in + t0, out, k, here, shift, digits, pass, base, status, head, T, keys, polls);
  else sort_tile<kBits, false>(in + t0, out, k, here, shift, digits, pass, base, status, head, T, keys, polls);
}

}  // namespace

rg_status sort_begin(SortScratch& s, int64_t k, int passes, cudaStream_t st) {
  const int64_t tiles = (k + kTile - 1) / kTile;
  RG_TRY(s.hist.reserve(4 * (kHead + 256 * (size_t)passes)));
  RG_TRY(s.status.reserve(8 * 256 * (size_t)std::max<int64_t>(tiles, 1)));
  RG_CUDA(cudaMemsetAsync(s.hist.p, 0, 4 * (kHead + 256 * (size_t)passes), st));
  RG_CUDA(cudaMemsetAsync(s.status.p, 0, 8 * 256 * (size_t)std::max<int64_t>(tiles, 1), st));
  return RG_OK;
}

rg_status sort_count(SortScratch& s, const uint64_t* keys, int64_t k, int lo, int hi, cudaStream_t st) {
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((k + 2047) / 2048, (int64_t)device_sms() * 8));
  sort_hist_all<<<(unsigned)blocks, 256, 0, st>>>(keys, k, lo, hi, sort_passes(lo, hi), sort_counts(s));
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

namespace {

template <int kBits>
rg_status sort_passes_of(SortScratch& s, uint64_t** keys, uint64_t** other, int64_t k, int lo, int hi,
                         cudaStream_t st) {
  static std::atomic<uint64_t> limit_set{0};
  RG_TRY(allow_max_dyn_smem(limit_set, sort_sweep<kBits>));
  const int passes = sort_passes(lo, hi), width = sort_width(lo, hi);
  const int64_t tiles = (k + kTile - 1) / kTile;
  for (int p = 0; p < passes; p++) {
    const int shift = lo + width * p;
    const uint32_t digits = (1u << std::min(width, hi - shift)) - 1u;
    sort_sweep<kBits><<<(unsigned)tiles, kThreads, kTile * sizeof(uint64_t), st>>>(
        *keys, *other, k, shift, digits, (uint32_t)p, sort_counts(s) + 256 * p, s.status.as<uint64_t>(),
        s.hist.as<uint32_t>(), g_wait_polls >= 0 ? (unsigned)g_wait_polls : kPolls);
    std::swap(*keys, *other);
  }
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

}  // namespace

rg_status sort_run(SortScratch& s, uint64_t** keys, uint64_t** other, int64_t k, int lo, int hi, cudaStream_t st) {
  if (k == 0) return RG_OK;
  sort_bases<<<sort_passes(lo, hi), 256, 0, st>>>(sort_counts(s));
  const int width = sort_width(lo, hi);
  auto run = width > 7 ? sort_passes_of<8> : width > 6 ? sort_passes_of<7> : width > 5 ? sort_passes_of<6>
                                                                                        : sort_passes_of<5>;
  return run(s, keys, other, k, lo, hi, st);
}

uint32_t* sort_counts(SortScratch& s) { return s.hist.as<uint32_t>() + kHead; }
const uint32_t* sort_failed(const SortScratch& s) { return s.hist.as<uint32_t>() + 8; }

}  // namespace rg
