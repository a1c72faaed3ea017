// Stable LSD radix sort of 64-bit keys on a range of their bits (sort.cu): the
// device CSR builder's entry pairs, the in-lists' entries and the degree sort's
// (degree, id) pairs.
#pragma once

#include "rg_device.cuh"

namespace rg {

constexpr int kMaxSortPasses = 8;

// The passes a sort on bits [lo, hi) takes, of up to 8 bits each, and the bits of
// each: evenly many, as a pass ranks its keys bit by bit (42 bits as 8 8 8 8 8 2 took
// 2.17 ms for 67e6 keys, as six times 7 2.07).
__host__ __device__ inline int sort_passes(int lo, int hi) { return (hi - lo + 7) / 8; }
__host__ __device__ inline int sort_width(int lo, int hi) {
  const int passes = sort_passes(lo, hi);
  return passes > 0 ? (hi - lo + passes - 1) / passes : 0;
}

// Scratch of one sort, kept by the caller until its stream has passed the sort.
struct SortScratch {
  DevBuf hist, status;  // digit counts per pass; the tiles' published counts
  explicit SortScratch(cudaStream_t st) : hist(true, st), status(true, st) {}
};

// Sizes and clears the scratch for k keys.
rg_status sort_begin(SortScratch& s, int64_t k, int passes, cudaStream_t st);
// Digit counts of every pass from the keys.  A kernel that makes the keys can
// count them instead (sort_count_key, added to sort_counts).
rg_status sort_count(SortScratch& s, const uint64_t* keys, int64_t k, int lo, int hi, cudaStream_t st);
// Sorts; the result is in *keys (the two buffers change places as needed).
rg_status sort_run(SortScratch& s, uint64_t** keys, uint64_t** other, int64_t k, int lo, int hi, cudaStream_t st);

uint32_t* sort_counts(SortScratch& s);             // 256 per pass
const uint32_t* sort_failed(const SortScratch& s);  // nonzero once a bounded wait gave up: the result is not sorted

// Sorted entries (row << bits | value) -> offsets (n + 1) and values, the tail of
// a CSR build (graph.cu).  clean: repeats and row = value are dropped; *kept
// entries stay.  Syncs `st` once and checks the sort.
rg_status csr_from_sorted_rows(Workspace& ws, const uint64_t* key, int64_t k, int bits, int64_t n, bool clean,
                               DevBuf& off, DevBuf& adj, int64_t* kept, const SortScratch& sort, const char* who,
                               cudaStream_t st);

// Shared-memory digit counts of a kernel that makes keys: zeroed, filled by
// sort_count_key and added to the global ones (256 per pass) by sort_flush.
__device__ __forceinline__ void sort_zero(uint32_t* sh, int passes) {
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) sh[i] = 0;
  __syncthreads();
}
__device__ __forceinline__ void sort_count_key(uint32_t* sh, uint64_t key, int lo, int hi, int passes) {
  const uint64_t x = hi >= 64 ? key : key & ((1ull << hi) - 1);
  const int width = sort_width(lo, hi);
  const uint32_t digits = (1u << width) - 1u;
  for (int p = 0; p < passes; p++) atomicAdd(sh + p * 256 + ((uint32_t)(x >> (lo + width * p)) & digits), 1u);
}
__device__ __forceinline__ void sort_flush(const uint32_t* sh, uint32_t* hist, int passes) {
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) {
    if (sh[i]) atomicAdd(hist + i, sh[i]);
  }
}

}  // namespace rg
