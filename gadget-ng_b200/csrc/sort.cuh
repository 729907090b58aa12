// Radix sort of (uint64 key, uint32 value) pairs on one stream.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace tpm {
// Keys per thread of one digit pass (tiles of 256 threads).  8 for large sorts
// (sort 2.84 -> 2.30 ms at 256^3 against 16, 4 is slower there); fewer where
// tiles of 2,048 keys would leave most of the 148 SMs without a block.
constexpr int SORT_BLOCK = 256;
constexpr int sort_items(int64_t n) { return n <= 131072 ? 2 : n <= 524288 ? 4 : 8; }
// Tiles of the largest table a sort of at most n pairs needs (it grows within
// each range of sort_items and restarts lower in the next).
constexpr int64_t sort_tiles(int64_t n) {
  const int64_t t = (n + SORT_BLOCK * sort_items(n) - 1) / (SORT_BLOCK * sort_items(n));
  const int64_t before = n > 524288 ? 512 : n > 131072 ? 256 : 1;
  return t > before ? t : before;
}
// Scratch bytes radix_sort_u64 needs for n pairs (ping-pong copies, per-tile
// digit counts, the 8x256 histogram, 256-byte alignment of each).
constexpr size_t radix_sort_scratch_bytes(int64_t n) {
  return (size_t)n * (sizeof(uint64_t) + sizeof(uint32_t)) + (size_t)sort_tiles(n) * 256 * sizeof(uint32_t) +
         8 * 256 * sizeof(uint32_t) + 1024;
}
// Stable ascending sort of keys[0..n) (low key_bits bits) carrying vals.
// Synchronises the stream once (to skip constant-digit passes).
void radix_sort_u64(uint64_t* keys, uint32_t* vals, int64_t n, int key_bits, void* scratch, size_t scratch_bytes,
                    cudaStream_t s);
// Sorts of up to this many pairs run in one block.
constexpr int64_t SORT_SMALL_MAX = 8192;
// Same sort with every digit pass run unconditionally: no host
// synchronisation and no device-to-host copy, so it can run on memory the
// caller cannot free or reallocate mid-stream.
void radix_sort_u64_all_passes(uint64_t* keys, uint32_t* vals, int64_t n, void* scratch, size_t scratch_bytes,
                               cudaStream_t s);
}  // namespace tpm
