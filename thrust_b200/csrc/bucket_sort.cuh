// Host interface of the bucket plan of large sorts (bucket_sort.cu).
#pragma once

#include "common.cuh"

namespace tb200 {

// Threads, items per thread, bins and CTAs per SM of the tile sort, smallest capacity first. The tile sort is bound by
// shared-memory wavefronts (77 % of that pipe's peak; issue slots 40 %, DRAM 44 %: 2^26 (u64,u32) pairs; about 9 us per
// tile of 4096 pairs and CTA, 2 CTAs per SM, 2^28 pairs: 2.0 ms at 3.2 TB/s; shape 2 takes 12.5 ms for 2^30); 8192 bins (0.4 % slower), 768 x 6 (3 % slower), 512 x 9 three times per SM with
// 40 registers (5 % slower on 64-bit keys) and 384 x 12 (equal) were tried.
template <int SIZE> struct TileShape;
template <> struct TileShape<0> { static constexpr int kThreads = 512, kItems = 9, kBins = 16384, kMinCtas = 2; };
template <> struct TileShape<1> { static constexpr int kThreads = 1024, kItems = 9, kBins = 16384, kMinCtas = 1; };
template <> struct TileShape<2> { static constexpr int kThreads = 1024, kItems = 17, kBins = 16384, kMinCtas = 1; };

// Scratch behind the radix sort's own for n elements (0: this size and these types take no bucket plan).
size_t bucket_scratch_bytes(uint64_t n, int key_bytes, int val_bytes);

// False: no keys of this size and type take a plan, and none need be enqueued (where there is scratch for one).
bool bucket_plan_possible(uint64_t n, int key_bytes, int val_bytes);

// First half, instead of clearing the scratch: clears [d_temp, d_temp + clear_bytes) (control block first), samples
// the keys, counts the buckets and, when they fit, writes the plan into the control block.
int bucket_plan(void* d_ctl, size_t clear_bytes, void* d_bucket_scratch, const void* d_keys, uint64_t n, int key_bytes,
                int val_bytes, int kind, int descending, cudaStream_t stream);

// Second half, behind the radix passes: sorts the buckets; without a plan copies the result back from the
// alternate arrays if it ended there.
int bucket_finish(void* d_ctl, void* d_bucket_scratch, void* d_keys, void* d_keys_alt, void* d_vals, void* d_vals_alt,
                  uint64_t n, int key_bytes, int val_bytes, int kind, int descending, cudaStream_t stream);

}  // namespace tb200
