// Host interface of the shared-memory sort (block_sort.cu).
#pragma once

#include "common.cuh"

namespace tb200 {

// Largest input that one CTA sorts in shared memory: 1024 x 9 elements, which fit with the widest keys and values.
constexpr uint64_t kBlockSortCapacity = 9216;

// Sorts n <= kBlockSortCapacity keys (and values) in place with one CTA; `kind` as in tb200_radix_sort (0 unsigned,
// 1 signed, 2 floating point). Clears the status word at d_status.
int block_sort_single(void* d_keys, void* d_vals, uint64_t n, int key_bytes, int val_bytes, int kind, int descending,
                      int* d_status, cudaStream_t stream);

}  // namespace tb200
