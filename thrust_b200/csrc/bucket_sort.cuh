// Host interface of the bucket plan of large sorts (bucket_sort.cu).
#pragma once

#include "common.cuh"

namespace tb200 {

// Scratch behind the radix sort's own for n elements (0: this size and these types take no bucket plan).
size_t bucket_scratch_bytes(uint64_t n, int key_bytes, int val_bytes);

// First half, instead of clearing the scratch: clears [d_temp, d_temp + clear_bytes) (control block first), samples
// the keys, counts the buckets and, when they fit, writes the plan into the control block.
int bucket_plan(void* d_ctl, size_t clear_bytes, void* d_bucket_scratch, const void* d_keys, uint64_t n, int key_bytes,
                int val_bytes, int kind, int descending, cudaStream_t stream);

// Second half, behind the radix passes: sorts the buckets; without a plan copies the result back from the
// alternate arrays if it ended there.
int bucket_finish(void* d_ctl, void* d_bucket_scratch, void* d_keys, void* d_keys_alt, void* d_vals, void* d_vals_alt,
                  uint64_t n, int key_bytes, int val_bytes, int kind, int descending, cudaStream_t stream);

}  // namespace tb200
