// Sorts that fit one CTA: one launch, no scratch (block_sort_impl.cuh has the algorithm).
#include "block_sort_impl.cuh"
#include "block_sort.cuh"

namespace tb200 {
namespace {

template <typename UK, int VB, int THREADS, int ITEMS, int BINS>
__global__ void __launch_bounds__(THREADS)
block_sort_kernel(UK* keys, typename ValueOf<VB>::type* vals, unsigned n, Encoding enc, int* status) {
  using B = BlockSort<UK, VB, THREADS, ITEMS, BINS>;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned s_red[B::kRedWords];
  if (threadIdx.x == 0) *status = 0;
  B::template sort<true>(keys, vals, keys, vals, n, -1, enc, smem, s_red);
}

template <typename UK, int VB, int THREADS, int ITEMS, int BINS> struct BlockTag {};

template <typename UK, int VB, int THREADS, int ITEMS, int BINS>
int launch_single(void* d_keys, void* d_vals, uint64_t n, const Encoding& enc, int* d_status, cudaStream_t stream) {
  using B = BlockSort<UK, VB, THREADS, ITEMS, BINS>;
  auto kernel = block_sort_kernel<UK, VB, THREADS, ITEMS, BINS>;
  int per_sm = 0;
  const int rc = resident_ctas<BlockTag<UK, VB, THREADS, ITEMS, BINS>>(kernel, THREADS, B::kSmem, &per_sm);
  if (rc) return rc;
  kernel<<<1, THREADS, B::kSmem, stream>>>(static_cast<UK*>(d_keys), static_cast<typename B::V*>(d_vals), (unsigned)n, enc,
                                           d_status);
  trace_mark(stream, kTraceSortBlock);
  return (int)cudaGetLastError();
}

// Threads, items per thread and bins of the CTA by the number of elements.
template <typename UK, int VB>
int single(void* d_keys, void* d_vals, uint64_t n, const Encoding& enc, int* d_status, cudaStream_t stream) {
  if (n <= 1024) return launch_single<UK, VB, 256, 4, 2048>(d_keys, d_vals, n, enc, d_status, stream);
  if (n <= 4608) return launch_single<UK, VB, 384, 12, 8192>(d_keys, d_vals, n, enc, d_status, stream);
  return launch_single<UK, VB, 1024, 9, 16384>(d_keys, d_vals, n, enc, d_status, stream);
}

template <typename UK>
int single_vals(int vb, void* k, void* v, uint64_t n, const Encoding& enc, int* st, cudaStream_t s) {
  switch (vb) {
    case 0: return single<UK, 0>(k, v, n, enc, st, s);
    case 1: return single<UK, 1>(k, v, n, enc, st, s);
    case 2: return single<UK, 2>(k, v, n, enc, st, s);
    case 4: return single<UK, 4>(k, v, n, enc, st, s);
    case 8: return single<UK, 8>(k, v, n, enc, st, s);
    case 16: return single<UK, 16>(k, v, n, enc, st, s);
    default: return TB200_ERR_UNSUPPORTED;
  }
}

}  // namespace

int block_sort_single(void* d_keys, void* d_vals, uint64_t n, int key_bytes, int val_bytes, int kind, int descending,
                      int* d_status, cudaStream_t stream) {
  const Encoding enc = make_encoding(key_bytes, kind, descending);
  switch (key_bytes) {
    case 1: return single_vals<uint8_t>(val_bytes, d_keys, d_vals, n, enc, d_status, stream);
    case 2: return single_vals<uint16_t>(val_bytes, d_keys, d_vals, n, enc, d_status, stream);
    case 4: return single_vals<uint32_t>(val_bytes, d_keys, d_vals, n, enc, d_status, stream);
    case 8: return single_vals<unsigned long long>(val_bytes, d_keys, d_vals, n, enc, d_status, stream);
    default: return TB200_ERR_UNSUPPORTED;
  }
}

}  // namespace tb200
