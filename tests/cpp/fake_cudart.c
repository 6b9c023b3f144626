/* Stand-in for the few runtime calls of a read-back, for a test without a GPU: "device" memory is host memory, and every
 * call is counted. Loaded in front of the CUDA runtime (LD_PRELOAD). */
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

size_t fake_copies, fake_host_allocs, fake_host_frees, fake_syncs;
const void* fake_from[1024];
size_t fake_bytes[1024];
int fake_fail_copy = -1; /* this copy fails */

int cudaMemcpyAsync(void* dst, const void* src, size_t bytes, int kind, void* stream) {
  size_t i = __atomic_fetch_add(&fake_copies, 1, __ATOMIC_SEQ_CST);
  (void)kind, (void)stream;
  if (i < 1024) {
    fake_from[i] = src;
    fake_bytes[i] = bytes;
  }
  if ((int)i == fake_fail_copy) return 1;
  memcpy(dst, src, bytes);
  return 0;
}
int cudaStreamSynchronize(void* stream) {
  (void)stream;
  __atomic_fetch_add(&fake_syncs, 1, __ATOMIC_SEQ_CST);
  return 0;
}
int cudaHostAlloc(void** p, size_t bytes, unsigned flags) {
  (void)flags;
  __atomic_fetch_add(&fake_host_allocs, 1, __ATOMIC_SEQ_CST);
  *p = malloc(bytes);
  return 0;
}
int cudaFreeHost(void* p) {
  __atomic_fetch_add(&fake_host_frees, 1, __ATOMIC_SEQ_CST);
  free(p);
  return 0;
}
