// Bucket plan of large sorts: one or two radix passes on the TOP bits, then every bucket in shared memory.
//
// An LSD sort moves every element once per key byte: eight passes for 64-bit keys. Two passes on the sixteen bits
// below the keys' common prefix already leave every run of equal top bits (a bucket) contiguous and in input order;
// if the largest bucket fits a CTA, one more read and write of the array, with the rest of the key compared in
// shared memory (block_sort_impl.cuh), finishes the sort. 64-bit pairs move three times instead of eight.
//
//   bucket_prepare_kernel  clears the scratch; one CTA samples 8192 keys for their common prefix and for buckets
//                          that are clearly too large (heavy duplicates), another one 32-bit keys for copies: then
//                          nothing further is spent on the plan
//   bucket_count_kernel    counts all 2^B buckets exactly in shared memory, 16 bits each. A key outside the sampled
//                          window is not counted and a counter that overflows loses 65535 or 65536, so the sum
//                          equals n exactly if every count is right. The last CTA decides: buckets of the top eight
//                          bits all fit: one pass; of all B bits: two; else no plan and the byte-wise LSD sort runs.
//                          It also groups neighbouring buckets into tiles of at most one CTA's capacity.
//   (radix_sort.cu)        the radix passes, on the plan's digits
//   bucket_sort_kernel     sorts the tiles
//
// The decision is taken on the device: the host enqueues the same launches either way, and those not needed return
// at once.
#include "block_sort_impl.cuh"
#include "bucket_sort.cuh"

namespace tb200 {
namespace {

constexpr int kCountThreads = 1024;
constexpr int kSamples = 8192;
constexpr int kMaxBucketBits = 16;
constexpr int kMinBucketBits = 13;
constexpr uint64_t kTwoPassMin = 1ull << 22;

// Scratch behind the radix sort's: bucket counts, then where every tile begins.
struct BucketScratch {
  unsigned count[1 << kMaxBucketBits];
  unsigned tile_begin[(1 << kMaxBucketBits) + 8];
  unsigned copies;  // the keys have copies: no plan
};

template <typename UK>
__device__ __forceinline__ bool in_window(UK k, unsigned window_bits, unsigned long long prefix) {
  return window_bits >= 8 * sizeof(UK) || (unsigned long long)(k >> window_bits) == prefix;
}

// This thread's samples of part `part` of `parts` of the keys: groups of 16 bytes, evenly spread with a jitter (single keys
// would cost a sector each: one CTA fetches about two sectors per cycle).
template <typename UK>
__device__ __forceinline__ void load_samples(const UK* __restrict__ keys, uint64_t n, int aligned, unsigned part,
                                             unsigned parts, UK (&key)[kSamples / kCountThreads]) {
  constexpr int VEC = 16 / sizeof(UK), GROUPS = kSamples / kCountThreads / VEC;
  const uint64_t step = n / (kSamples * parts);  // n >= kSamples * parts
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const unsigned s = (part * GROUPS + i) * kCountThreads + threadIdx.x;
    const unsigned long long room = step < 0xffffffffull ? step : 0xffffffffull;
    const unsigned long long jitter = (unsigned long long)(s * 2654435761u) * room >> 32;  // < step
    const uint64_t at = (s * step + jitter) * VEC;
    if (aligned) {
      const KeyVec<UK> v = *reinterpret_cast<const KeyVec<UK>*>(keys + at);
#pragma unroll
      for (int e = 0; e < VEC; ++e) key[i * VEC + e] = v.v[e];
    } else {
#pragma unroll
      for (int e = 0; e < VEC; ++e) key[i * VEC + e] = keys[at + e];
    }
  }
}

// Two passes and the tile sort of 32-bit keys save a sixth of the byte-wise sort's time, and lose a third if the keys have
// copies, because crowded tiles take longer and are more (2^25 keys: 599 us byte-wise; 517 us with the plan if all are
// distinct, 794 us with 16 copies of each). So there is no plan when sampled keys are met again: c copies of each of n / c
// keys give c 2^25 / n pairs among 8192 samples. Where that is too few, four times as many are looked at, and those kept
// whose hash ends in two zeros: four times the pairs. (A key that finds its two cells taken by others is not kept, nor is
// the key 0.) Neighbours in one group of 16 bytes are counted apart: sorted keys would meet there by chance. A CTA of its
// own does this: behind the other one's work it took 4 us of the sort.
template <typename UK>
__device__ void look_for_copies(const UK* __restrict__ keys, uint64_t n, int aligned, BucketScratch* scratch,
                                unsigned* s_seen) {
  constexpr int VEC = 16 / sizeof(UK);
  __shared__ unsigned s_again, s_beside;
  constexpr int kMine = kSamples / kCountThreads, kParts = 4;
  const unsigned parts = n < (1ull << 26) ? 1 : kParts;
  UK key[kParts][kMine];
#pragma unroll
  for (int p = 0; p < kParts; ++p)
    if (p < (int)parts) load_samples(keys, n, aligned, p, parts, key[p]);
  for (int i = threadIdx.x; i < kSamples; i += kCountThreads) s_seen[i] = 0;  // sampled keys by their hash, 0: free
  if (threadIdx.x == 0) s_again = s_beside = 0;
  __syncthreads();
  unsigned again = 0, beside = 0;
#pragma unroll
  for (int p = 0; p < kParts; ++p) {
    if (p >= (int)parts) break;
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const unsigned k = (unsigned)key[p][i], hash = k * 2654435761u;
      if (i % VEC != 0 && key[p][i] == key[p][i % VEC != 0 ? i - 1 : i]) { ++beside; continue; }
      if ((hash >> 17 & (parts - 1)) != 0) continue;
      for (unsigned probe = 0; probe < 2; ++probe) {
        unsigned* cell = &s_seen[((hash >> 19) + probe) % kSamples];
        unsigned old = *(volatile unsigned*)cell;  // a frequent key is there as a rule: no queue of atomics on its cell
        if (old == 0) old = atomicCAS(cell, 0u, k);
        if (old == 0 || old == k) { again += old != 0; break; }
      }
    }
  }
  again = __reduce_add_sync(0xffffffffu, again);
  beside = __reduce_add_sync(0xffffffffu, beside);
  if (lane_id() == 0 && again) atomicAdd(&s_again, again);
  if (lane_id() == 0 && beside) atomicAdd(&s_beside, beside);
  __syncthreads();
  if (threadIdx.x == 0) scratch->copies = s_again >= 2 || s_beside >= kSamples / 4 * parts;
}

template <typename UK>
__global__ void __launch_bounds__(kCountThreads)
bucket_prepare_kernel(const UK* __restrict__ keys, uint64_t n, Encoding enc, SortCtl* ctl, uint64_t clear_bytes,
                      BucketScratch* scratch, int min_bits, int max_bits, unsigned capacity, int aligned) {
  chain_begin();
  constexpr uint64_t kCtlBytes = align_up(sizeof(SortCtl), 256);
  char* base = reinterpret_cast<char*>(ctl);
  const uint4 zero = make_uint4(0, 0, 0, 0);
  __shared__ unsigned s_cell[sizeof(UK) == 4 ? kSamples : 4096];
  const bool ask_copies = sizeof(UK) == 4 && n >= kTwoPassMin;
  const unsigned clear_from = ask_copies ? 2 : 1;  // CTAs in front of those that clear
  if (blockIdx.x >= clear_from) {  // look-back descriptors and bucket counts
    const uint64_t stride = (uint64_t)(gridDim.x - clear_from) * kCountThreads;
    const uint64_t tid = (uint64_t)(blockIdx.x - clear_from) * kCountThreads + threadIdx.x;
    uint4* desc = reinterpret_cast<uint4*>(base + kCtlBytes);
    for (uint64_t i = tid; i < (clear_bytes - kCtlBytes) / 16; i += stride) desc[i] = zero;
    uint4* count = reinterpret_cast<uint4*>(scratch->count);
    for (uint64_t i = tid; i < (uint64_t)(1 << max_bits) / 4; i += stride) count[i] = zero;
    return;
  }
  if (blockIdx.x == 1) return look_for_copies(keys, n, aligned, scratch, s_cell);
  if (!ask_copies && threadIdx.x == 0) scratch->copies = 0;
  __shared__ unsigned s_diff[2], s_most;
  UK key[kSamples / kCountThreads];
  const uint64_t step = n / kSamples;
  load_samples(keys, n, aligned, 0, 1, key);
  const UK ref = encode_key(keys[0], enc);
  for (uint64_t i = threadIdx.x; i < kCtlBytes / 16; i += kCountThreads) reinterpret_cast<uint4*>(base)[i] = zero;
  for (int i = threadIdx.x; i < 4096; i += kCountThreads) s_cell[i] = 0;
  if (threadIdx.x == 0) s_diff[0] = s_diff[1] = s_most = 0;
  __syncthreads();
  unsigned long long diff = 0;
#pragma unroll
  for (int i = 0; i < kSamples / kCountThreads; ++i) {
    key[i] = encode_key(key[i], enc);
    diff |= (unsigned long long)(UK)(key[i] ^ ref);
  }
  const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)diff);
  const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(diff >> 32));
  if (lane_id() == 0) {
    atomicOr(&s_diff[0], lo);
    atomicOr(&s_diff[1], hi);
  }
  __syncthreads();
  diff = (unsigned long long)s_diff[1] << 32 | s_diff[0];
  const int bits = diff ? 64 - __clzll((long long)diff) : 0;
  int bytes = 0;  // passes that the byte-wise sort would take
#pragma unroll
  for (int b = 0; b < 8; ++b) bytes += ((diff >> (8 * b)) & 0xffull) != 0;
  // three bytes or fewer: the byte-wise passes are no dearer than the plan
  bool ok = bytes >= 4 && bits >= max_bits;
  if (ok) {
#pragma unroll
    for (int i = 0; i < kSamples / kCountThreads; ++i)
      atomicAdd(&s_cell[digit_of(key[i], bits - 12, 4095u)], 1u);
  }
  __syncthreads();
  unsigned most = 0;
  for (int i = threadIdx.x; i < 4096; i += kCountThreads) most = max(most, s_cell[i]);
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane_id() == 0) atomicMax(&s_most, most);
  __syncthreads();
  if (threadIdx.x == 0) {
    // The fullest of 4096 cells holds about s_most * step keys. Up to 16 of 8192 samples in one cell are chance and
    // the smallest number of buckets will do; else there are as many as make this cell's fit, if that is enough.
    int bucket_bits = min_bits;
    if (s_most > 16) {
      const unsigned long long cell = (unsigned long long)s_most * step;
      while (bucket_bits < max_bits && (cell >> (bucket_bits - 12)) > capacity / 2) ++bucket_bits;
      ok = ok && (cell >> (bucket_bits - 12)) <= 2ull * capacity;
    }
    // below kTwoPassMin 32-bit keys only a plan of one pass is worth its count (bucket_plan_possible)
    if (sizeof(UK) == 4 && n < kTwoPassMin) ok = ok && s_most <= 16;
    ctl->window_ok = ok;
    ctl->bucket_bits = (unsigned)bucket_bits;
    ctl->window_bits = (unsigned)bits;
    ctl->window_prefix = bits >= 64 ? 0ull : (unsigned long long)ref >> bits;
  }
}

// The last CTA of the count: checks the counts, chooses passes and tiles, writes the plan.
__device__ void decide(SortCtl* ctl, BucketScratch* scratch, uint64_t n, int bucket_bits, unsigned capacity,
                       unsigned* s_mem) {
  unsigned* s_max = s_mem;            // [16] largest group of 2^g neighbouring buckets
  unsigned* s_warp = s_mem + 16;      // [32]
  unsigned* s_digit = s_mem + 64;     // [256]
  unsigned long long* s_sum = reinterpret_cast<unsigned long long*>(s_mem + 48);
  const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid / kWarp;
  const int own_bits = bucket_bits - 10;       // 2^own_bits buckets per thread, eight at least
  const unsigned own = 1u << own_bits;
  const uint4* mine = reinterpret_cast<const uint4*>(scratch->count + tid * own);
  if (tid < 16) s_max[tid] = 0;
  if (tid == 0) *s_sum = 0;
  __syncthreads();

  unsigned m0 = 0, m1 = 0, m2 = 0, m3 = 0, m4 = 0, m5 = 0, a4 = 0, a5 = 0, total = 0;
#pragma unroll 4
  for (unsigned c = 0; c < own / 8; ++c) {
    const uint4 x = __ldcg(mine + 2 * c), y = __ldcg(mine + 2 * c + 1);
    const unsigned p0 = x.x + x.y, p1 = x.z + x.w, p2 = y.x + y.y, p3 = y.z + y.w;
    const unsigned q0 = p0 + p1, q1 = p2 + p3, r = q0 + q1;
    m0 = max(max(max(m0, max(x.x, x.y)), max(x.z, x.w)), max(max(y.x, y.y), max(y.z, y.w)));
    m1 = max(max(m1, max(p0, p1)), max(p2, p3));
    m2 = max(m2, max(q0, q1));
    m3 = max(m3, r);
    a4 += r;
    a5 += r;
    if ((c & 1u) == 1u) { m4 = max(m4, a4); a4 = 0; }
    if ((c & 3u) == 3u) { m5 = max(m5, a5); a5 = 0; }
    total += r;
  }
  auto level = [&](int g, unsigned m) {
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) atomicMax(&s_max[g], m);
  };
  level(0, m0); level(1, m1); level(2, m2); level(3, m3);
  if (own_bits >= 4) level(4, m4);
  if (own_bits >= 5) level(5, m5);
  unsigned group = total;
  for (int s = 0; s <= 5; ++s) {
    if (s > 0) group += __shfl_xor_sync(0xffffffffu, group, 1 << (s - 1));
    level(own_bits + s, group);
  }
  // `group` is the warp's total now; totals fit 32 bits (n <= 2^30)
  unsigned long long sum = lane == 0 ? group : 0;
  if (lane == 0) atomicAdd(s_sum, sum);
  // exclusive start of this thread's buckets
  unsigned incl = total;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned t = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= (unsigned)off) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  unsigned start = lane < warp ? s_warp[lane] : 0;
  start = __reduce_add_sync(0xffffffffu, start) + incl - total;

  const int top = bucket_bits - 8;  // buckets of the top eight bits are groups of 2^top
  if (*s_sum != n) return;          // a key outside the window, or a counter that overflowed: no plan
  int grain, passes;
  if (s_max[top] <= capacity) { grain = top; passes = 1; }
  else if (s_max[0] <= capacity) { grain = 0; passes = 2; }
  else return;

  // Tiles: groups of 2^g whole buckets, or the buckets that begin in [t T, (t + 1) T). Either way a tile holds at
  // most `capacity` elements; the fewer tiles win.
  int g = grain;
  while (g + 1 <= bucket_bits - 5 && s_max[g + 1] <= capacity) ++g;
  const unsigned even_tiles = 1u << (bucket_bits - g);
  const unsigned T = capacity - s_max[grain] + 1;
  const unsigned cut_tiles = (unsigned)(n / T) + 1;
  const bool even = even_tiles <= cut_tiles;
  auto for_each_own = [&](auto f) {  // sixteen counts at a time: their loads overlap
    for (unsigned i = 0; i < own; i += 16) {
      uint4 x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = i + 4 * q < own ? __ldcg(mine + i / 4 + q) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (i + 4 * q < own) { f(i + 4 * q, x[q].x); f(i + 4 * q + 1, x[q].y); f(i + 4 * q + 2, x[q].z); f(i + 4 * q + 3, x[q].w); }
      }
    }
  };
  if (even) {
    if (g >= own_bits) {
      if (((tid << own_bits) & ((1u << g) - 1u)) == 0) scratch->tile_begin[(tid << own_bits) >> g] = start;
    } else {
      unsigned s = start;
      for_each_own([&](unsigned i, unsigned x) {
        if ((i & ((1u << g) - 1u)) == 0) scratch->tile_begin[(tid * own + i) >> g] = s;
        s += x;
      });
    }
    if (tid == 0) scratch->tile_begin[even_tiles] = (unsigned)n;
  } else {
    // a group of buckets [s, e) makes e the begin of every tile t with s < t T <= e
    auto mark = [&](unsigned s, unsigned e) {
      if (e == s) return;
      for (unsigned t = s / T + 1; (unsigned long long)t * T <= e; ++t) scratch->tile_begin[t] = e;
    };
    if (grain == 0) {
      unsigned s = start, t = start / T + 1;
      unsigned long long next = (unsigned long long)t * T;
      for_each_own([&](unsigned, unsigned x) {
        s += x;
        for (; next <= s; next += T) scratch->tile_begin[t++] = s;
      });
    } else {  // a grain spans 2^(top - own_bits) = 4 threads
      unsigned e = total;
      e += __shfl_xor_sync(0xffffffffu, e, 1);
      e += __shfl_xor_sync(0xffffffffu, e, 2);
      if ((tid & 3u) == 0) mark(start, start + e);
    }
    if (tid == 0) {
      scratch->tile_begin[0] = 0;
      scratch->tile_begin[cut_tiles] = (unsigned)n;
    }
  }

  // digit offsets of the passes. Top eight bits: 2^top buckets each, held by four threads.
  __syncthreads();
  {
    if ((tid & 3u) == 0) ctl->offs[passes - 1][tid >> 2] = start;
  }
  const unsigned low = 1u << top;
  if (passes == 2) {  // low digit: every 2^top-th bucket, the rows divided among the threads
    if (tid < 256) s_digit[tid] = 0;
    __syncthreads();
    const unsigned d = tid & (low - 1u), part = tid >> top;
    unsigned c = 0;
#pragma unroll 8
    for (unsigned i = 0; i < own; ++i) c += __ldcg(scratch->count + (((part << own_bits) + i) << top) + d);
    atomicAdd(&s_digit[d], c);
    __syncthreads();
    if (warp < 8) {
      const unsigned x = tid < low ? s_digit[tid] : 0;
      unsigned run = x;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, run, off);
        if (lane >= (unsigned)off) run += t;
      }
      if (lane == 31) s_warp[warp] = run;
      named_barrier(1, 256);
      unsigned before = lane < warp ? s_warp[lane] : 0;
      before = __reduce_add_sync(0xffffffffu, before);
      ctl->offs[0][tid] = before + run - x;
    }
  }
  if (tid < (unsigned)kMaxPasses) {
    ctl->skip[tid] = tid >= (unsigned)passes;
    ctl->exec_before[tid] = tid;
  }
  if (tid == 0) {
    const unsigned w = ctl->window_bits - (unsigned)bucket_bits;
    ctl->pass_shift[0] = passes == 2 ? w : w + (unsigned)top;
    ctl->pass_mask[0] = passes == 2 ? low - 1u : 255u;
    ctl->pass_shift[1] = w + (unsigned)top;
    ctl->pass_mask[1] = 255u;
    ctl->total_exec = (unsigned)passes;
    ctl->last_pass = ~0u;  // the passes leave the keys encoded: the tiles are decoded
    // keys of one tile differ below this bit only (a cut tile may span any two neighbouring groups)
    ctl->tile_bits = even ? w + (unsigned)g : ctl->window_bits;
    ctl->num_bucket_tiles = even ? even_tiles : cut_tiles;
    ctl->bucket_mode = 1;
  }
}

template <typename UK>
__global__ void __launch_bounds__(kCountThreads, 1)
bucket_count_kernel(const UK* __restrict__ keys, uint64_t n, Encoding enc, SortCtl* ctl, BucketScratch* scratch,
                    unsigned capacity, int aligned) {
  constexpr int VEC = 16 / sizeof(UK);
  constexpr int T = kCountThreads;
  constexpr int UNROLL = 4;
  extern __shared__ __align__(16) unsigned s_mem[];  // 2^(bucket_bits - 1) words, two counters each
  __shared__ unsigned s_last;
  chain_begin();
  if (!ctl->window_ok || scratch->copies) return;
  const unsigned window_bits = ctl->window_bits;
  const int bucket_bits = (int)ctl->bucket_bits;
  const unsigned long long prefix = ctl->window_prefix;
  const int shift = (int)window_bits - bucket_bits;
  const unsigned mask = (1u << bucket_bits) - 1u;
  const unsigned words = 1u << (bucket_bits - 1);
  for (unsigned i = threadIdx.x; i < words; i += T) s_mem[i] = 0;
  __syncthreads();
  auto count = [&](UK raw) {
    const UK k = encode_key(raw, enc);
    if (!in_window(k, window_bits, prefix)) return;
    const unsigned b = digit_of(k, shift, mask);
    atomicAdd(&s_mem[b >> 1], (b & 1u) ? 0x10000u : 1u);
  };
  constexpr uint64_t CHUNK = (uint64_t)T * VEC * UNROLL;
  const uint64_t full = aligned ? n / CHUNK : 0;
  for (uint64_t c = blockIdx.x; c < full; c += gridDim.x) {
    const KeyVec<UK>* src = reinterpret_cast<const KeyVec<UK>*>(keys + c * CHUNK);
    KeyVec<UK> v[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) v[u] = src[u * T + threadIdx.x];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
#pragma unroll
      for (int j = 0; j < VEC; ++j) count(v[u].v[j]);
  }
  for (uint64_t i = full * CHUNK + (uint64_t)blockIdx.x * T + threadIdx.x; i < n; i += (uint64_t)gridDim.x * T)
    count(keys[i]);
  __syncthreads();
  // a pair of counters of the CTA joins its pair of 32-bit counters with one 64-bit add (no carry: sums <= n)
  unsigned long long* out = reinterpret_cast<unsigned long long*>(scratch->count);
  for (unsigned i = threadIdx.x; i < words; i += T) {
    const unsigned w = s_mem[i];
    if (w) atomicAdd(out + i, (unsigned long long)(w & 0xffffu) | ((unsigned long long)(w >> 16) << 32));
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&ctl->joint_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  decide(ctl, scratch, n, bucket_bits, capacity, s_mem);
}

template <typename UK, int VB, int THREADS, int ITEMS, int BINS, int MIN_CTAS>
__global__ void __launch_bounds__(THREADS, MIN_CTAS)
bucket_sort_kernel(UK* main_keys, UK* alt_keys, typename ValueOf<VB>::type* main_vals,
                   typename ValueOf<VB>::type* alt_vals, uint64_t n, Encoding enc, const SortCtl* ctl,
                   const BucketScratch* scratch) {
  using B = BlockSort<UK, VB, THREADS, ITEMS, BINS>;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned s_red[B::kRedWords];
  chain_begin();
  const bool odd = ctl->total_exec & 1u;
  if (!ctl->bucket_mode) {
    if (odd) {
      copy_back(reinterpret_cast<uint4*>(main_keys), reinterpret_cast<const uint4*>(alt_keys), n * sizeof(UK));
      if (VB) copy_back(reinterpret_cast<uint4*>(main_vals), reinterpret_cast<const uint4*>(alt_vals), n * (uint64_t)VB);
    }
    return;
  }
  const UK* src_keys = odd ? alt_keys : main_keys;
  const typename B::V* src_vals = odd ? alt_vals : main_vals;
  const unsigned tiles = ctl->num_bucket_tiles;
  const int shift = max(0, (int)ctl->tile_bits - 32);
  unsigned begin = 0, end = 0;
  if (blockIdx.x < tiles) { begin = scratch->tile_begin[blockIdx.x]; end = scratch->tile_begin[blockIdx.x + 1]; }
  for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
    const unsigned m = end - begin, at = begin;
    if (t + gridDim.x < tiles) {  // the next tile comes into L2 while this one is sorted
      begin = scratch->tile_begin[t + gridDim.x];
      end = scratch->tile_begin[t + gridDim.x + 1];
      const char* k = reinterpret_cast<const char*>(src_keys + begin);
      for (unsigned i = threadIdx.x * 128; i < (end - begin) * (unsigned)sizeof(UK); i += THREADS * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(k + i));
      if constexpr (VB != 0) {
        const char* v = reinterpret_cast<const char*>(src_vals + begin);
        for (unsigned i = threadIdx.x * 128; i < (end - begin) * (unsigned)VB; i += THREADS * 128)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(v + i));
      }
    }
    if (m == 0) continue;
    B::template sort<false>(src_keys + at, VB ? src_vals + at : nullptr, main_keys + at, VB ? main_vals + at : nullptr, m,
                            shift, enc, smem, s_red);
    __syncthreads();
  }
}

template <int SIZE> constexpr uint64_t tile_capacity() { return (uint64_t)TileShape<SIZE>::kThreads * TileShape<SIZE>::kItems; }

// The shape whose capacity leaves five standard deviations above the mean of 2^16 evenly filled buckets; -1: none.
int tile_size_of(uint64_t n, int val_bytes) {
  const uint64_t mean = n >> kMaxBucketBits;
  if (n > (1ull << 30)) return -1;
  if (mean <= 4270) return 0;
  if (mean <= 8700) return 1;
  if (mean <= 16700 && val_bytes <= 8) return 2;
  return -1;
}
uint64_t capacity_of(int size) {
  return size == 0 ? tile_capacity<0>() : (size == 1 ? tile_capacity<1>() : tile_capacity<2>());
}
// Fewest and most bits of a bucket number: evenly spread keys fill half a tile per bucket.
int min_bucket_bits(uint64_t n, uint64_t capacity) {
  int bits = 1;
  while (bits < kMaxBucketBits && (capacity << (bits - 1)) < n) ++bits;
  return bits < kMinBucketBits ? kMinBucketBits : bits;
}

template <typename UK> struct CountTag {};
template <typename UK, int VB, int SIZE> struct TileTag {};

template <typename UK>
int plan(SortCtl* ctl, size_t clear_bytes, BucketScratch* scratch, const UK* keys, uint64_t n, int val_bytes,
         const Encoding& enc, cudaStream_t stream) {
  int sms = 0;
  int rc = sm_count_of_device(&sms);
  if (rc) return rc;
  const uint64_t capacity = capacity_of(tile_size_of(n, val_bytes));
  const int min_bits = min_bucket_bits(n, capacity), max_bits = kMaxBucketBits;
  const uint64_t vecs = (clear_bytes + (sizeof(unsigned) << max_bits)) / 16;
  const int aligned = reinterpret_cast<uintptr_t>(keys) % 16 == 0;
  const uint64_t want = 3 + vecs / (4 * kCountThreads);  // two CTAs at most look at the keys, the others clear
  const unsigned grid = (unsigned)(want < (uint64_t)sms ? want : (uint64_t)(sms < 3 ? 3 : sms));
  TB200_CUDA_TRY(launch_chained(bucket_prepare_kernel<UK>, grid, kCountThreads, 0, stream, keys, n, enc, ctl,
                                (uint64_t)clear_bytes, scratch, min_bits, max_bits, (unsigned)capacity, aligned));
  trace_mark(stream, kTraceSortPlan);
  auto kernel = bucket_count_kernel<UK>;
  constexpr size_t kMaxSmem = sizeof(uint16_t) << kMaxBucketBits;
  int per_sm = 0;
  rc = resident_ctas<CountTag<UK>>(kernel, kCountThreads, kMaxSmem, &per_sm);
  if (rc) return rc;
  const uint64_t ctas = (n + 32767) / 32768;
  TB200_CUDA_TRY(launch_chained(kernel, (unsigned)(ctas < (uint64_t)sms ? ctas : (uint64_t)sms), kCountThreads,
                                sizeof(uint16_t) << max_bits, stream, keys, n, enc, ctl, scratch, (unsigned)capacity,
                                aligned));
  trace_mark(stream, kTraceSortPlan);
  return TB200_OK;
}

template <typename UK, int VB, int SIZE>
int finish(const SortCtl* ctl, const BucketScratch* scratch, void* keys, void* keys_alt, void* vals, void* vals_alt,
           uint64_t n, const Encoding& enc, cudaStream_t stream) {
  using S = TileShape<SIZE>;
  using B = BlockSort<UK, VB, S::kThreads, S::kItems, S::kBins>;
  constexpr int kMinCtas = VB == 16 && SIZE == 0 ? 2 : S::kMinCtas;
  auto kernel = bucket_sort_kernel<UK, VB, S::kThreads, S::kItems, S::kBins, kMinCtas>;
  int per_sm = 0, sms = 0;
  int rc = sm_count_of_device(&sms);
  if (rc) return rc;
  rc = resident_ctas<TileTag<UK, VB, SIZE>>(kernel, S::kThreads, B::kSmem, &per_sm);
  if (rc) return rc;
  TB200_CUDA_TRY(launch_chained(kernel, (unsigned)(per_sm * sms), S::kThreads, B::kSmem, stream, static_cast<UK*>(keys),
                                static_cast<UK*>(keys_alt), static_cast<typename B::V*>(vals),
                                static_cast<typename B::V*>(vals_alt), n, enc, ctl, scratch));
  trace_mark(stream, kTraceSortTiles);
  return TB200_OK;
}

template <typename UK, int VB>
int finish_size(const SortCtl* ctl, const BucketScratch* scratch, void* k, void* ka, void* v, void* va, uint64_t n,
                const Encoding& enc, cudaStream_t s) {
  switch (tile_size_of(n, VB)) {
    case 0: return finish<UK, VB, 0>(ctl, scratch, k, ka, v, va, n, enc, s);
    case 1: return finish<UK, VB, 1>(ctl, scratch, k, ka, v, va, n, enc, s);
    default:
      if constexpr (VB <= 8) return finish<UK, VB, 2>(ctl, scratch, k, ka, v, va, n, enc, s);
      return TB200_ERR_UNSUPPORTED;
  }
}

template <typename UK>
int finish_vals(int vb, const SortCtl* ctl, const BucketScratch* scratch, void* k, void* ka, void* v, void* va,
                uint64_t n, const Encoding& enc, cudaStream_t s) {
  switch (vb) {
    case 0: return finish_size<UK, 0>(ctl, scratch, k, ka, v, va, n, enc, s);
    case 1: return finish_size<UK, 1>(ctl, scratch, k, ka, v, va, n, enc, s);
    case 2: return finish_size<UK, 2>(ctl, scratch, k, ka, v, va, n, enc, s);
    case 4: return finish_size<UK, 4>(ctl, scratch, k, ka, v, va, n, enc, s);
    case 8: return finish_size<UK, 8>(ctl, scratch, k, ka, v, va, n, enc, s);
    case 16: return finish_size<UK, 16>(ctl, scratch, k, ka, v, va, n, enc, s);
    default: return TB200_ERR_UNSUPPORTED;
  }
}

}  // namespace

size_t bucket_scratch_bytes(uint64_t n, int key_bytes, int val_bytes) {
  if (key_bytes < 4 || n < kSamples || tile_size_of(n, val_bytes) < 0) return 0;
  return align_up(sizeof(BucketScratch), 256);
}

// 32-bit keys have four byte-wise passes at most: below kTwoPassMin keys only a plan of one pass is worth its count, and one
// pass leaves 256 buckets: more than 237 times a tile's capacity cannot be expected to fit them all (evenly spread keys: a
// mean of 237 / 256 of the capacity leaves five standard deviations at 4608).
bool bucket_plan_possible(uint64_t n, int key_bytes, int val_bytes) {
  return key_bytes != 4 || n >= kTwoPassMin || n <= 237 * capacity_of(tile_size_of(n, val_bytes));
}

int bucket_plan(void* d_ctl, size_t clear_bytes, void* d_bucket_scratch, const void* d_keys, uint64_t n, int key_bytes,
                int val_bytes, int kind, int descending, cudaStream_t stream) {
  const Encoding enc = make_encoding(key_bytes, kind, descending);
  auto* ctl = static_cast<SortCtl*>(d_ctl);
  auto* scratch = static_cast<BucketScratch*>(d_bucket_scratch);
  if (key_bytes == 4) return plan(ctl, clear_bytes, scratch, static_cast<const uint32_t*>(d_keys), n, val_bytes, enc, stream);
  return plan(ctl, clear_bytes, scratch, static_cast<const unsigned long long*>(d_keys), n, val_bytes, enc, stream);
}

int bucket_finish(void* d_ctl, void* d_bucket_scratch, void* d_keys, void* d_keys_alt, void* d_vals, void* d_vals_alt,
                  uint64_t n, int key_bytes, int val_bytes, int kind, int descending, cudaStream_t stream) {
  const Encoding enc = make_encoding(key_bytes, kind, descending);
  const auto* ctl = static_cast<const SortCtl*>(d_ctl);
  const auto* scratch = static_cast<const BucketScratch*>(d_bucket_scratch);
  if (key_bytes == 4)
    return finish_vals<uint32_t>(val_bytes, ctl, scratch, d_keys, d_keys_alt, d_vals, d_vals_alt, n, enc, stream);
  return finish_vals<unsigned long long>(val_bytes, ctl, scratch, d_keys, d_keys_alt, d_vals, d_vals_alt, n, enc, stream);
}

}  // namespace tb200
