// Device side of the shared-memory sort: stable sort of up to a few thousand elements by one CTA.
//
// A radix pass over the whole array costs a launch, a look-back chain and eight ballots per key whatever the
// size; a range that fits one CTA needs none of that. The CTA
//   1. parks its keys (and values) in shared memory as they come and finds the smallest and the largest 32-bit
//      window of the bits that vary,
//   2. counts the keys in a few thousand bins that divide [min, max] evenly: one shared-memory atomic per key, whose
//      return value is the key's (arbitrary) rank inside its bin. Counters are 8 bits wide, four to a word: an
//      overflow changes the sum of all counters, and then the other way below is taken,
//   3. scans the words of four bins and drops every key's 16-bit index at its place,
//   4. repairs the order inside the bins of two and more by (key, index), so equal keys come out in input order
//      whatever order the atomics took. Bins hold a quarter of a key on average: one key in nine is the second of
//      its bin, and the warp that placed it sorts the bin; each warp gathers its bins in a list first, so that its
//      lanes work side by side,
//   5. gathers keys and values through the indices and writes them out with consecutive lanes.
// Insertion takes steps by the square of a bin's size. Keys with copies fill bins of kCrowd and more: then the CTA ranks
// its keys a second time, in the order of their indices (crowded_way). Counters that overflow leave a least-significant-
// digit radix sort in shared memory over the bits in which the keys differ, ranked by warp match (radix_way). No input
// is refused. 2^24 (u64,u32) pairs in tiles of 4096: distinct keys 145 us; 4 copies of each key 222 us (by insertion 315),
// 16 copies 212 us (655), 100 copies 197 us (by digits 505).
#pragma once

#include "sort_common.cuh"

namespace tb200 {
namespace {

template <typename UK, int VB, int THREADS, int ITEMS, int BINS>
struct BlockSort {
  using V = typename ValueOf<VB>::type;
  static constexpr int kWarps = THREADS / kWarp;
  static constexpr int kCap = THREADS * ITEMS;
  // Bins in words of four 8-bit counters; the padding behind the last element counts in bins of its own, so that no
  // step but the first load and the last store asks whether an element exists. A word sits beside its scan.
  // in_front() adds the counters of a word in one byte, so three of them have to stay below 256: crowded_way sees to it
  // for the real bins, a padding bin holds up to kCap / kPadBins (136 of 17408 elements in 128 bins would be too many).
  static constexpr int kPadBins = 3 * (kCap / 128) < 256 ? 128 : 256;
  // A crowded bin holds kCrowd elements or more, a power of two: one mask finds it among the four of a word. Distinct keys
  // practically never crowd one: eight in a bin of a quarter of a key on average (one tile of 4096 keys in 10^5), sixteen
  // in a bin of half a key or one key. At two copies of every key both ways of ordering a bin cost the same.
  static constexpr unsigned kCrowd = 2 * kCap <= BINS ? 8 : 16;
  static constexpr unsigned kCrowdMask = 0x01010101u * (256u - kCrowd);
  static constexpr int kRealWords = BINS / 4;
  static constexpr int kWords = kRealWords + kPadBins / 4;
  static constexpr int kWordsPerThread = ((kWords + THREADS - 1) / THREADS) | 1;
  static constexpr int kBinBits = 31 - __builtin_clz((unsigned)BINS);
  // Shared memory: keys, values (beside the keys, or in their place once the keys are out), counters and the scan of
  // their words (later the warps' lists; or the digit counters of the radix way), indices.
  static constexpr size_t kBinBytes = (size_t)kWords * sizeof(uint2);
  static constexpr size_t kRadixBytes = (size_t)kWarps * kRadix * sizeof(unsigned);
  static constexpr size_t kCountBytes = kBinBytes > kRadixBytes ? kBinBytes : kRadixBytes;
  static constexpr size_t kIndexBytes = align_up((size_t)kCap * 2, 16);
  static constexpr size_t kParkBytes = align_up((size_t)kCap * sizeof(UK), 16) + align_up((size_t)kCap * VB, 16);
  static constexpr size_t kTurnBytes = align_up((size_t)kCap * (sizeof(UK) > VB ? sizeof(UK) : VB), 16);
  static constexpr size_t kSmemOfCta = (size_t)227 * 1024 / (THREADS <= 512 ? 2 : 1) - 2048;
  static constexpr bool kBeside = VB != 0 && kParkBytes + kCountBytes + kIndexBytes <= kSmemOfCta;
  static constexpr size_t kCountOff = kBeside ? kParkBytes : kTurnBytes;
  static constexpr size_t kIndexOff = kCountOff + kCountBytes;
  static constexpr size_t kSmem = kIndexOff + kIndexBytes;
  static constexpr int kListEntries = (int)(kCountBytes / 4 / kWarps);  // per warp
  static_assert(kListEntries >= 2 * kWarp, "a list is emptied when the next keys might not fit");
  static constexpr int kRedWords = 3 * kWarps;  // static shared words the caller provides
  static_assert(kCap < 65536, "places are 16-bit");
  static_assert(THREADS % kPadBins == 0 && kCap % kPadBins == 0, "the padding fills its bins evenly");
  static_assert(3 * (kCap / kPadBins) < 256 && 4 * kCrowd < 256, "sums of three counters are 8 bits wide too");

  __host__ __device__ static unsigned pad_bin(unsigned thread) { return BINS + thread % kPadBins; }
  // Elements that the counters of `word` in front of counter `b` hold.
  __host__ __device__ static unsigned in_front(unsigned word, unsigned b) {
#ifdef __CUDA_ARCH__
    return __byte_perm(word * 0x01010100u, 0, 0x4440u | b);
#else
    return (word * 0x01010100u >> (8 * b)) & 0xffu;
#endif
  }

  // Exclusive scan of one number per thread.
  __device__ static unsigned scan_threads(unsigned x, unsigned* s_red) {
    const unsigned lane = lane_id(), warp = threadIdx.x / kWarp;
    unsigned incl = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= (unsigned)off) incl += t;
    }
    if (lane == 31) s_red[warp] = incl;
    __syncthreads();
    unsigned before = lane < warp && lane < (unsigned)kWarps ? s_red[lane] : 0;
    before = __reduce_add_sync(0xffffffffu, before);
    return before + incl - x;
  }

  template <bool ENCODE>
  __device__ static UK load_key(const UK* src, unsigned i, unsigned m, const Encoding& enc) {
    UK k = (UK)~(UK)0;
    if (i < m) {
      k = src[i];
      if constexpr (ENCODE) k = encode_key(k, enc);
    }
    return k;
  }

  // 32 bits of a key from bit `shift` (0..32) up.
  __device__ static unsigned window(UK k, int shift) {
    if constexpr (sizeof(UK) == 8) return __funnelshift_rc((unsigned)k, (unsigned)(k >> 32), shift);
    else return (unsigned)k;
  }

  // Radix way. Round j of lane l holds element warp * 32 * ITEMS + 32 j + l, in order; the padding (all-ones keys
  // behind the last element) stays last. A call of its own: its registers are not the common way's.
  template <bool ENCODE>
  __device__ __noinline__ static void radix_way(const UK* src_keys, const V* src_vals, UK* dst_keys, V* dst_vals,
                                                unsigned m, const Encoding enc, unsigned char* smem, unsigned* s_red) {
    UK* s_keys = reinterpret_cast<UK*>(smem);
    unsigned* s_count = reinterpret_cast<unsigned*>(smem + kCountOff);
    unsigned short* s_pos = reinterpret_cast<unsigned short*>(smem + kIndexOff);
    const unsigned lane = lane_id(), warp = threadIdx.x / kWarp;
    const unsigned first = warp * (kWarp * ITEMS) + lane;
    const unsigned lt_mask = lanemask_lt();
    UK key[ITEMS];
    unsigned short at[ITEMS];
    const UK ref = load_key<ENCODE>(src_keys, 0, m, enc);
    unsigned long long differ = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      at[j] = (unsigned short)(first + j * kWarp);
      key[j] = load_key<ENCODE>(src_keys, at[j], m, enc);
      if (at[j] < m) differ |= (unsigned long long)(UK)(key[j] ^ ref);
    }
    __syncthreads();  // s_red has been read
    const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)differ);
    const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(differ >> 32));
    if (lane == 0) { s_red[warp] = lo; s_red[kWarps + warp] = hi; }
    __syncthreads();
    differ = lane < (unsigned)kWarps ? ((unsigned long long)s_red[kWarps + lane] << 32 | s_red[lane]) : 0ull;
    differ = (unsigned long long)__reduce_or_sync(0xffffffffu, (unsigned)(differ >> 32)) << 32 |
             __reduce_or_sync(0xffffffffu, (unsigned)differ);
    const int bits = differ ? 64 - __clzll((long long)differ) : 0;  // all keys agree above these
    for (int shift = 0; shift < bits; shift += 8) {
      if (((differ >> shift) & 0xffull) == 0) continue;
      __syncthreads();  // the counters (or bins) and the sorted slots have been read
      for (int i = threadIdx.x; i < kWarps * kRadix; i += THREADS) s_count[i] = 0;
      __syncthreads();
      unsigned* mine = s_count + warp * kRadix;
      unsigned short rank[ITEMS];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned d = digit_of(key[j], shift, kRadix - 1u);
        const unsigned peers = match_digit(d);
        const unsigned ahead = __popc(peers & lt_mask);
        const unsigned old = mine[d];
        __syncwarp();
        if (ahead == 0) mine[d] = old + __popc(peers);
        __syncwarp();
        rank[j] = (unsigned short)(old + ahead);
      }
      __syncthreads();
      unsigned count = 0;
      if (threadIdx.x < kRadix) {
        for (int w = 0; w < kWarps; ++w) {
          const unsigned c = s_count[w * kRadix + threadIdx.x];
          s_count[w * kRadix + threadIdx.x] = count;
          count += c;
        }
      }
      const unsigned start = scan_threads(count, s_red);
      if (threadIdx.x < kRadix)
        for (int w = 0; w < kWarps; ++w) s_count[w * kRadix + threadIdx.x] += start;
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned p = mine[digit_of(key[j], shift, kRadix - 1u)] + rank[j];
        s_keys[p] = key[j];
        if constexpr (VB != 0) s_pos[p] = at[j];
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        key[j] = s_keys[first + j * kWarp];
        if constexpr (VB != 0) at[j] = s_pos[first + j * kWarp];
      }
    }
    // the values are fetched in sorted order while the source is still whole
    V val[VB ? ITEMS : 1];
    if constexpr (VB != 0) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (first + j * kWarp < m) val[j] = src_vals[at[j]];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (first + j * kWarp < m) {
        dst_keys[first + j * kWarp] = decode_key(key[j], enc);
        if constexpr (VB != 0) dst_vals[first + j * kWarp] = val[j];
      }
    }
  }

  // The bin of a key is (window >> narrow) - bin0, below BINS; s_red holds the warps' smallest and largest windows.
  __device__ __forceinline__ static void find_bins(const unsigned* s_red, int& narrow, unsigned& bin0) {
    const unsigned lane = lane_id();
    const unsigned mn = __reduce_min_sync(0xffffffffu, lane < (unsigned)kWarps ? s_red[lane] : ~0u);
    const unsigned mx = __reduce_max_sync(0xffffffffu, lane < (unsigned)kWarps ? s_red[kWarps + lane] : 0u);
    narrow = max(0, 32 - __clz((int)(mx - mn)) - kBinBits);
    if ((mx >> narrow) - (mn >> narrow) >= (unsigned)BINS) ++narrow;
    bin0 = mn >> narrow;
  }

  // Crowded way: bins of kCrowd elements and more, as keys with many copies give. Repairing such a bin by insertion takes
  // steps by the square of its size, so the elements are ranked a second time, in the order of their indices: the warps
  // take turns, and a warp's atomics on one word are carried out in the order of its lanes. Equal keys then lie in order.
  // Nothing depends on that: the order is checked, and a bin that is not in order (several different keys as a rule) is
  // ranked by comparing all its elements with one another, one place per thread.
  template <bool ENCODE>
  __device__ __noinline__ static void crowded_way(const UK* src_keys, const V* src_vals, UK* dst_keys, V* dst_vals,
                                                  unsigned m, int shift, const Encoding enc, unsigned* s_red) {
    extern __shared__ __align__(16) unsigned char smem[];
    const UK* s_keys = reinterpret_cast<const UK*>(smem);
    uint2* s_bins = reinterpret_cast<uint2*>(smem + kCountOff);
    unsigned short* s_index = reinterpret_cast<unsigned short*>(smem + kIndexOff);
    const unsigned lane = lane_id(), warp = threadIdx.x / kWarp;
    const unsigned first = warp * (kWarp * ITEMS) + lane;
    int narrow;
    unsigned bin0;
    find_bins(s_red, narrow, bin0);
    __syncthreads();  // the sums of the warps have been read
    auto bin_of = [&](UK key) { return (window(key, shift) >> narrow) - bin0; };
    unsigned sum = 0;
    bool over = false;  // the counters of a word together pass 255: in_front() cannot tell its places
    const unsigned w0 = threadIdx.x * kWordsPerThread;
    for (int i = 0; i < kWordsPerThread; ++i) {
      if (w0 + i >= (unsigned)kWords) break;
      const unsigned x = s_bins[w0 + i].x, in_word = __dp4a(x, 0x01010101u, 0u);
      over |= in_word > 255u && w0 + i < (unsigned)kRealWords;
      sum += in_word;
    }
    unsigned run = scan_threads(sum, s_red + 2 * kWarps);
    for (int i = 0; i < kWordsPerThread; ++i) {
      if (w0 + i >= (unsigned)kWords) break;
      s_bins[w0 + i].y = run;
      run = __dp4a(s_bins[w0 + i].x, 0x01010101u, run);
    }
    if (__syncthreads_or(over)) {
      radix_way<ENCODE>(src_keys, src_vals, dst_keys, dst_vals, m, enc, smem, s_red);
      return;
    }
    unsigned at[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const unsigned i = first + j * kWarp;
      const unsigned bin = i < m ? bin_of(s_keys[i]) : pad_bin(threadIdx.x);
      const uint2 w = s_bins[bin >> 2];
      at[j] = bin | (w.y + in_front(w.x, bin & 3u)) << 16;
    }
    __syncthreads();
    for (int w = threadIdx.x; w < kWords; w += THREADS) s_bins[w].x = 0;
    __syncthreads();
    for (unsigned turn = 0; turn < (unsigned)kWarps; turn += 16) {  // sixteen warps in turn: a barrier between two of them
      if (warp - turn < 16u) {
        if (VB != 0 && warp > turn) asm volatile("bar.sync %0, 64;" ::"r"(warp - turn) : "memory");
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
          const unsigned bin = at[j] & 0xffffu, sh = (bin & 3u) * 8u;
          const unsigned old = atomicAdd(&s_bins[bin >> 2].x, 1u << sh);
          at[j] = (at[j] >> 16) + (old >> sh & 0xffu);
        }
        if (VB != 0 && warp - turn < 15u && warp + 1 < (unsigned)kWarps)
          asm volatile("bar.arrive %0, 64;" ::"r"(warp - turn + 1) : "memory");
      }
      if (turn + 16 < (unsigned)kWarps) __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) s_index[at[j]] = (unsigned short)(first + j * kWarp);
    __syncthreads();
    bool any = false;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const unsigned place = j * THREADS + threadIdx.x;
      if (place > 0 && place < m) {
        const unsigned x = s_index[place], y = s_index[place - 1];
        const UK k = s_keys[x], ky = s_keys[y];
        if (k < ky || (VB != 0 && k == ky && x < y)) {  // both are in one bin: the bins themselves lie in order
          const unsigned bin = bin_of(k);
          atomicOr(&s_bins[bin >> 2].y, 0x10000u << (bin & 3u));  // the low half holds the elements in front
          any = true;
        }
      }
    }
    if (__syncthreads_or(any)) {
      unsigned moved[ITEMS];  // index | place << 16
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        unsigned place = j * THREADS + threadIdx.x;
        const unsigned index = s_index[place];
        if (place < m) {
          const UK key = s_keys[index];
          const unsigned bin = bin_of(key);
          const uint2 w = s_bins[bin >> 2];
          if (w.y >> (16 + (bin & 3u)) & 1u) {
            const unsigned begin = (w.y & 0xffffu) + in_front(w.x, bin & 3u);
            const unsigned end = begin + __byte_perm(w.x, 0, 0x4440u | (bin & 3u));
            place = begin;
            for (unsigned t = begin; t < end; ++t) {
              const unsigned x = s_index[t];
              const UK k = s_keys[x];
              place += k < key || (k == key && x < index);
            }
          }
        }
        moved[j] = index | place << 16;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) s_index[moved[j] >> 16] = (unsigned short)moved[j];
      __syncthreads();
    }
    if constexpr (VB == 0 || kBeside) {
      const V* s_vals = reinterpret_cast<const V*>(smem + align_up((size_t)kCap * sizeof(UK), 16));
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned place = j * THREADS + threadIdx.x;
        if (place < m) {
          const unsigned x = s_index[place];
          dst_keys[place] = decode_key(s_keys[x], enc);
          if constexpr (VB != 0) dst_vals[place] = s_vals[x];
        }
      }
    } else {
      V val[ITEMS];  // fetched in sorted order while the source is still whole
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned place = j * THREADS + threadIdx.x;
        if (place < m) val[j] = src_vals[s_index[place]];
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned place = j * THREADS + threadIdx.x;
        if (place < m) {
          dst_keys[place] = decode_key(s_keys[s_index[place]], enc);
          dst_vals[place] = val[j];
        }
      }
    }
  }

  // Sorts m <= kCap elements (m >= 1) from src to dst, which may be the same arrays. ENCODE: the source holds raw
  // keys. The keys are decoded on their way out. All keys agree above bit shift + 32 (shift < 0: find out here); the
  // fewer bits vary below that, the better the bins tell the keys apart.
  template <bool ENCODE>
  __device__ static void sort(const UK* src_keys, const V* src_vals, UK* dst_keys, V* dst_vals, unsigned m, int shift,
                              const Encoding& enc, unsigned char* smem, unsigned* s_red) {
    UK* s_keys = reinterpret_cast<UK*>(smem);
    V* s_vals = reinterpret_cast<V*>(smem + (kBeside ? align_up((size_t)kCap * sizeof(UK), 16) : 0));
    uint2* s_bins = reinterpret_cast<uint2*>(smem + kCountOff);  // x: four counters, y: elements in front of them
    unsigned short* s_index = reinterpret_cast<unsigned short*>(smem + kIndexOff);
    const unsigned lane = lane_id(), warp = threadIdx.x / kWarp;
    const unsigned first = warp * (kWarp * ITEMS) + lane;  // element j of this thread: first + 32 j

    // Elements behind the last one are copies of it that count in bins of their own and come out behind all others,
    // so that no step but the last store depends on m (branches around single elements cost more registers than
    // there are). `have`: elements j < have of this thread exist.
    const int have = ((int)m - (int)first + kWarp - 1) / kWarp;
    const bool all = (warp + 1) * (kWarp * ITEMS) <= m;
    auto load = [&](const auto* src, auto& out) {
      if (all) {
        src += first;  // constant offsets from one address
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) out[j] = src[j * kWarp];
      } else {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) out[j] = src[min(first + j * kWarp, m - 1)];
      }
    };
    static_assert(sizeof(uint2) * kWords % 16 == 0, "cleared 16 bytes at a time");
    unsigned win[ITEMS];
    {
      UK key[ITEMS];
      load(src_keys, key);
      V val[kBeside ? ITEMS : 1];
      if constexpr (kBeside) load(src_vals, val);
      for (int w = threadIdx.x; w < kWords / 2; w += THREADS) reinterpret_cast<uint4*>(s_bins)[w] = make_uint4(0, 0, 0, 0);
      if constexpr (ENCODE) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) key[j] = encode_key(key[j], enc);
      }
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) s_keys[first + j * kWarp] = key[j];
      if (sizeof(UK) == 8 && shift < 0) {
        const UK ref = load_key<ENCODE>(src_keys, 0, m, enc);
        unsigned hi = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) hi |= (unsigned)((unsigned long long)(key[j] ^ ref) >> 32);
        hi = __reduce_or_sync(0xffffffffu, hi);
        if (lane == 0) s_red[2 * kWarps + warp] = hi;
        __syncthreads();
        hi = __reduce_or_sync(0xffffffffu, lane < (unsigned)kWarps ? s_red[2 * kWarps + lane] : 0u);
        shift = 32 - __clz((int)hi);
      }
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) win[j] = window(key[j], shift);
      if constexpr (kBeside) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) s_vals[first + j * kWarp] = val[j];
      }
    }
    unsigned mn = ~0u, mx = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      mn = min(mn, win[j]);
      mx = max(mx, win[j]);
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) { s_red[warp] = mn; s_red[kWarps + warp] = mx; }
    __syncthreads();
    int narrow;
    unsigned bin0;
    find_bins(s_red, narrow, bin0);
    const unsigned pad = pad_bin(threadIdx.x);

    unsigned at[ITEMS];  // bin | rank inside the bin << 16
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      unsigned bin = (win[j] >> narrow) - bin0;
      if (j >= have) bin = pad;
      const unsigned sh = (bin & 3u) * 8u;
      at[j] = atomicAdd(&s_bins[bin >> 2].x, 1u << sh);
      at[j] = bin | (((at[j] >> sh) & 0xffu) << 16);
    }
    __syncthreads();

    // exclusive scan of the words
    unsigned sum = 0, full = 0;
    const unsigned w0 = threadIdx.x * kWordsPerThread;
    unsigned cnt[kWordsPerThread];
#pragma unroll
    for (int i = 0; i < kWordsPerThread; ++i) cnt[i] = w0 + i < (unsigned)kWords ? s_bins[w0 + i].x : 0u;
#pragma unroll
    for (int i = 0; i < kWordsPerThread; ++i) {
      sum = __dp4a(cnt[i], 0x01010101u, sum);
      if (w0 + i < (unsigned)kRealWords) full |= cnt[i];
    }
    unsigned incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= (unsigned)off) incl += t;
    }
    const unsigned crowd = __any_sync(0xffffffffu, (full & kCrowdMask) != 0) ? 1u << 31 : 0u;
    if (lane == 31) s_red[2 * kWarps + warp] = incl | crowd;
    __syncthreads();
    const unsigned of_warp = lane < (unsigned)kWarps ? s_red[2 * kWarps + lane] : 0u;
    const unsigned total = __reduce_add_sync(0xffffffffu, of_warp & ~(1u << 31));
    if (__any_sync(0xffffffffu, of_warp >> 31) || total != (unsigned)kCap) {
      if (total != (unsigned)kCap) radix_way<ENCODE>(src_keys, src_vals, dst_keys, dst_vals, m, enc, smem, s_red);
      else crowded_way<ENCODE>(src_keys, src_vals, dst_keys, dst_vals, m, shift, enc, s_red);
      return;
    }
    unsigned run = __reduce_add_sync(0xffffffffu, lane < warp ? of_warp : 0u) + incl - sum;
#pragma unroll
    for (int i = 0; i < kWordsPerThread; ++i) {
      if (w0 + i < (unsigned)kWords) s_bins[w0 + i].y = run;
      run = __dp4a(cnt[i], 0x01010101u, run);
    }
    __syncthreads();
    // (loads and stores are kept in loops of their own: the compiler does not move a load over a store)
    unsigned second = 0;  // items that are the second of their bin
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const unsigned bin = at[j] & 0xffffu, rank = at[j] >> 16;
      const uint2 w = s_bins[bin >> 2];
      const unsigned begin = w.y + in_front(w.x, bin & 3u);
      const unsigned size = __byte_perm(w.x, 0, 0x4440u | (bin & 3u));
      at[j] = (begin + rank) | (size << 16);
      if (rank == 1 && j < have) second |= 1u << j;
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) s_index[at[j] & 0xffffu] = (unsigned short)(first + j * kWarp);
    V val[!kBeside && VB ? ITEMS : 1];
    if constexpr (!kBeside && VB != 0 && VB <= 8) load(src_vals, val);  // under way while the order is repaired
    __syncthreads();
    // Order inside the bins. The counters are no longer needed: each warp lists the bins it has to sort in its share
    // of their memory, begin | size << 16.
    unsigned* list = reinterpret_cast<unsigned*>(s_bins) + warp * kListEntries;
    unsigned entries = 0;
    auto sort_listed = [&]() {
      __syncwarp();
      for (unsigned e = lane; e < entries; e += kWarp) {
        const unsigned begin = list[e] & 0xffffu, size = list[e] >> 16;
        const unsigned short x0 = s_index[begin], x1 = s_index[begin + 1];  // two keys as a rule
        const UK k0 = s_keys[x0], k1 = s_keys[x1];
        if (k1 < k0 || (k1 == k0 && x1 < x0)) {
          s_index[begin] = x1;
          s_index[begin + 1] = x0;
        }
        for (unsigned a = 2; a < size; ++a) {  // insertion of the others
          const unsigned short x = s_index[begin + a];
          const UK k = s_keys[x];
          unsigned c = a;
          for (; c > 0; --c) {
            const unsigned short y = s_index[begin + c - 1];
            const UK ky = s_keys[y];
            if (ky < k || (ky == k && y < x)) break;
            s_index[begin + c] = y;
          }
          if (c != a) s_index[begin + c] = x;
        }
      }
    };
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      if (kListEntries < kWarp * ITEMS && entries + kWarp > (unsigned)kListEntries) {
        sort_listed();
        __syncwarp();
        entries = 0;
      }
      const bool mine = second >> j & 1u;
      const unsigned votes = __ballot_sync(0xffffffffu, mine);
      if (mine) list[entries + __popc(votes & lanemask_lt())] = at[j] - 1u;
      entries += __popc(votes);
    }
    sort_listed();
    __syncthreads();

    const int out = ((int)m - (int)threadIdx.x + THREADS - 1) / THREADS;  // places j * THREADS + thread, j < out
    const unsigned short* my_index = s_index + threadIdx.x;
    UK* to_keys = dst_keys + threadIdx.x;
    unsigned from[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) from[j] = my_index[j * THREADS];
    const bool plain = (enc.cmask | enc.dmask) == 0;
    UK key[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) key[j] = s_keys[from[j]];
    if (!plain) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) key[j] = decode_key(key[j], enc);
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
      if (j < out) to_keys[j * THREADS] = key[j];
    if constexpr (VB != 0) {
      if constexpr (!kBeside) {
        __syncthreads();
        if constexpr (VB > 8) load(src_vals, val);
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) s_vals[first + j * kWarp] = val[j];
        __syncthreads();
      }
      V* to_vals = dst_vals + threadIdx.x;
      V last[ITEMS];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) last[j] = s_vals[from[j]];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (j < out) to_vals[j * THREADS] = last[j];
    }
  }
};

}  // namespace
}  // namespace tb200
