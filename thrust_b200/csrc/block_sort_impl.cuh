// Device side of the shared-memory sort: stable sort of up to a few thousand elements by one CTA.
//
// A radix pass over the whole array costs a launch, a look-back chain and eight ballots per key whatever the
// size; a range that fits one CTA needs none of that. The CTA
//   1. holds its keys in registers and finds the smallest and the largest 32-bit window of the bits that vary,
//   2. counts them in a few thousand bins that divide [min, max] evenly: one shared-memory atomic per key, whose
//      return value is the key's (arbitrary) rank inside its bin. Counters are 8 bits wide, four to a word: an
//      overflow changes the sum of all counters, and then the other way below is taken,
//   3. scans the words of four bins and drops every key (and, in bins of two and more, its original position) at
//      its place,
//   4. repairs the order inside each bin: a key's place is the number of (key, position) pairs of its bin below
//      its own, so equal keys come out in input order whatever order the atomics took. Bins hold half a key on
//      average; a warp needs about three compares per key,
//   5. drops keys and values at their final places and writes them out with consecutive lanes.
// Keys that crowd into few bins (kCrowd or more in one) take the other way: a least-significant-digit radix sort in
// shared memory over the bits in which the keys differ, ranked by warp match; no input is slow beyond that, and
// none is refused.
#pragma once

#include "sort_common.cuh"

namespace tb200 {
namespace {

constexpr unsigned kCrowd = 32;  // a power of two: one mask finds a crowded bin among the four of a word
constexpr unsigned kCrowdMask = 0x01010101u * (256u - kCrowd);

template <typename UK, int VB, int THREADS, int ITEMS, int BINS>
struct BlockSort {
  using V = typename ValueOf<VB>::type;
  static constexpr int kWarps = THREADS / kWarp;
  static constexpr int kCap = THREADS * ITEMS;
  // Bins in words of four 8-bit counters; the padding behind the last element counts in bins of its own, so that no
  // step but the first load and the last store asks whether an element exists. A word sits beside its scan.
  static constexpr int kPadBins = 128;
  static constexpr int kRealWords = BINS / 4;
  static constexpr int kWords = kRealWords + kPadBins / 4;
  static constexpr int kWordsPerThread = ((kWords + THREADS - 1) / THREADS) | 1;
  static constexpr int kBinBits = 31 - __builtin_clz((unsigned)BINS);
  static constexpr size_t kKeysBytes = align_up((size_t)kCap * (sizeof(UK) > 4 ? sizeof(UK) : 4), 16);  // or windows
  // counters and the scan of their words (or the digit counters of the radix way), then the positions; the values
  // overlay all of it
  static constexpr size_t kBinBytes = (size_t)kWords * sizeof(uint2);
  static constexpr size_t kRadixBytes = (size_t)kWarps * kRadix * sizeof(unsigned);
  static constexpr size_t kCountBytes = kBinBytes > kRadixBytes ? kBinBytes : kRadixBytes;
  static constexpr size_t kWorkBytes = kCountBytes + align_up((size_t)kCap * 2, 16);
  static constexpr size_t kValsBytes = align_up((size_t)kCap * VB, 16);
  static constexpr size_t kSmem = kKeysBytes + (kWorkBytes > kValsBytes ? kWorkBytes : kValsBytes);
  static constexpr int kRedWords = 3 * kWarps;  // static shared words the caller provides
  static_assert(kCap < 65536, "places are 16-bit");
  static_assert(kCap / kPadBins < 256 && THREADS % kPadBins == 0, "the padding's counters are 8 bits wide too");

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
    unsigned* s_count = reinterpret_cast<unsigned*>(smem + kKeysBytes);
    unsigned short* s_pos = reinterpret_cast<unsigned short*>(smem + kKeysBytes + kCountBytes);
    V* s_vals = reinterpret_cast<V*>(smem + kKeysBytes);
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
    // the values are fetched in sorted order while the source is still whole, then both are laid out
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
        s_keys[first + j * kWarp] = key[j];
        if constexpr (VB != 0) s_vals[first + j * kWarp] = val[j];
      }
    }
    __syncthreads();
    write_out(dst_keys, dst_vals, s_keys, s_vals, m, enc);
  }

  __device__ static void write_out(UK* dst_keys, V* dst_vals, const UK* s_keys, const V* s_vals, unsigned m,
                                   const Encoding& enc) {
    UK* to_keys = dst_keys + threadIdx.x;
    V* to_vals = VB ? dst_vals + threadIdx.x : nullptr;
    const UK* from_keys = s_keys + threadIdx.x;
    const V* from_vals = s_vals + threadIdx.x;
    const int have = ((int)m - (int)threadIdx.x + THREADS - 1) / THREADS;
    auto write = [&](auto plain) {
      UK key[ITEMS];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) key[j] = from_keys[j * THREADS];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (j < have) to_keys[j * THREADS] = decltype(plain)::value ? key[j] : decode_key(key[j], enc);
      if constexpr (VB != 0) {
        V val[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) val[j] = from_vals[j * THREADS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
          if (j < have) to_vals[j * THREADS] = val[j];
      }
    };
    if ((enc.cmask | enc.dmask) == 0) write(std::true_type{});
    else write(std::false_type{});
  }

  // Sorts m <= kCap elements (m >= 1) from src to dst, which may be the same arrays. ENCODE: the source holds raw
  // keys. The keys are decoded on their way out. All keys agree above bit shift + 32 (shift < 0: find out here); the
  // fewer bits vary below that, the better the windows tell the keys apart.
  template <bool ENCODE>
  __device__ static void sort(const UK* src_keys, const V* src_vals, UK* dst_keys, V* dst_vals, unsigned m, int shift,
                              const Encoding& enc, unsigned char* smem, unsigned* s_red) {
    UK* s_keys = reinterpret_cast<UK*>(smem);
    unsigned* s_win = reinterpret_cast<unsigned*>(smem);  // the windows, until the keys are dropped at their places
    uint2* s_bins = reinterpret_cast<uint2*>(smem + kKeysBytes);  // x: four counters, y: elements in front of them
    unsigned short* s_pos = reinterpret_cast<unsigned short*>(smem + kKeysBytes + kCountBytes);
    V* s_vals = reinterpret_cast<V*>(smem + kKeysBytes);
    const unsigned lane = lane_id(), warp = threadIdx.x / kWarp;
    const unsigned first = warp * (kWarp * ITEMS) + lane;  // element j of this thread: first + 32 j
    // Elements behind the last one are copies of it that count in bins of their own and come out behind all others,
    // so that no step but the last store depends on m (branches around single elements cost more registers than
    // there are). `have`: elements j < have of this thread exist.
    const int have = ((int)m - (int)first + kWarp - 1) / kWarp;
    const bool all = (warp + 1) * (kWarp * ITEMS) <= m;
    auto load = [&](const auto* src, auto& out, auto anew) {
      auto one = [&](unsigned i) {  // `anew`: a load that the compiler cannot take for an earlier one
        if constexpr (decltype(anew)::value) return __ldcg(src + i);
        else return src[i];
      };
      if (all) {
        src += first;  // constant offsets from one address
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) out[j] = one(j * kWarp);
      } else {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) out[j] = one(min(first + j * kWarp, m - 1));
      }
    };
    // A thread keeps the windows of its keys. 64-bit keys are read a second time (from L2) when their places are
    // known: held in registers all along they would halve the number of warps.
    auto load_keys = [&](UK (&key)[ITEMS], auto anew) {
      load(src_keys, key, anew);
      if constexpr (ENCODE) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) key[j] = encode_key(key[j], enc);
      }
    };
    static_assert(sizeof(uint2) * kWords % 16 == 0, "cleared 16 bytes at a time");
    unsigned win[ITEMS];
    {
      UK key[ITEMS];
      load_keys(key, std::false_type{});
      for (int w = threadIdx.x; w < kWords / 2; w += THREADS) reinterpret_cast<uint4*>(s_bins)[w] = make_uint4(0, 0, 0, 0);
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
    mn = __reduce_min_sync(0xffffffffu, lane < (unsigned)kWarps ? s_red[lane] : ~0u);
    mx = __reduce_max_sync(0xffffffffu, lane < (unsigned)kWarps ? s_red[kWarps + lane] : 0u);

    // bin of a key: (window >> narrow) - bin0 < BINS
    int narrow = max(0, 32 - __clz((int)(mx - mn)) - kBinBits);
    if ((mx >> narrow) - (mn >> narrow) >= (unsigned)BINS) ++narrow;
    const unsigned bin0 = mn >> narrow;
    const unsigned pad_bin = BINS + threadIdx.x % kPadBins;

    unsigned at[ITEMS];  // bin | rank inside the bin << 16, later place of the bin | size << 16 | rank << 22 | below << 27
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      unsigned bin = (win[j] >> narrow) - bin0;
      if (j >= have) bin = pad_bin;
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
    unsigned run = scan_threads(sum, s_red + 2 * kWarps);
    if (__syncthreads_or((full & kCrowdMask) != 0 || (threadIdx.x == THREADS - 1 && run + sum != (unsigned)kCap))) {
      radix_way<ENCODE>(src_keys, src_vals, dst_keys, dst_vals, m, enc, smem, s_red);
      return;
    }
#pragma unroll
    for (int i = 0; i < kWordsPerThread; ++i) {
      if (w0 + i < (unsigned)kWords) s_bins[w0 + i].y = run;
      run = __dp4a(cnt[i], 0x01010101u, run);
    }
    __syncthreads();
    auto size_of = [&](int j) { return (at[j] >> 16) & 0x3fu; };  // <= 31
    auto rank_of = [&](int j) { return (at[j] >> 22) & 0x1fu; };
    auto own_place = [&](int j) { return (at[j] & 0xffffu) + rank_of(j); };
    // (loads and stores are kept in loops of their own: the compiler does not move a load over a store)
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const unsigned bin = at[j] & 0xffffu, rank = at[j] >> 16;
      const uint2 w = s_bins[bin >> 2];
      const unsigned pick = 0x4440u | (bin & 3u);
      const unsigned begin = w.y + __byte_perm(w.x * 0x01010100u, 0, pick);  // counters of a word: 31 each at most
      const unsigned size = __byte_perm(w.x, 0, pick);
      at[j] = begin | (size << 16) | (rank << 22);
      if (j >= have) at[j] = (begin + rank) | (1u << 16);  // alone
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const unsigned p = own_place(j);
      s_win[p] = win[j];
      if (VB != 0 && size_of(j) > 1) s_pos[p] = (unsigned short)(first + j * kWarp);
    }
    __syncthreads();
    // Order inside the bins, by window: step i compares with the key i ranks on, round and round. Two steps are
    // taken for all elements at once, so that their loads overlap; few bins hold more than three keys.
    const bool whole = sizeof(UK) < 8 || shift == 0;  // the window is all of the key that varies
    unsigned again = 0;
    auto other = [&](int j, unsigned i) -> unsigned {
      unsigned q = rank_of(j) + i;
      q = q >= size_of(j) ? q - size_of(j) : q;
      return (at[j] & 0xffffu) + q;
    };
    auto earlier = [&](int j, unsigned q) -> bool {  // the equal key at place q stays in front of key j
      return VB != 0 ? (unsigned)s_pos[q] < first + j * kWarp : q < own_place(j);
    };
    auto step = [&](int j, unsigned i) {
      if (i < size_of(j)) {
        const unsigned q = other(j, i), w = s_win[q];
        bool below = w < win[j];
        if (w == win[j]) {
          if (whole) below = earlier(j, q);
          else again = 1;
        }
        if (below) at[j] += 1u << 27;
      }
    };
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) step(j, 1);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) step(j, 2);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
      for (unsigned i = 3; i < size_of(j); ++i) step(j, i);
    if (!whole && __syncthreads_or(again)) {  // equal windows: whole keys, then positions
      UK key[ITEMS];
      load_keys(key, std::true_type{});
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (size_of(j) > 1) s_keys[own_place(j)] = key[j];
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        if (size_of(j) > 1) at[j] &= (1u << 27) - 1u;
        for (unsigned i = 1; i < size_of(j); ++i) {
          const unsigned q = other(j, i);
          const UK k = s_keys[q];
          if (k < key[j] || (k == key[j] && earlier(j, q))) at[j] += 1u << 27;
        }
      }
    }
    {
      UK key[ITEMS];
      V val[VB ? ITEMS : 1];
      if constexpr (sizeof(UK) == 8) load_keys(key, std::true_type{});
      if constexpr (VB != 0) load(src_vals, val, std::false_type{});
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const unsigned p = (at[j] & 0xffffu) + (at[j] >> 27);
        if constexpr (sizeof(UK) == 8) s_keys[p] = key[j];
        else s_keys[p] = (UK)win[j];
        if constexpr (VB != 0) s_vals[p] = val[j];
      }
    }
    __syncthreads();
    write_out(dst_keys, dst_vals, s_keys, s_vals, m, enc);
  }
};

}  // namespace
}  // namespace tb200
