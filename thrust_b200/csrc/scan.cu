// Single-pass prefix sum (inclusive / exclusive, plus) with a decoupled look-back
// chain of tile descriptors. Streaming kernel: 1 read + 1 write per element, no
// tensor cores (nothing here is a contraction).
//
// Data layout of one tile (kThreads * kVecs 16-byte vectors): warp w owns a
// contiguous slice; inside the slice lane l holds vectors l, l+32, l+64, ... so
// that every load/store instruction of a warp touches 512 contiguous bytes.
// Order of summation: left to right inside a vector, Kogge-Stone across the
// lanes of a warp, left to right across warps and tiles. Integer results are
// exact (two's complement wrap); floating-point results differ from a strictly
// sequential sum only by re-association.
#include "common.cuh"

#include <mutex>
#include <type_traits>

namespace tb200 {
namespace {

// 512 threads x 8 vectors = 64 KiB per tile. Large tiles keep the number of tiles
// per microsecond (about 50 at full HBM speed) well below what the look-back chain
// can resolve: a warp inspects 64 predecessors per L2 round trip.
constexpr int kScanThreads = 512;
constexpr int kScanMinCtas = 2;
constexpr int kScanWarps = kScanThreads / kWarp;
constexpr int kScanVecs = 8;  // 16-byte vectors per thread

template <typename T>
struct alignas(16) Vec16 {
  T v[16 / sizeof(T)];
};

template <typename T>
struct Words {
  static constexpr int W = sizeof(T) / 4;
  __device__ static void pack(T x, unsigned (&p)[W]) {
    if constexpr (W == 1) {
      p[0] = __builtin_bit_cast(unsigned, x);
    } else {
      unsigned long long b = __builtin_bit_cast(unsigned long long, x);
      p[0] = (unsigned)b;
      p[1] = (unsigned)(b >> 32);
    }
  }
  __device__ static T unpack(const unsigned (&p)[W]) {
    if constexpr (W == 1) {
      return __builtin_bit_cast(T, p[0]);
    } else {
      return __builtin_bit_cast(T, ((unsigned long long)p[1] << 32) | p[0]);
    }
  }
};

// What a descriptor of the look-back chain carries: the sum of a tile, or of everything up to its end.
template <typename T>
struct Link {
  static constexpr int W = Words<T>::W;
  using Sum = T;
  __device__ static void publish(TileWords<W>* d, unsigned state, Sum x) {
    unsigned payload[W];
    Words<T>::pack(x, payload);
    tb200::publish<W>(d, state, payload);
  }
  __device__ static unsigned peek(const TileWords<W>* d, Sum& x) {
    unsigned payload[W];
    const unsigned state = tb200::peek<W>(d, payload);
    x = Words<T>::unpack(payload);
    return state;
  }
  __device__ static Sum settle(Sum x) { return x; }
};
// Prefixes of floats travel in 64 bits: a prefix is the end of a long chain of additions, and every one of them would round
// it (2^28 whole numbers, 26215 tiles: errors of up to 24 times 2^-24 of the result, 3 this way; random numbers: 1.1e-6 of
// the norm, 2e-7 this way; 391 us and 395 us). The state takes the two lowest bits of the word, so a descriptor stays as
// small as a float's. A sum beyond the floats becomes the infinity that it would have become as a float.
template <>
struct Link<float> {
  using Sum = double;
  __device__ static void publish(TileWords<1>* d, unsigned state, Sum x) {
    st_relaxed_u64(&d->w[0], (__builtin_bit_cast(unsigned long long, x) & ~3ull) | state);
  }
  __device__ static unsigned peek(const TileWords<1>* d, Sum& x) {
    const unsigned long long w = ld_relaxed_u64(&d->w[0]);
    x = __builtin_bit_cast(double, w & ~3ull);
    return (unsigned)w & 3u;
  }
  // (2^128 - 2^103 is the first number that rounds to an infinity)
  __device__ static Sum settle(Sum x) { return fabs(x) >= 0x1.ffffffp127 ? copysign((double)INFINITY, x) : x; }
};

// Warp 0 walks back over predecessor descriptors, 32 * kLookSlots at a time (kLookSlots
// per lane, all loads in flight together), until it meets one that carries a full prefix.
// Returns the sum of everything before `tile`.
constexpr int kLookSlots = 1;
template <typename T>
__device__ typename Link<T>::Sum lookback_sum(const TileWords<Words<T>::W>* tiles, unsigned tile, int* status) {
  using Sum = typename Link<T>::Sum;
  const unsigned lane = lane_id();
  Sum acc = Sum(0);
  long long base = (long long)tile - 1;
  bool timed_out = false;
  while (true) {
    // slot 0 is the nearest part of the window (tiles base-lane), higher slots lie farther
    // back. All loads are issued first; slots are then consumed nearest first and the
    // walk stops at the first prefix, so descriptors behind it are never waited for.
    unsigned st[kLookSlots];
    Sum found_sum[kLookSlots];
#pragma unroll
    for (int s = 0; s < kLookSlots; ++s) {
      const long long idx = base - 32 * s - lane;
      st[s] = kStatePrefix;
      found_sum[s] = Sum(0);
      if (idx >= 0) st[s] = Link<T>::peek(&tiles[idx], found_sum[s]);
    }
    bool found = false;
#pragma unroll
    for (int s = 0; s < kLookSlots; ++s) {
      if (found) break;
      const long long idx = base - 32 * s - lane;
      Sum v = Sum(0);
      if (idx >= 0) {
        unsigned polls = 0;
        while (st[s] == kStateEmpty) {
          backoff(++polls);
          if (polls >= kSpinLimit || ((polls & 255u) == 0 && ld_relaxed_s32(status) != 0)) {
            timed_out = true;
            st[s] = kStatePrefix;
            break;
          }
          st[s] = Link<T>::peek(&tiles[idx], found_sum[s]);
        }
        v = timed_out ? Sum(0) : found_sum[s];
      }
      const unsigned pm = __ballot_sync(0xffffffffu, st[s] == kStatePrefix);
      const unsigned first = pm ? (unsigned)(__ffs(pm) - 1) : 31u;
      // far predecessors (high lanes) are summed before near ones
      auto tree = [lane](auto x) {
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const auto o = __shfl_down_sync(0xffffffffu, x, off);
          if (lane + off < 32) x = o + x;
        }
        return __shfl_sync(0xffffffffu, x, 0);
      };
      if constexpr (std::is_same<Sum, T>::value) {
        if (lane > first) v = Sum(0);
        v = tree(v);
      } else {  // the sums of the tiles are Ts: only what they add up to joins the prefix in Sum (a tree of Sums took 2.5 %)
        const T tiles_only = tree(pm == 0 || lane < first ? (T)v : T(0));
        v = (pm ? __shfl_sync(0xffffffffu, v, first) : Sum(0)) + (Sum)tiles_only;
      }
      acc = v + acc;
      found = pm != 0;
    }
    if (found) break;
    base -= 32 * kLookSlots;
  }
  if (__any_sync(0xffffffffu, timed_out) && lane == 0) atomicExch(status, (int)TB200_ERR_WAIT_TIMEOUT);
  return Link<T>::settle(acc);
}

// Pointers that are not 16-byte aligned (the streaming kernel's bulk copies need them aligned), above one wave of tiles.
template <typename T, bool EXCLUSIVE>
__global__ void __launch_bounds__(kScanThreads, kScanMinCtas)
scan_kernel(const T* in, T* out, uint64_t n, T init, TempHeader* hdr,
            TileWords<Words<T>::W>* tiles) {
  constexpr int VEC = 16 / sizeof(T);
  constexpr int K = kScanVecs;
  constexpr int WARP_ITEMS = kWarp * K * VEC;
  constexpr int TILE = kScanThreads * K * VEC;

  __shared__ unsigned s_tile;
  __shared__ T s_warp_total[kScanWarps];
  __shared__ T s_tile_prefix;

  if (threadIdx.x == 0) s_tile = atomicAdd(&hdr->ticket, 1u);
  __syncthreads();
  const unsigned tile = s_tile;
  const unsigned warp = threadIdx.x / kWarp;
  const unsigned lane = lane_id();
  const uint64_t tile_base = (uint64_t)tile * TILE;
  const uint64_t warp_base = tile_base + (uint64_t)warp * WARP_ITEMS;

  T x[K][VEC];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      const uint64_t i = warp_base + (uint64_t)(k * kWarp + lane) * VEC + j;
      x[k][j] = i < n ? in[i] : T(0);
    }

  // inclusive sums inside each vector, then across the lanes of the warp
  T excl[K];
  T carry = T(0);
#pragma unroll
  for (int k = 0; k < K; ++k) {
#pragma unroll
    for (int j = 1; j < VEC; ++j) x[k][j] = x[k][j - 1] + x[k][j];
    T s = x[k][VEC - 1];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      T t = __shfl_up_sync(0xffffffffu, s, off);
      if (lane >= off) s = t + s;
    }
    T e = __shfl_up_sync(0xffffffffu, s, 1);
    if (lane == 0) e = T(0);
    excl[k] = carry + e;
    carry = carry + __shfl_sync(0xffffffffu, s, 31);
  }
  if (lane == 31) s_warp_total[warp] = carry;
  __syncthreads();

  T warp_prefix = T(0), tile_total = T(0);
#pragma unroll
  for (int w = 0; w < kScanWarps; ++w) {
    const T t = s_warp_total[w];
    if (w < (int)warp) warp_prefix = warp_prefix + t;
    tile_total = tile_total + t;
  }

  if (warp == 0) {
    typename Link<T>::Sum prefix = init;  // the seed: in front of the first element in both forms
    if (tile != 0) {
      if (lane == 0) Link<T>::publish(&tiles[tile], kStateAggregate, tile_total);
      prefix = lookback_sum<T>(tiles, tile, &hdr->status);
    }
    if (lane == 0) {
      Link<T>::publish(&tiles[tile], kStatePrefix, Link<T>::settle(prefix + tile_total));
      s_tile_prefix = (T)prefix;
    }
  }
  __syncthreads();
  const T base = s_tile_prefix + warp_prefix;

#pragma unroll
  for (int k = 0; k < K; ++k) {
    const T p = base + excl[k];
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      const uint64_t i = warp_base + (uint64_t)(k * kWarp + lane) * VEC + j;
      T r;
      if (EXCLUSIVE) r = j == 0 ? p : p + x[k][j - 1];
      else           r = p + x[k][j];
      if (i < n) out[i] = r;
    }
  }
}

// ---------------------------------------------------------------------------------------
// Inputs of which every CTA takes ONE tile: all tiles are in flight at once, so a tile needs no chain of prefixes.
// Every CTA publishes the sum of its tile and adds up the sums of ALL tiles in front of it itself, one tile per
// thread: one trip to L2 whatever the number of tiles (a 32-wide chain takes a trip per 32 tiles, and the streaming
// kernel's ring of five tiles per CTA leaves four SMs in five without work at these sizes). The sums are added in a
// fixed order, so results do not vary from run to run.
//   CLUSTER: at most kClusterTiles tiles, one thread-block cluster. The sums travel through distributed shared memory:
//            nothing in the scratch needs clearing, the scan is a single launch.
//   else:    tiles are drawn by ticket (a tile only waits for running CTAs) and the sums travel through the scratch.
// Latency-bound, device time in a replayed graph: 100003 int64 elements 21.4 -> 9.8 us, 1048576 int64 25 -> 16 us,
// 4194304 float 29 -> 17.5 us (clear and launch included; an empty call measures about 8.5 us this way).
// ---------------------------------------------------------------------------------------
constexpr int kClusterTiles = 16;

template <typename T, bool EXCLUSIVE, int K, bool CLUSTER>
__global__ void __launch_bounds__(kScanThreads, kScanMinCtas)
scan_wave_kernel(const T* in, T* out, uint64_t n, T init, TempHeader* hdr, TileWords<Words<T>::W>* tiles, int aligned) {
  constexpr int W = Words<T>::W;
  constexpr int VEC = 16 / sizeof(T);
  constexpr int WARP_ITEMS = kWarp * K * VEC;
  constexpr int TILE = kScanThreads * K * VEC;
  __shared__ unsigned s_tile;
  __shared__ T s_warp_total[kScanWarps];
  __shared__ T s_before[kScanWarps];
  __shared__ T s_total;  // CLUSTER: the tile's sum, read by the tiles behind it

  unsigned tile;
  if constexpr (CLUSTER) {
    tile = blockIdx.x;
    if (tile == 0 && threadIdx.x == 0) hdr->status = 0;
  } else {
    if (threadIdx.x == 0) s_tile = atomicAdd(&hdr->ticket, 1u);
    __syncthreads();
    tile = s_tile;
  }
  const unsigned warp = threadIdx.x / kWarp;
  const unsigned lane = lane_id();
  const uint64_t tile_base = (uint64_t)tile * TILE;
  const uint64_t warp_base = tile_base + (uint64_t)warp * WARP_ITEMS;
  const bool full = aligned && tile_base + TILE <= n;

  T x[K][VEC];
  if (full) {
    const Vec16<T>* src = reinterpret_cast<const Vec16<T>*>(in + warp_base);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const Vec16<T> v = src[k * kWarp + lane];
#pragma unroll
      for (int j = 0; j < VEC; ++j) x[k][j] = v.v[j];
    }
  } else {
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const uint64_t i = warp_base + (uint64_t)(k * kWarp + lane) * VEC + j;
        x[k][j] = i < n ? in[i] : T(0);
      }
  }

  // inclusive sums inside each vector, then across the lanes of the warp
  T excl[K];
  T carry = T(0);
#pragma unroll
  for (int k = 0; k < K; ++k) {
#pragma unroll
    for (int j = 1; j < VEC; ++j) x[k][j] = x[k][j - 1] + x[k][j];
    T s = x[k][VEC - 1];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const T t = __shfl_up_sync(0xffffffffu, s, off);
      if (lane >= off) s = t + s;
    }
    T e = __shfl_up_sync(0xffffffffu, s, 1);
    if (lane == 0) e = T(0);
    excl[k] = carry + e;
    carry = carry + __shfl_sync(0xffffffffu, s, 31);
  }
  if (lane == 31) s_warp_total[warp] = carry;
  __syncthreads();
  T warp_prefix = T(0), tile_total = T(0);
#pragma unroll
  for (int w = 0; w < kScanWarps; ++w) {
    const T t = s_warp_total[w];
    if (w < (int)warp) warp_prefix = warp_prefix + t;
    tile_total = tile_total + t;
  }

  // the sum of the tile, and thread i's share of what lies in front of it: the sum of tile i
  T before = T(0);
  if constexpr (CLUSTER) {
    if (threadIdx.x == 0) s_total = tile_total;
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (threadIdx.x < tile) {
      unsigned remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(&s_total)), "r"(threadIdx.x));
      unsigned w[W];
#pragma unroll
      for (int i = 0; i < W; ++i)
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(w[i]) : "r"(remote + 4u * i) : "memory");
      before = Words<T>::unpack(w);
    }
  } else {
    if (threadIdx.x == 0) {
      unsigned payload[W];
      Words<T>::pack(tile_total, payload);
      publish<W>(&tiles[tile], kStateAggregate, payload);
    }
    if (threadIdx.x < tile) {
      unsigned payload[W], polls = 0;
      bool timed_out = false;
      while (peek<W>(&tiles[threadIdx.x], payload) == kStateEmpty) {
        backoff(++polls);
        if (polls >= kSpinLimit || ((polls & 255u) == 0 && ld_relaxed_s32(&hdr->status) != 0)) {
          timed_out = true;
          break;
        }
      }
      if (timed_out) atomicExch(&hdr->status, (int)TB200_ERR_WAIT_TIMEOUT);
      else before = Words<T>::unpack(payload);
    }
  }
  // add the shares in the order of the tiles (tile <= kScanThreads, so one share per thread is all there is)
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const T o = __shfl_down_sync(0xffffffffu, before, off);
    if (lane + off < 32) before = before + o;
  }
  if (lane == 0) s_before[warp] = before;
  __syncthreads();
  T base = init;  // the seed: in front of the first element in both forms
#pragma unroll
  for (int w = 0; w < kScanWarps; ++w) base = base + s_before[w];
  base = base + warp_prefix;

#pragma unroll
  for (int k = 0; k < K; ++k) {
    const T p = base + excl[k];
    Vec16<T> v;
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      if (EXCLUSIVE) v.v[j] = j == 0 ? p : p + x[k][j - 1];
      else           v.v[j] = p + x[k][j];
    }
    if (full) {
      reinterpret_cast<Vec16<T>*>(out + warp_base)[k * kWarp + lane] = v;
    } else {
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const uint64_t i = warp_base + (uint64_t)(k * kWarp + lane) * VEC + j;
        if (i < n) out[i] = v.v[j];
      }
    }
  }
  if constexpr (CLUSTER) {  // a CTA's shared memory stays until every tile behind it has read its sum
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
}

// ---------------------------------------------------------------------------------------
// Streaming variant (16-byte aligned input and output): persistent CTAs, one per SM, each
// with 16 compute warps and one look-back warp.
//  * a ring of (park + 2) tiles in shared memory is filled by bulk asynchronous copies
//    (one elected thread, completion on an mbarrier), issued one to two tiles ahead of use;
//  * the compute warps scan tile i locally — thread t owns a contiguous run of the tile, so
//    one warp scan per tile suffices — publish the tile's aggregate and park the locally
//    resolved values in the tile's own ring slot;
//  * the look-back warp resolves the prefix of tile i while the compute warps go on with
//    tiles i+1 .. i+park, so the look-back latency (several L2 round trips) is off the
//    data path;
//  * the compute warps then re-read the parked tile lane-strided, add the prefix and store
//    it with coalesced 16-byte stores, after which the slot is refilled.
// Every tile, the first ring-full of a CTA included, is drawn from one atomic ticket counter:
// a tile is only ever owned by a CTA that is already running, so a look-back never waits for a
// CTA that has not been scheduled (whatever else occupies the GPU), and the tiles in flight
// are neighbours in the look-back chain.
// ---------------------------------------------------------------------------------------
constexpr int kStreamThreads = 512;  // compute threads; the CTA has one more warp
constexpr int kStreamWarps = kStreamThreads / kWarp;
constexpr int kStreamCta = kStreamThreads + kWarp;
// Per element size: 16-byte vectors per thread (tile = threads x vectors x 16 B) and the
// number of iterations a scanned tile stays parked waiting for its prefix. The ring has
// park + 2 slots. Measured best on B200: 40 KiB tiles parked for 3 iterations (4-byte
// types), 48 KiB tiles parked for 2 (8-byte types).
template <int ELEM_BYTES> struct StreamShape {
  static constexpr int kVecs = ELEM_BYTES == 4 ? 5 : 6;
  static constexpr int kPark = ELEM_BYTES == 4 ? 3 : 2;
  static constexpr int kStages = kPark + 2;
  static constexpr int kTileBytes = kStreamThreads * kVecs * 16;
};
constexpr unsigned kNoTile = 0xffffffffu;

template <typename T, bool EXCLUSIVE>
__global__ void __launch_bounds__(kStreamCta, 1)
scan_stream_kernel(const T* in, T* out, uint64_t n, T init, TempHeader* hdr, TileWords<Words<T>::W>* tiles,
                   unsigned num_tiles) {
  constexpr int VEC = 16 / sizeof(T);
  constexpr int K = StreamShape<sizeof(T)>::kVecs;
  constexpr int kStreamPark = StreamShape<sizeof(T)>::kPark;
  constexpr int kStreamTileBytes = StreamShape<sizeof(T)>::kTileBytes;
  constexpr int WARP_ITEMS = kWarp * K * VEC;
  constexpr int TILE = kStreamThreads * K * VEC;
  constexpr int S = StreamShape<sizeof(T)>::kStages;

  extern __shared__ __align__(128) unsigned char ring[];
  __shared__ __align__(8) unsigned long long s_full[S];    // bulk load of the slot has landed
  __shared__ __align__(8) unsigned long long s_handoff[S]; // slot's tile id and total are set
  __shared__ __align__(8) unsigned long long s_resolved[S];// slot's prefix is set
  __shared__ unsigned s_tile[S];      // tile loaded (or being loaded) into the slot
  __shared__ unsigned s_look_tile[S]; // tile handed to the look-back warp (kNoTile: stop)
  __shared__ T s_look_total[S];
  __shared__ T s_prefix[S];
  __shared__ T s_warp_total[kStreamWarps];

  const unsigned warp = threadIdx.x / kWarp;
  const unsigned lane = lane_id();
  int* status = &hdr->status;

  unsigned pending = 0;  // thread 0: the next tile of this CTA, already drawn
  auto start_load = [&](int slot, unsigned t) {
    s_tile[slot] = t;
    if (t < num_tiles && (uint64_t)(t + 1) * TILE <= n) {
      fence_proxy_async_smem();  // the slot was last touched by ordinary loads and stores
      mbar_expect_tx(&s_full[slot], kStreamTileBytes);
      bulk_load(ring + (size_t)slot * kStreamTileBytes, in + (uint64_t)t * TILE, kStreamTileBytes, &s_full[slot]);
    }
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_handoff[s], 1);
      mbar_init(&s_resolved[s], 1);
    }
    mbar_init_fence();
    // Ticket after ticket, each drawn when the one before has arrived: drawn in one burst, a CTA's first tiles would be
    // neighbours, every other CTA's first tile would wait for all of them, and few CTAs would share a short input
    // (10 M floats 43 -> 25 us, 2^28 floats 409 -> 388 us).
#pragma unroll
    for (int s = 0; s < S; ++s) start_load(s, atomicAdd(&hdr->ticket, 1u));
    pending = atomicAdd(&hdr->ticket, 1u);
  }
  __syncthreads();

  // ------------------------------------------------------------------ look-back warp
  if (warp == kStreamWarps) {
    for (unsigned j = 0;; ++j) {
      const int slot = j % S;
      if (!mbar_wait_bounded(&s_handoff[slot], (j / S) & 1u, status)) break;
      const unsigned tile = s_look_tile[slot];
      if (tile == kNoTile) break;
      const T total = s_look_total[slot];
      typename Link<T>::Sum prefix = init;  // the seed: in front of the first element in both forms
      if (tile != 0) prefix = lookback_sum<T>(tiles, tile, status);
      if (lane == 0) {
        Link<T>::publish(&tiles[tile], kStatePrefix, Link<T>::settle(prefix + total));
        s_prefix[slot] = (T)prefix;
        mbar_arrive(&s_resolved[slot]);
      }
      __syncwarp();
    }
    return;
  }

  // ------------------------------------------------------------------ compute warps
  // adds the resolved prefix to the values parked in `slot` and stores the tile
  auto finalize = [&](unsigned it_prev, bool refill) {
    const int slot = it_prev % S;
    const unsigned tile = s_tile[slot];
    mbar_wait_bounded(&s_resolved[slot], (it_prev / S) & 1u, status);
    const T prefix = s_prefix[slot];
    const uint64_t warp_base = (uint64_t)tile * TILE + (uint64_t)warp * WARP_ITEMS;
    const Vec16<T>* parked = reinterpret_cast<const Vec16<T>*>(ring + (size_t)slot * kStreamTileBytes) +
                             warp * (kWarp * K);
    if ((uint64_t)(tile + 1) * TILE <= n) {
      Vec16<T>* dst = reinterpret_cast<Vec16<T>*>(out + warp_base);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        Vec16<T> v = parked[k * kWarp + lane];
#pragma unroll
        for (int j = 0; j < VEC; ++j) v.v[j] = prefix + v.v[j];
        dst[k * kWarp + lane] = v;
      }
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const Vec16<T> v = parked[k * kWarp + lane];
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
          const uint64_t i = warp_base + (uint64_t)(k * kWarp + lane) * VEC + j;
          if (i < n) out[i] = prefix + v.v[j];
        }
      }
    }
    if (refill) {
      named_barrier(1, kStreamThreads);  // the slot has been read by every compute thread
      if (threadIdx.x == 0) {
        start_load(slot, pending);
        pending = atomicAdd(&hdr->ticket, 1u);
      }
    }
  };

  unsigned it = 0;
  for (;; ++it) {
    const int slot = it % S;
    const unsigned tile = s_tile[slot];
    if (tile >= num_tiles) break;  // tickets only grow: no load of this CTA is still in flight
    const uint64_t tile_base = (uint64_t)tile * TILE;
    const bool full = tile_base + TILE <= n;
    // blocked layout for the local scan: thread t owns vectors [t*K, (t+1)*K) of the tile,
    // so one warp scan per tile suffices (the parked tile is re-read lane-strided later)
    Vec16<T>* mine = reinterpret_cast<Vec16<T>*>(ring + (size_t)slot * kStreamTileBytes) + threadIdx.x * K;

    T x[K][VEC];
    if (full) {
      mbar_wait_bounded(&s_full[slot], (it / S) & 1u, status);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const Vec16<T> v = mine[k];
#pragma unroll
        for (int j = 0; j < VEC; ++j) x[k][j] = v.v[j];
      }
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
          const uint64_t i = tile_base + (uint64_t)(threadIdx.x * K + k) * VEC + j;
          x[k][j] = i < n ? in[i] : T(0);
        }
    }

    // sequential inclusive scan of the thread's K*VEC elements, then one scan across lanes
    T run = T(0);
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        run = (k == 0 && j == 0) ? x[0][0] : run + x[k][j];
        x[k][j] = run;
      }
    T s = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      T t = __shfl_up_sync(0xffffffffu, s, off);
      if (lane >= off) s = t + s;
    }
    T lane_excl = __shfl_up_sync(0xffffffffu, s, 1);
    if (lane == 0) lane_excl = T(0);
    if (lane == 31) s_warp_total[warp] = s;
    named_barrier(1, kStreamThreads);

    T warp_prefix = T(0), tile_total = T(0);
#pragma unroll
    for (int w = 0; w < kStreamWarps; ++w) {
      const T t = s_warp_total[w];
      if (w < (int)warp) warp_prefix = warp_prefix + t;
      tile_total = tile_total + t;
    }
    if (threadIdx.x == 0) {
      if (tile != 0) Link<T>::publish(&tiles[tile], kStateAggregate, tile_total);
      s_look_tile[slot] = tile;
      s_look_total[slot] = tile_total;
      mbar_arrive(&s_handoff[slot]);
    }
    // park the locally resolved values in the tile's own slot
    {
      const T p = warp_prefix + lane_excl;
      T before = p;  // exclusive form: value in front of the element
#pragma unroll
      for (int k = 0; k < K; ++k) {
        Vec16<T> v;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
          const T incl = p + x[k][j];
          v.v[j] = EXCLUSIVE ? before : incl;
          before = incl;
        }
        mine[k] = v;
      }
    }
    // the barrier inside finalize (or this one) also orders this tile's parking stores
    // before other threads read them when the tile is finalized kStreamPark iterations on
    if (it >= (unsigned)kStreamPark) finalize(it - kStreamPark, true);
    else named_barrier(1, kStreamThreads);
  }
  // tiles of this CTA that are still parked
  named_barrier(1, kStreamThreads);
#pragma unroll
  for (int p = kStreamPark; p >= 1; --p)
    if (it >= (unsigned)p) finalize(it - p, false);
  if (threadIdx.x == 0) {  // release the look-back warp
    const int slot = it % S;
    s_look_tile[slot] = kNoTile;
    mbar_arrive(&s_handoff[slot]);
  }
}

template <typename T, bool EXCLUSIVE, int K, bool CLUSTER> struct WaveTag {};
template <typename T, bool EXCLUSIVE> struct StreamTag {};

template <int K, typename T>
constexpr uint64_t wave_tile() { return (uint64_t)kScanThreads * K * (16 / sizeof(T)); }

constexpr int kNoCluster = -1000;  // the GPU (or the part of it this process has) holds no cluster of that size

// One launch, one tile per CTA: at most kClusterTiles tiles in one cluster, or as many as the GPU holds at once.
template <typename T, bool EXCLUSIVE, int K, bool CLUSTER>
int launch_wave(const T* in, T* out, uint64_t n, T init, TempHeader* hdr, TileWords<Words<T>::W>* desc, int aligned,
                cudaStream_t stream) {
  auto kernel = scan_wave_kernel<T, EXCLUSIVE, K, CLUSTER>;
  const unsigned tiles = (unsigned)((n + wave_tile<K, T>() - 1) / wave_tile<K, T>());
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles);
  cfg.blockDim = dim3(kScanThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  if constexpr (CLUSTER) {
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = tiles;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (tiles > 8) {
      // More than eight CTAs per cluster are an opt-in, and need room for all of them in one part of the GPU: asked
      // once per device (benign race: the answer is always the same).
      static signed char answer[64] = {};  // 0: not asked, 1: fits, -1: does not
      int dev = 0;
      TB200_CUDA_TRY(cudaGetDevice(&dev));
      signed char fits = dev < 64 ? answer[dev] : 0;
      if (fits == 0) {
        TB200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t largest = cfg;
        largest.gridDim = dim3(kClusterTiles);
        cudaLaunchAttribute of = attr;
        of.val.clusterDim.x = kClusterTiles;
        largest.attrs = &of;
        int clusters = 0;
        fits = cudaOccupancyMaxActiveClusters(&clusters, kernel, &largest) == cudaSuccess && clusters > 0 ? 1 : -1;
        (void)cudaGetLastError();
        if (dev < 64) answer[dev] = fits;
      }
      if (fits < 0) return kNoCluster;
    }
  }
  TB200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, in, out, n, init, hdr, desc, aligned));
  trace_mark(stream, kTraceScan);
  return TB200_OK;
}

template <typename T>
int launch_scan(void* d_temp, size_t* temp_bytes, const void* d_in, void* d_out, uint64_t n,
                int exclusive, const void* h_init, cudaStream_t stream) {
  constexpr int W = Words<T>::W;
  constexpr uint64_t TILE = (uint64_t)kScanThreads * kScanVecs * (16 / sizeof(T));
  constexpr uint64_t STREAM_TILE = (uint64_t)kStreamThreads * StreamShape<sizeof(T)>::kVecs * (16 / sizeof(T));
  const uint64_t tiles = (n + TILE - 1) / TILE;
  const uint64_t stream_tiles = (n + STREAM_TILE - 1) / STREAM_TILE;  // the smaller tile sizes the scratch
  const size_t need = kHeaderBytes + (size_t)stream_tiles * sizeof(TileWords<W>);
  // inputs of one wave of CTAs may take smaller tiles, if the scratch has room for their descriptors
  const uint64_t small_tiles = (n + wave_tile<4, T>() - 1) / wave_tile<4, T>();
  const size_t small_need = kHeaderBytes + (size_t)small_tiles * sizeof(TileWords<W>);
  if (d_temp == nullptr) {
    *temp_bytes = small_tiles <= (uint64_t)kScanThreads && small_need > need ? small_need : need;
    return TB200_OK;
  }
  if (*temp_bytes < need) return TB200_ERR_TEMP_TOO_SMALL;
  if (reinterpret_cast<uintptr_t>(d_temp) % 256) return TB200_ERR_INVALID_ARGUMENT;
  if (stream_tiles > 0x7fffffffull) return TB200_ERR_UNSUPPORTED;
  // One cluster serves up to 1 MiB of input and needs no cleared scratch.
  const bool cluster = n != 0 && n <= kClusterTiles * wave_tile<8, T>();
  int sms = 0;
  {
    const int rc = sm_count_of_device(&sms);
    if (rc) return rc;
  }
  // One wave: as many tiles as the GPU holds CTAs of that kernel (19 MiB of input on 148 SMs in 64 KiB tiles).
  const uint64_t resident = (uint64_t)sms * kScanMinCtas < kScanThreads ? (uint64_t)sms * kScanMinCtas : kScanThreads;
  const bool wave_small = small_tiles <= resident && *temp_bytes >= small_need;
  const bool wave_large = n <= resident * wave_tile<8, T>();
  if (n != 0 && (d_in == nullptr || d_out == nullptr)) return TB200_ERR_INVALID_ARGUMENT;

  T init = T(0);
  if (h_init) init = *static_cast<const T*>(h_init);
  auto* hdr = static_cast<TempHeader*>(d_temp);
  auto* desc = reinterpret_cast<TileWords<W>*>(static_cast<char*>(d_temp) + kHeaderBytes);
  const T* in = static_cast<const T*>(d_in);
  T* out = static_cast<T*>(d_out);
  const bool aligned = ((reinterpret_cast<uintptr_t>(d_in) | reinterpret_cast<uintptr_t>(d_out)) % 16) == 0;
  auto wave = [&](auto k, auto in_cluster) -> int {
    constexpr int K = decltype(k)::value;
    constexpr bool C = decltype(in_cluster)::value;
    return exclusive ? launch_wave<T, true, K, C>(in, out, n, init, hdr, desc, aligned, stream)
                     : launch_wave<T, false, K, C>(in, out, n, init, hdr, desc, aligned, stream);
  };
  if (cluster) {
    const int rc = n <= kClusterTiles * wave_tile<2, T>() ? wave(std::integral_constant<int, 2>{}, std::true_type{})
                                                          : wave(std::integral_constant<int, 8>{}, std::true_type{});
    if (rc != kNoCluster) return rc;
  }
  TB200_CUDA_TRY(cudaMemsetAsync(d_temp, 0, wave_small ? small_need : need, stream));
  if (n == 0) return TB200_OK;
  if (wave_small) return wave(std::integral_constant<int, 4>{}, std::false_type{});
  if (wave_large) return wave(std::integral_constant<int, 8>{}, std::false_type{});
  if (aligned) {
    constexpr int smem = StreamShape<sizeof(T)>::kStages * StreamShape<sizeof(T)>::kTileBytes;
    auto run = [&](auto kernel, auto tag) -> int {
      int per_sm = 0;
      const int rc = resident_ctas<decltype(tag)>(kernel, kStreamCta, smem, &per_sm);
      if (rc) return rc;
      // one CTA per slot of the GPU: more would only queue behind them
      const uint64_t slots = (uint64_t)sms * per_sm;
      const unsigned grid = (unsigned)(stream_tiles < slots ? stream_tiles : slots);
      kernel<<<grid, kStreamCta, smem, stream>>>(in, out, n, init, hdr, desc, (unsigned)stream_tiles);
      return TB200_OK;
    };
    const int rc = exclusive ? run(scan_stream_kernel<T, true>, StreamTag<T, true>{})
                             : run(scan_stream_kernel<T, false>, StreamTag<T, false>{});
    if (rc) return rc;
    trace_mark(stream, kTraceScan);
    return (int)cudaGetLastError();
  }
  const dim3 grid((unsigned)tiles), block(kScanThreads);
  if (exclusive) scan_kernel<T, true><<<grid, block, 0, stream>>>(in, out, n, init, hdr, desc);
  else           scan_kernel<T, false><<<grid, block, 0, stream>>>(in, out, n, init, hdr, desc);
  trace_mark(stream, kTraceScan);
  return (int)cudaGetLastError();
}

}  // namespace
}  // namespace tb200

extern "C" int tb200_scan(void* d_temp, size_t* temp_bytes, const void* d_in, void* d_out, uint64_t n,
                          int dtype, int exclusive, const void* h_init, tb200_stream_t stream) {
  using namespace tb200;
  if (temp_bytes == nullptr) return TB200_ERR_INVALID_ARGUMENT;
  switch (dtype) {
    // signed integers wrap like unsigned ones in two's complement
    case TB200_I32: case TB200_U32:
      return launch_scan<uint32_t>(d_temp, temp_bytes, d_in, d_out, n, exclusive, h_init, stream);
    case TB200_I64: case TB200_U64:
      return launch_scan<unsigned long long>(d_temp, temp_bytes, d_in, d_out, n, exclusive, h_init, stream);
    case TB200_F32:
      return launch_scan<float>(d_temp, temp_bytes, d_in, d_out, n, exclusive, h_init, stream);
    case TB200_F64:
      return launch_scan<double>(d_temp, temp_bytes, d_in, d_out, n, exclusive, h_init, stream);
    default:
      return TB200_ERR_UNSUPPORTED;
  }
}

// ---------------------------------------------------------------------------------------
// tb200_scan_static: the same scan, with its scratch in a fixed device array
// ---------------------------------------------------------------------------------------
namespace tb200 {
namespace {

// Look-back descriptors of tb200_scan_static. Lives in every GPU that loads this library,
// from load until the process exits. The size is whatever the streaming kernel's tiles need
// at the documented limits (checked below), rounded up to 2 MiB.
constexpr uint64_t kStaticScanMaxN4 = 1ull << 31;  // 4-byte element types
constexpr uint64_t kStaticScanMaxN8 = 1ull << 29;  // 8-byte element types
constexpr size_t kStaticScanBytes = kHeaderBytes + (2u << 20);
template <int ELEM_BYTES>
constexpr size_t static_scan_need(uint64_t n) {
  constexpr uint64_t tile = (uint64_t)kStreamThreads * StreamShape<ELEM_BYTES>::kVecs * (16 / ELEM_BYTES);
  return kHeaderBytes + (size_t)((n + tile - 1) / tile) * sizeof(TileWords<ELEM_BYTES / 4>);
}
static_assert(static_scan_need<4>(kStaticScanMaxN4) <= kStaticScanBytes, "static scratch too small for 2^31 4-byte elements");
static_assert(static_scan_need<8>(kStaticScanMaxN8) <= kStaticScanBytes, "static scratch too small for 2^29 8-byte elements");
static __device__ __align__(256) unsigned char g_static_scan_scratch[kStaticScanBytes];

constexpr int kMaxDevices = 64;
std::mutex g_static_scan_mutex;
void* g_static_scan_ptr[kMaxDevices] = {};

// In host code `g_static_scan_scratch` is only a handle for the runtime, not an address a
// kernel can use; the device address is looked up once per device, with that device current.
int static_scan_scratch(void** out) {
  int dev = 0;
  TB200_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return TB200_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_static_scan_mutex);
  if (g_static_scan_ptr[dev] == nullptr) {
    void* p = nullptr;
    TB200_CUDA_TRY(cudaGetSymbolAddress(&p, g_static_scan_scratch));
    g_static_scan_ptr[dev] = p;
  }
  *out = g_static_scan_ptr[dev];
  return TB200_OK;
}

}  // namespace
}  // namespace tb200

extern "C" int tb200_scan_static(const void* d_in, void* d_out, uint64_t n, int dtype, int exclusive,
                                 const void* h_init, tb200_stream_t stream) {
  using namespace tb200;
  const int eb = dtype_bytes(dtype);
  if (eb != 4 && eb != 8) return TB200_ERR_UNSUPPORTED;
  // the documented limits, checked before anything touches the device
  if (n > (eb == 4 ? kStaticScanMaxN4 : kStaticScanMaxN8)) return TB200_ERR_OVERFLOW;
  size_t need = 0;
  int rc = tb200_scan(nullptr, &need, nullptr, nullptr, n, dtype, exclusive, h_init, stream);
  if (rc) return rc;
  if (need > kStaticScanBytes) return TB200_ERR_OVERFLOW;  // cannot happen inside the limits (static_assert above)
  void* scratch = nullptr;
  rc = static_scan_scratch(&scratch);
  if (rc) return rc;
  size_t have = kStaticScanBytes;
  // tb200_scan clears the part of the scratch that its kernel reads on `stream` (header and descriptors; a scan by one
  // cluster reads none and sets the status word itself), so what the previous call left behind is never read.
  return tb200_scan(scratch, &have, d_in, d_out, n, dtype, exclusive, h_init, stream);
}

extern "C" int tb200_scan_static_status(tb200_stream_t stream) {
  using namespace tb200;
  void* scratch = nullptr;
  const int rc = static_scan_scratch(&scratch);
  if (rc) return rc;
  return tb200_temp_status(scratch, stream);
}
