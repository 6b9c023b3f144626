// The shared-memory sort in each of its launch shapes, without the sizes that lead to them (the largest tile shape is
// used above 570 million elements only).
//   test_tile_sort places   on the CPU: the places that the padding behind m elements takes, for every shape and every m
//   test_tile_sort sort     on the GPU: tiles of every kind of size, small ones first, against std::stable_sort
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <random>
#include <vector>

#include "../../thrust_b200/csrc/block_sort_impl.cuh"
#include "../../thrust_b200/csrc/bucket_sort.cuh"

namespace tb200 {
namespace {

// ---- places of the padding ---------------------------------------------------------------------
// Replays steps 2 and 3 of the sort for the padding alone: the rank of an element is what its bin counted before it,
// its place the elements in front of its word and of its counter, and its rank. m real elements lie in front of all.
template <int THREADS, int ITEMS, int BINS>
bool places_ok(const char* name) {
  using B = BlockSort<uint32_t, 4, THREADS, ITEMS, BINS>;
  constexpr unsigned cap = B::kCap;
  std::vector<unsigned> count(B::kPadBins), before(B::kPadBins / 4);
  std::vector<unsigned char> taken(cap);
  for (unsigned m = 1; m <= cap; ++m) {
    std::fill(count.begin(), count.end(), 0u);
    auto each = [&](auto f) {  // thread t holds elements t / 32 * 32 * ITEMS + 32 j + t % 32
      for (unsigned i = m; i < cap; ++i) f(B::pad_bin(i / (kWarp * ITEMS) * kWarp + i % kWarp) - BINS);
    };
    each([&](unsigned bin) { ++count[bin]; });
    std::vector<unsigned> word(B::kPadBins / 4, 0u);
    unsigned sum = m;
    for (unsigned w = 0; w < word.size(); ++w) {
      before[w] = sum;
      for (unsigned b = 0; b < 4; ++b) {
        if (count[4 * w + b] > 255) { std::printf("FAILED %s m=%u: counter\n", name, m); return false; }
        word[w] |= count[4 * w + b] << (8 * b);
        sum += count[4 * w + b];
      }
    }
    std::fill(count.begin(), count.end(), 0u);
    std::memset(taken.data(), 0, cap);
    unsigned wrong = 0;
    each([&](unsigned bin) {
      const unsigned place = before[bin / 4] + B::in_front(word[bin / 4], bin % 4) + count[bin]++;
      if (place < m || place >= cap || taken[place]) ++wrong;
      else taken[place] = 1;
    });
    if (wrong || sum != cap) {
      std::printf("FAILED %s m=%u: %u padding elements without a place of their own\n", name, m, wrong);
      return false;
    }
  }
  return true;
}

// ---- tiles on the GPU --------------------------------------------------------------------------
template <typename UK, int VB, int THREADS, int ITEMS, int BINS, int MIN_CTAS>
__global__ void __launch_bounds__(THREADS, MIN_CTAS)
tiles_kernel(const UK* src_keys, const typename ValueOf<VB>::type* src_vals, UK* keys, typename ValueOf<VB>::type* vals,
             const unsigned* begin, unsigned tiles, int shift, Encoding enc) {
  using B = BlockSort<UK, VB, THREADS, ITEMS, BINS>;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned s_red[B::kRedWords];
  for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
    const unsigned at = begin[t], m = begin[t + 1] - at;
    if (m == 0) continue;
    B::template sort<false>(src_keys + at, VB ? src_vals + at : nullptr, keys + at, VB ? vals + at : nullptr, m, shift, enc,
                            smem, s_red);
    __syncthreads();
  }
}

template <typename T>
struct Device {
  T* ptr = nullptr;
  explicit Device(const std::vector<T>& h) {
    if (cudaMalloc(&ptr, h.size() * sizeof(T) + 16) != cudaSuccess) std::abort();
    if (cudaMemcpy(ptr, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) std::abort();
  }
  ~Device() { cudaFree(ptr); }
};

template <typename UK, int VB, int SIZE>
bool tiles_ok(const char* name) {
  using S = TileShape<SIZE>;
  using B = BlockSort<UK, VB, S::kThreads, S::kItems, S::kBins>;
  using V = typename B::V;
  constexpr unsigned cap = B::kCap;
  std::mt19937_64 rng(SIZE + 10 * VB);
  // first the small tiles: they meet whatever the shared memory held before
  std::vector<unsigned> sizes = {1, 2, 600, 3000, 31, 33, 6499, 6500, 6526, 6527, cap / 2, cap - 1, cap, 0, 1, cap / 3, cap, 5};
  for (int i = 0; i < 60; ++i) sizes.push_back((unsigned)(rng() % (cap + 1)));
  for (unsigned& m : sizes) m = std::min(m, cap);
  std::vector<unsigned> begin(1, 0u);
  for (unsigned m : sizes) begin.push_back(begin.back() + m);
  const unsigned n = begin.back(), guard = 64;
  // What all keys of a tile share lies above `bits`; the keys are encoded already (descending signed keys).
  for (int bits : {8 * (int)sizeof(UK), 8 * (int)sizeof(UK) - 16}) {
    const Encoding enc = make_encoding(sizeof(UK), 1, 1);
    std::vector<UK> k(n);
    std::vector<V> v(n + 1);
    for (size_t t = 0; t < sizes.size(); ++t) {
      const UK high = bits < 8 * (int)sizeof(UK) ? (UK)((UK)t << bits) : (UK)0;
      const UK mask = bits < 8 * (int)sizeof(UK) ? (UK)(((UK)1 << bits) - 1) : (UK)~(UK)0;
      for (unsigned i = begin[t]; i < begin[t + 1]; ++i) {
        const UK r = (UK)rng();
        const UK step = mask / 3 / (UK)(sizes[t] + 1) + 1;
        UK x = r;
        switch (t % 7) {
          case 2: x = (UK)(r % (mask / 3 * 2)); break;                         // a range that is no power of two
          case 3: x = (UK)(r % 37) << (bits - 8); break;                       // many copies: counters overflow
          case 4: x = (UK)(r % (sizes[t] / 5 + 1)) * step; break;              // five copies of every key
          case 5: x = (UK)(r % (sizes[t] / 30 + 1)) * (30 * step); break;      // thirty
          case 6: x = (UK)(r % (sizes[t] / 40 + 1)) * (40 * step) + (UK)(rng() % 3); break;  // three keys to a bin
        }
        k[i] = high | (x & mask);
      }
    }
    for (unsigned i = 0; i < n; ++i) {
      unsigned char bytes[16] = {};
      std::memcpy(bytes, &i, sizeof(i));
      std::memcpy(&v[i], bytes, VB ? sizeof(V) : 0);
    }
    Device<UK> src_k(k);
    Device<V> src_v(v);
    std::vector<UK> out_k(n + 2 * guard, (UK)0x5a);
    std::vector<V> out_v(n + 2 * guard);
    std::memset(out_v.data(), 0x5a, out_v.size() * sizeof(V));
    Device<UK> dst_k(out_k);
    Device<V> dst_v(out_v);
    Device<unsigned> d_begin(begin);
    auto kernel = tiles_kernel<UK, VB, S::kThreads, S::kItems, S::kBins, S::kMinCtas>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B::kSmem);
    if (err == cudaSuccess) {
      kernel<<<7, S::kThreads, B::kSmem>>>(src_k.ptr, src_v.ptr, dst_k.ptr + guard, dst_v.ptr + guard, d_begin.ptr,
                                           (unsigned)sizes.size(), std::max(0, bits - 32), enc);
      err = cudaDeviceSynchronize();
    }
    if (err != cudaSuccess) { std::printf("FAILED %s: %s\n", name, cudaGetErrorString(err)); return false; }
    cudaMemcpy(out_k.data(), dst_k.ptr, out_k.size() * sizeof(UK), cudaMemcpyDeviceToHost);
    cudaMemcpy(out_v.data(), dst_v.ptr, out_v.size() * sizeof(V), cudaMemcpyDeviceToHost);
    auto decoded = [](UK x) { return (UK)(~x ^ ((UK)1 << (8 * sizeof(UK) - 1))); };
    for (size_t t = 0; t < sizes.size(); ++t) {
      std::vector<unsigned> order(sizes[t]);
      std::iota(order.begin(), order.end(), begin[t]);
      std::stable_sort(order.begin(), order.end(), [&](unsigned a, unsigned b) { return k[a] < k[b]; });
      for (unsigned i = 0; i < sizes[t]; ++i) {
        const unsigned at = guard + begin[t] + i;
        if (out_k[at] != decoded(k[order[i]]) || (VB && std::memcmp(&out_v[at], &v[order[i]], sizeof(V)))) {
          std::printf("FAILED %s bits=%d tile %zu (%u elements) at %u\n", name, bits, t, sizes[t], i);
          return false;
        }
      }
    }
    for (unsigned i = 0; i < guard; ++i)
      if (out_k[i] != (UK)0x5a || out_k[guard + n + i] != (UK)0x5a) { std::printf("FAILED %s: guard\n", name); return false; }
  }
  return true;
}

template <typename UK, int VB>
bool all_tiles(const char* name) {
  bool ok = tiles_ok<UK, VB, 0>(name) && tiles_ok<UK, VB, 1>(name);
  if constexpr (VB <= 8) ok = ok && tiles_ok<UK, VB, 2>(name);
  return ok;
}

template <int SIZE>
bool shape_places(const char* name) {
  return places_ok<TileShape<SIZE>::kThreads, TileShape<SIZE>::kItems, TileShape<SIZE>::kBins>(name);
}

}  // namespace
}  // namespace tb200

int main(int argc, char** argv) {
  using namespace tb200;
  bool ok = false;
  if (argc == 2 && !std::strcmp(argv[1], "places"))
    ok = places_ok<256, 4, 2048>("256 x 4") && places_ok<384, 12, 8192>("384 x 12") && shape_places<0>("512 x 9") &&
         shape_places<1>("1024 x 9") && shape_places<2>("1024 x 17");
  else if (argc == 2 && !std::strcmp(argv[1], "sort"))
    ok = all_tiles<uint32_t, 0>("u32") && all_tiles<uint32_t, 4>("u32, 4") && all_tiles<unsigned long long, 4>("u64, 4") &&
         all_tiles<unsigned long long, 8>("u64, 8") && all_tiles<uint32_t, 16>("u32, 16");
  if (ok) std::printf("PASSED\n");
  return ok ? 0 : 1;
}
