// What the kernels of the radix sort share: the control block in the caller's scratch, the key
// encoding, digit extraction, the warp match and the residency query.
#pragma once

#include "common.cuh"

#include <type_traits>

namespace tb200 {
namespace {

constexpr int kRadix = 256;
constexpr int kMaxPasses = 8;

struct SortCtl {
  int status;                    // must stay first: tb200_temp_status reads it
  unsigned hist_done;            // CTAs of the histogram kernel that have finished
  unsigned total_exec;           // number of passes that are not skipped
  unsigned last_pass;            // index of the last executed pass
  unsigned tickets[kMaxPasses];  // dynamic tile counters, one per pass
  unsigned skip[kMaxPasses];
  unsigned exec_before[kMaxPasses];  // executed passes before pass p (ping-pong parity)
  // Bucket plan (bucket_sort.cu). bucket_mode != 0: passes 0 and 1 take the digits below instead of bytes 0 and 1,
  // every later pass is skipped, and the tiles listed behind the plan are sorted in shared memory.
  unsigned bucket_mode;
  unsigned pass_shift[2], pass_mask[2];
  unsigned window_ok;            // the sample found a window that looks worth counting
  unsigned window_bits;          // keys differ below this bit only
  unsigned bucket_bits;          // the buckets are told apart by the top bucket_bits of the window
  unsigned joint_done;           // CTAs of the bucket count that have finished
  unsigned num_bucket_tiles;
  unsigned tile_bits;            // the keys of one tile differ below this bit only
  unsigned long long window_prefix;  // what all keys hold above the window
  unsigned long long hist[kMaxPasses][kRadix];
  unsigned long long offs[kMaxPasses][kRadix];
};

struct Encoding {
  unsigned long long cmask;  // constant xor (sign bit for signed and float keys)
  unsigned long long fmask;  // all ones for floating point, else 0
  unsigned long long dmask;  // all ones for descending, else 0
};

inline Encoding make_encoding(int key_bytes, int kind, int descending) {
  const unsigned long long sign = 1ull << (8 * key_bytes - 1);
  return Encoding{kind == 0 ? 0ull : sign, kind == 2 ? ~0ull : 0ull, descending ? ~0ull : 0ull};
}

template <typename UK>
__device__ __forceinline__ UK encode_key(UK x, const Encoding& e) {
  using SK = typename std::make_signed<UK>::type;
  const UK sra = (UK)((SK)x >> (8 * sizeof(UK) - 1));
  return x ^ (UK)((sra & (UK)e.fmask) | (UK)e.cmask) ^ (UK)e.dmask;
}
template <typename UK>
__device__ __forceinline__ UK decode_key(UK y, const Encoding& e) {
  using SK = typename std::make_signed<UK>::type;
  y ^= (UK)e.dmask;
  const UK sra = (UK)((SK)y >> (8 * sizeof(UK) - 1));
  return y ^ (UK)(((UK)~sra & (UK)e.fmask) | (UK)e.cmask);
}

// Digit of an encoded key. 64-bit keys: the 32-bit window that starts at bit `shift` is
// taken with one funnel shift (or from the high word alone), never a 64-bit shift.
template <typename UK>
__device__ __forceinline__ unsigned digit_of(UK k, int shift, unsigned mask) {
  if constexpr (sizeof(UK) == 8) {
    const unsigned lo = (unsigned)k, hi = (unsigned)(k >> 32);
    const unsigned w = shift < 32 ? __funnelshift_r(lo, hi, shift) : hi >> (shift - 32);
    return w & mask;
  } else {
    return ((unsigned)k >> shift) & mask;
  }
}

template <int BYTES> struct ValueOf;
template <> struct ValueOf<1> { using type = uint8_t; };
template <> struct ValueOf<2> { using type = uint16_t; };
template <> struct ValueOf<4> { using type = uint32_t; };
template <> struct ValueOf<8> { using type = unsigned long long; };
template <> struct ValueOf<16> { using type = uint4; };
template <> struct ValueOf<0> { using type = uint8_t; };  // unused

template <typename UK>
struct alignas(16) KeyVec {
  UK v[16 / sizeof(UK)];
};

template <int B>
__device__ __forceinline__ void match_bit(unsigned& peers, unsigned d) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b32 t, m, nm;\n"
      "and.b32 t, %1, %2;\n"
      "setp.ne.u32 p, t, 0;\n"
      "vote.sync.ballot.b32 m, p, 0xffffffff;\n"
      "not.b32 nm, m;\n"
      "@p and.b32 %0, %0, m;\n"
      "@!p and.b32 %0, %0, nm;\n"
      "}\n"
      : "+r"(peers)
      : "r"(d), "n"(1 << B));
}

// Lanes of the warp that hold the same 8-bit digit. One ballot per bit; a lane keeps
// the voters that agree with its own bit: peers &= ~(ballot ^ sign_extend(bit)).
__device__ __forceinline__ unsigned match_digit(unsigned d) {
  // four instructions per bit: test, vote, and one predicated AND for either polarity
  unsigned peers = 0xffffffffu;
  match_bit<0>(peers, d); match_bit<1>(peers, d); match_bit<2>(peers, d); match_bit<3>(peers, d);
  match_bit<4>(peers, d); match_bit<5>(peers, d); match_bit<6>(peers, d); match_bit<7>(peers, d);
  return peers;
}

// Copies `bytes` with the whole grid. The source is 256-byte aligned scratch; the destination is the caller's and is
// written byte by byte when it is not 16-byte aligned.
__device__ __forceinline__ void copy_back(uint4* __restrict__ dst, const uint4* __restrict__ src, uint64_t bytes) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nvec = (reinterpret_cast<uintptr_t>(dst) & 15) == 0 ? bytes / 16 : 0;
  uint64_t i = tid;
  for (; i + 3 * stride < nvec; i += 4 * stride) {  // four loads in flight per thread
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = src[i + u * stride];
#pragma unroll
    for (int u = 0; u < 4; ++u) dst[i + u * stride] = v[u];
  }
  for (; i < nvec; i += stride) dst[i] = src[i];
  unsigned char* d8 = reinterpret_cast<unsigned char*>(dst);
  const unsigned char* s8 = reinterpret_cast<const unsigned char*>(src);
  for (uint64_t b = nvec * 16 + tid; b < bytes; b += stride) d8[b] = s8[b];
}

}  // namespace
}  // namespace tb200
