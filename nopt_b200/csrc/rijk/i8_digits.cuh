// i8_digits.cuh — FP64 values as seven balanced byte digits, and the sums of their exact products back in
// FP64 (see k_exchange_i8.cu for the scheme and its error), shared by the half-transform and K.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "tc_util.cuh"

namespace rijk {

constexpr int kDigits = 7;                     // byte digits of a value
constexpr int kGroups = 8;                     // groups s + t kept
constexpr int kChunk = 32;                     // k per stage and per MMA
constexpr uint32_t kDigitA = 128 * kChunk;     // one digit of a 128-row panel: 4 KB
constexpr uint32_t kBlockBytes = kDigits * kDigitA;  // 28 KB
constexpr int kNonFinite = 1 << 20;            // exponent of values with an infinity or NaN among them

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}

// 2^e exactly for |e| <= 1000 (the exponent bits), else through ldexp.
__device__ __forceinline__ double pow2i(int e) {
  return (e >= -1000 && e <= 1000) ? __longlong_as_double(static_cast<long long>(e + 1023) << 52) : ldexp(1.0, e);
}

// Magnitudes are compared by the leading words of their bit patterns: these order as the magnitudes do,
// infinities and NaN above all finite ones.
__device__ __forceinline__ uint32_t magnitude(double x) {
  return static_cast<uint32_t>(__double2hiint(x)) & 0x7fffffffu;
}

// The exponent x of values whose largest magnitude has the leading word `top`: max / 2^x <= 127.49 2^48.
__device__ __forceinline__ int value_exponent(uint32_t top) {
  if (top >= 0x7ff00000u) return kNonFinite;
  const double m = __hiloint2double(static_cast<int>(top), -1);  // at least the largest magnitude
  const int e = ilogb(m) + 1;                                    // m < 2^e
  return (ldexp(m, -e) <= 0.995 ? e : e + 1) - 55;
}

// 2^(x + 55) of an exponent x, about twice the largest magnitude; NaN when a value was not finite.  A product
// of two joined sums (join8) is its value times 2^-38 times both operands' scales.
__device__ __forceinline__ double value_scale(int x) {
  return x == kNonFinite ? __longlong_as_double(0x7ff8000000000000ll) : pow2i(x + 55);
}
constexpr double kJoined = 1.0 / 274877906944.0;  // 2^-38

// 16 values of one row as 16 bytes of each digit, digit 0 the leading one.
__device__ __forceinline__ void digits16(const double (&x)[16], int ex, uint4 (&d)[kDigits]) {
  uint32_t* out = reinterpret_cast<uint32_t*>(d);
  const bool plain = ex > -1000 && ex < 1000;
  const double f = plain ? pow2i(-ex) : 0.0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double y = plain ? x[4 * q + j] * f : ldexp(x[4 * q + j], -ex);
      const unsigned long long u =
          (static_cast<unsigned long long>(__double2ll_rn(y)) + 0x0080808080808080ull) ^ 0x0080808080808080ull;
      lo[j] = static_cast<uint32_t>(u);
      hi[j] = static_cast<uint32_t>(u >> 32);
    }
    // byte b of the four words, b = 0 .. 3 (of lo: digits 6 .. 3; of hi: digits 2 .. 0)
    const uint32_t l01 = __byte_perm(lo[0], lo[1], 0x5140), l23 = __byte_perm(lo[2], lo[3], 0x5140);
    const uint32_t m01 = __byte_perm(lo[0], lo[1], 0x7362), m23 = __byte_perm(lo[2], lo[3], 0x7362);
    const uint32_t h01 = __byte_perm(hi[0], hi[1], 0x5140), h23 = __byte_perm(hi[2], hi[3], 0x5140);
    const uint32_t n01 = __byte_perm(hi[0], hi[1], 0x7362), n23 = __byte_perm(hi[2], hi[3], 0x7362);
    out[6 * 4 + q] = __byte_perm(l01, l23, 0x5410);
    out[5 * 4 + q] = __byte_perm(l01, l23, 0x7632);
    out[4 * 4 + q] = __byte_perm(m01, m23, 0x5410);
    out[3 * 4 + q] = __byte_perm(m01, m23, 0x7632);
    out[2 * 4 + q] = __byte_perm(h01, h23, 0x5410);
    out[1 * 4 + q] = __byte_perm(h01, h23, 0x7632);
    out[0 * 4 + q] = __byte_perm(n01, n23, 0x5410);
  }
}

// sum_{g<4} v_g 256^(3-g) in one 64-bit integer (|v_g| < 2^31, so below 2^56)
__device__ __forceinline__ long long join4(uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3) {
  return static_cast<long long>(static_cast<int32_t>(v0)) * 16777216 +
         (static_cast<long long>(static_cast<int32_t>(v1)) * 65536 +
          (static_cast<long long>(static_cast<int32_t>(v2)) * 256 + static_cast<int32_t>(v3)));
}
// groups 0 - 3 joined in hi, 4 - 7 in lo: sum_g v_g 256^(3-g)
__device__ __forceinline__ double join8(long long hi, long long lo) {
  return fma(static_cast<double>(lo), 1.0 / 4294967296.0, static_cast<double>(hi));
}

// One chunk's MMAs: digit s of A (rows of a 128-row panel, digits kDigitA apart at sa) against digits
// 0 .. min(6, 7 - s) of B (NB rows a digit, side by side at sb), group s + t in the NB columns from
// NB (s + t).  The chunk that starts the sums (first) overwrites each group on its first product: digit s = 0
// starts groups 0 - 6, and (1, 6) starts group 7.  A_BITS, A_MN: A's descriptor bits and major-ness.  All of it
// is straight-line code: one thread issues an MMA about every 100 clocks, and with NB a run-time number its loops
// could not keep up (K of C40H82 9.3 instead of 7.7 ms).
template <int NB, uint64_t A_BITS, bool A_MN>
__device__ __forceinline__ void issue_digit_products(uint32_t tmem, uint32_t sa, uint32_t sb, bool first) {
  constexpr uint64_t kB = plain_desc_bits(128, 256);  // core matrices 128 B apart along k, 256 B along rows
  constexpr uint32_t mn = A_MN ? (1u << 15) : 0u;
  constexpr int per = 256 / NB;  // digits of B in one MMA
#pragma unroll
  for (int s = 0; s < kDigits; ++s) {
    const uint64_t da = sw128_desc(sa + s * kDigitA, A_BITS);
    const int n = kGroups - s < kDigits ? kGroups - s : kDigits;
    if (s == 1 && first) {  // its last digit is group 7's first product
#pragma unroll
      for (int t = 0; t < n - 1; t += per) {
        const int m = per < n - 1 - t ? per : n - 1 - t;
        umma_s8(tmem + (s + t) * NB, da, sw128_desc(sb + t * NB * kChunk, kB), idesc_s8_s32(128, NB * m) | mn, 1u);
      }
      umma_s8(tmem + (kGroups - 1) * NB, da, sw128_desc(sb + (kDigits - 1) * NB * kChunk, kB), idesc_s8_s32(128, NB) | mn, 0u);
      continue;
    }
#pragma unroll
    for (int t = 0; t < n; t += per) {
      const int m = per < n - t ? per : n - t;
      umma_s8(tmem + (s + t) * NB, da, sw128_desc(sb + t * NB * kChunk, kB), idesc_s8_s32(128, NB * m) | mn,
              (first && s == 0) ? 0u : 1u);
    }
  }
}

}  // namespace rijk
