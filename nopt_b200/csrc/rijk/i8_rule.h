// i8_rule.h — which FP64 exchanges run on the int8 tensor cores (plain host arithmetic).
#pragma once

namespace rijk {

// Terms of one sum of digit products: of up to 7 pairs of digits, each product at most 2^14 in magnitude, and
// 7 2^14 18720 < 2^31 - 1, so every s32 sum is exact.
constexpr long kMaxDigitSum = 18720;

// From about 1e10 FLOPs of exchange and more than 192 functions on (128-row blocks).  Whole FP64 builds, DMMA
// against int8: 278 against 294 us at n = 192, n_c = 40; 233 against 246 at 232, 20; 580 against 564 at 348, 30; 534
// against 449 at 250, 41; 628 against 457 at 240, 50; 2.30 against 1.56 ms at 384, 80; 80.3 against 33.6 ms at 970, 161.
inline bool int8_exchange(long npad, long kdim) { return npad > 192 && 3.0 * npad * npad * kdim >= 1e10; }

// Its half-transform, too: the contraction over all n functions is one sum, and the parts of K of kper k, whose row
// maxima it keeps, must be whole aux functions.
inline bool int8_half_transform(long n, long npad, long kdim, long noccp, long kper) {
  return int8_exchange(npad, kdim) && n <= kMaxDigitSum && kper % noccp == 0;
}

}  // namespace rijk
