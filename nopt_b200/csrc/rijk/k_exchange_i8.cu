// k_exchange_i8.cu — the exchange contraction K = X^T X of the FP64 form on tcgen05 tensor cores,
// with FP64 accuracy from exact int8 products (the Ozaki splitting scheme).
//
// tcgen05 has no FP64 kind.  Each row nu of X^T (the half-transformed tensor, k = Q n_c + i
// contiguous) is written, over the k range of one split-K part r, as the 56-bit integers
//     v = rint(X[nu][k] 2^-x(r,nu)),  |v| <= 127.49 2^48,   v = sum_{s=0}^{6} d_s 256^(6-s),
// with balanced byte digits d_s in [-128, 127] (k_slice_x: one conversion, one 64-bit add that propagates
// the carries, one exclusive or).  The rounding is at most 2^-55 of the row's maximum.  Then
//     K_mu,nu = 2^(x_mu + x_nu) sum_g 256^(12-g) sum_{s+t=g} (d_s[mu] . d_t[nu]),
// where every (d_s . d_t) is an exact s32 tensor-core sum (|d_s d_t| <= 2^14, a group sums at most 7
// pairs, and a part spans at most 18720 k: 7 2^14 18720 < 2^31 - 1).  The groups g < 8 (34 digit pairs) are
// kept.  The digits of a small value are as large as any other's, so a dropped group's products do not
// shrink with the values: those of g = 8, 5 pairs of about 74^2, come to 2^-66 of the scales' product per k and
// to 2^-57 over 7e5 k.  (Dropping g = 7 too would leave 2^-49, above the rounding of an FP64 sum.)
//
// Digit layout: for 128 rows and 32 k, one block of 28 KB holding the 7 digits' 128 x 32 matrices as the
// 8-row x 16-byte core matrices that an unswizzled K-major descriptor steps through.  A stage is then a
// bulk copy of the A panel's block and 7 of the B panel's 64 rows, with no tensor map.
//
// k_syrk_i8: one CTA per (128 x 64 tile (a, b), b <= 2 a + 1, split part).  TMEM holds the 8 groups'
// 64 columns side by side, and B's digits lie side by side in shared memory, so one MMA multiplies a digit s
// of A by several digits t of B, each result landing in the columns of its group s + t: 11 MMAs of up to
// 256 columns a chunk instead of 34, which read 103 bytes of shared memory a tensor clock (one digit pair per
// 128 x 128 MMA read 128, all that an SM delivers, before the copies into it).  One pass over the part fills
// every group.  The epilogue joins the groups in two 64-bit integers, scales, and stores the FP64 partials
// in the layout of k_syrk_f64, summed and unpacked by launch_unpack_sym.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>

#include "rijk_internal.h"
#include "tc_util.cuh"

namespace rijk {

int set_err(rijk_ctx* ctx, int code, const char* fmt, ...);
int cuda_check(rijk_ctx* ctx, cudaError_t e, const char* what);
int ensure(rijk_ctx* ctx, DeviceBuf& b, size_t bytes, const char* what);

namespace {

constexpr int kDigits = 7;                     // byte digits of a value
constexpr int kGroups = 8;                     // groups s + t kept
constexpr int kChunk = 32;                     // k per stage and per MMA
constexpr int kI8Threads = 192;                // warp 0 copies, warp 1 MMA, warps 2-5 epilogue
constexpr uint32_t kDigitA = 128 * kChunk;     // one digit of a 128-row panel: 4 KB
constexpr uint32_t kDigitB = 64 * kChunk;      // one digit of a 64-row panel: 2 KB
constexpr uint32_t kBlockBytes = kDigits * kDigitA;             // 28 KB
constexpr uint32_t kI8Stage = kDigits * (kDigitA + kDigitB);    // 42 KB
constexpr int kI8Stages = 5;
constexpr long kMaxPart = 18720;               // k per split part: 7 2^14 18720 < 2^31 - 1, every s32 sum exact
constexpr int kNonFinite = 1 << 20;            // row exponent of a row with an infinity or NaN

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}

// 2^e exactly for |e| <= 1000 (the exponent bits), else through ldexp.
__device__ __forceinline__ double pow2i(int e) {
  return (e >= -1000 && e <= 1000) ? __longlong_as_double(static_cast<long long>(e + 1023) << 52) : ldexp(1.0, e);
}

// ------------------------------------------------------------------ digits ----
// The exponent x of a row whose largest magnitude has the bits `top`: max / 2^x <= 127.49 2^48.
__device__ __forceinline__ int row_exponent(unsigned long long top) {
  if (top >= 0x7ff0000000000000ull) return kNonFinite;
  if (top == 0) return 0;
  const double m = __longlong_as_double(static_cast<long long>(top));
  const int e = ilogb(m) + 1;  // m < 2^e
  return (ldexp(m, -e) <= 0.995 ? e : e + 1) - 55;
}

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

// Digits of X^T.  One CTA per (8 rows, part): a first sweep takes the rows' maxima over the part (from
// HBM), a second one re-reads it (now in L2) and writes the digits, a lane per row and 16 k, so that 8
// lanes fill a 128-byte core matrix.  Rows at or past npad (the padding of the 128-row blocks), and k from
// kdim to the end of the last block, get zero digits.  HBM bounds it: 8 bytes read and 7 written per value.
constexpr int kSliceThreads = 256;

__global__ void __launch_bounds__(kSliceThreads) k_slice_x(const double* __restrict__ XT, long npad, long npad2,
                                                           long kdim, long kper, uint8_t* __restrict__ Xs,
                                                           int* __restrict__ E) {
  __shared__ unsigned long long top[8][kSliceThreads / 32];
  __shared__ int ex[8];
  const long r0 = static_cast<long>(blockIdx.x) * 8, part = blockIdx.y;
  const long k0 = part * kper, k1 = std::min(k0 + kper, kdim);
  const long kend = k1 == kdim ? (kdim + kChunk - 1) / kChunk * kChunk : k1;  // zero digits fill the last block
  const long nblk = (kdim + kChunk - 1) / kChunk;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool live = r0 < npad;  // npad is a multiple of 8
#pragma unroll 1
  for (int r = 0; r < 8; ++r) {
    unsigned long long m = 0;  // magnitudes order as their bit patterns, infinities and NaN above all
    if (live) {
      const double* x = XT + (r0 + r) * kdim;
      for (long k = k0 + 2L * t; k < k1; k += 2L * kSliceThreads) {  // kdim and kper are even
        const double2 a = *reinterpret_cast<const double2*>(x + k);
        const unsigned long long u = __double_as_longlong(a.x) & 0x7fffffffffffffffull;
        const unsigned long long v = __double_as_longlong(a.y) & 0x7fffffffffffffffull;
        m = max(m, max(u, v));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) top[r][warp] = m;
  }
  __syncthreads();
  if (t < 8) {
    unsigned long long m = 0;
    for (int w = 0; w < kSliceThreads / 32; ++w) m = max(m, top[t][w]);
    ex[t] = row_exponent(m);
    E[part * npad2 + r0 + t] = ex[t];
  }
  __syncthreads();
  // lane: row lane % 8, 16-k group warp * 4 + lane / 8 of each 512 k
  const int r = lane & 7;
  const int x = ex[r] == kNonFinite ? 0 : ex[r];
  const double* src = XT + (live ? r0 + r : 0) * kdim;
  uint8_t* base = Xs + (r0 / 128) * nblk * kBlockBytes + ((r0 % 128) / 8) * 256 + r * 16;
  for (long k = k0 + 16L * (warp * 4 + (lane >> 3)); k < kend; k += 16L * kSliceThreads / 8) {
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      double2 a = make_double2(0.0, 0.0);
      if (live && k + j < k1) a = *reinterpret_cast<const double2*>(src + k + j);
      v[j] = a.x;
      v[j + 1] = a.y;
    }
    uint4 d[kDigits];
    digits16(v, x, d);
    uint8_t* out = base + (k / kChunk) * kBlockBytes + ((k / 16) & 1) * 128;
#pragma unroll
    for (int s = 0; s < kDigits; ++s) *reinterpret_cast<uint4*>(out + s * kDigitA) = d[s];
  }
}

// ------------------------------------------------------------------ int8 SYRK ----
// The 8 groups of 16 columns (group g 64 columns after group g - 1) of this thread's TMEM lane, joined:
// sum_g v_g 256^(3-g), groups 0 - 3 and 4 - 7 each in one 64-bit integer (|v_g| < 2^31, so below 2^56).
__device__ __forceinline__ void join_groups16(uint32_t taddr, double (&w)[16]) {
  long long hi[16], lo[16];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t v[4][16];
#pragma unroll
    for (int g = 0; g < 4; ++g) tmem_ld16_nowait(taddr + (4 * h + g) * 64, v[g]);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      long long x = static_cast<int32_t>(v[0][j]);
#pragma unroll
      for (int g = 1; g < 4; ++g) x = x * 256 + static_cast<int32_t>(v[g][j]);
      (h == 0 ? hi[j] : lo[j]) = x;
    }
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) w[j] = fma(static_cast<double>(lo[j]), 1.0 / 4294967296.0, static_cast<double>(hi[j]));
}

// x 2^e
__device__ __forceinline__ double scale2(double x, int e) { return (e > -1000 && e < 1000) ? x * pow2i(e) : ldexp(x, e); }

struct I8Params {
  const uint8_t* Xs;
  long kdim, kper;
  int npad2, nt;
  double* Kpart;  // FP64 partials [part][ntile][64][64]
  long ntile;
  const int* E;   // row exponents [part][npad2]
  int* err;
};

// One chunk's MMAs: digit s of A against digits 0 .. min(6, 7 - s) of B, group s + t in the columns 64 (s + t).
// The chunk that starts the sums (first) overwrites each group on its first product: digit s = 0 starts
// groups 0 - 6, and (1, 6) starts group 7.
__device__ __forceinline__ void issue_chunk(uint32_t tmem, uint32_t sa, uint32_t sb, bool first) {
  constexpr uint64_t kDesc = plain_desc_bits(128, 256);  // core matrices 128 B apart along k, 256 B along rows
#pragma unroll
  for (int s = 0; s < kDigits; ++s) {
    const uint64_t da = sw128_desc(sa + s * kDigitA, kDesc);
    const int n = kGroups - s < kDigits ? kGroups - s : kDigits;  // digits of B
#pragma unroll
    for (int t = 0; t < n; t += 4) {
      const int m = n - t < 4 ? n - t : 4;  // up to 256 columns
      const uint64_t db = sw128_desc(sb + t * kDigitB, kDesc);
      const uint32_t d = tmem + (s + t) * 64;
      if (s == 1 && t + m == kDigits) {  // its last digit is group 7's first product
        if (m > 1) umma_s8(d, da, db, idesc_s8_s32(128, 64 * (m - 1)), 1u);
        umma_s8(d + 64 * (m - 1), da, sw128_desc(sb + (t + m - 1) * kDigitB, kDesc), idesc_s8_s32(128, 64), first ? 0u : 1u);
      } else {
        umma_s8(d, da, db, idesc_s8_s32(128, 64 * m), (first && s == 0) ? 0u : 1u);
      }
    }
  }
}

__global__ void __launch_bounds__(kI8Threads, 1) k_syrk_i8(I8Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kI8Stages * kI8Stage);
  uint64_t* empty = full + kI8Stages;
  uint64_t* tfull = empty + kI8Stages;  // the accumulators are final
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // tile (a, b): 128-row block a, 64-row block b <= 2 a + 1; blocks a' < a hold a (a + 1) tiles
  const int tile = blockIdx.x;
  int a = static_cast<int>((sqrtf(4.0f * tile + 1.0f) - 1.0f) * 0.5f);
  while (a * (a + 1) > tile) --a;
  while ((a + 1) * (a + 2) <= tile) ++a;
  const int b = tile - a * (a + 1);
  const long part = blockIdx.y;
  const long k0 = part * p.kper;
  const long k1 = std::min(k0 + p.kper, p.kdim);
  const int nch = static_cast<int>((k1 - k0 + kChunk - 1) / kChunk);
  const long nblk = (p.kdim + kChunk - 1) / kChunk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kI8Stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(tfull, 1);
    *abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint8_t* pa = p.Xs + (a * nblk + k0 / kChunk) * kBlockBytes;
      const uint8_t* pb = p.Xs + ((b / 2) * nblk + k0 / kChunk) * kBlockBytes + (b & 1) * kDigitB;
      for (int c = 0; c < nch; ++c) {
        if (!mbar_wait(&empty[stage], phase ^ 1, abort)) {
          ok = false;
          break;
        }
        uint8_t* st = smem + stage * kI8Stage;
        mbar_expect_tx(&full[stage], kI8Stage);
        bulk_load(st, pa, kBlockBytes, &full[stage]);
#pragma unroll
        for (int d = 0; d < kDigits; ++d)
          bulk_load(st + kBlockBytes + d * kDigitB, pb + d * kDigitA, kDigitB, &full[stage]);
        pa += kBlockBytes;
        pb += kBlockBytes;
        if (++stage == kI8Stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) {
        *abort = 1;
        atomicOr(p.err, DEVERR_TIMEOUT);
      }
      volatile int never = 0;  // every issued copy has landed before the CTA exits
      for (int i = 0; i < kI8Stages; ++i) {
        uint32_t par = (i < stage) ? phase : (phase ^ 1);
        mbar_wait(&full[i], par, &never);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int c = 0; c < nch; ++c) {
        if (!mbar_wait(&full[stage], phase, abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * kI8Stage);
        issue_chunk(tmem, sa, sa + kBlockBytes, c == 0);
        umma_commit(&empty[stage]);
        if (++stage == kI8Stages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) {
        *abort = 1;
        atomicOr(p.err, DEVERR_TIMEOUT);
      }
      umma_commit(tfull);  // also after a give-up: every MMA issued ends before TMEM is freed
      volatile int never = 0;
      if (!mbar_wait(tfull, 0, &never)) atomicOr(p.err, DEVERR_TIMEOUT);
    }
  } else {
    const int q = warp & 3;
    const int row = q * 32 + lane;     // row of the 128-row block
    const long ra = 2 * a + row / 64;  // 64-row tile, the same for the warp's 32 lanes
    const int r = row % 64;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(tfull, 0, abort)) && !__any_sync(0xffffffffu, *abort);
    tc_fence_after();
    // tiles above the diagonal (their mirror is stored) and rows past npad are left out
    if (ok && b <= ra && ra < p.nt) {
      const int* Ep = p.E + part * p.npad2;
      const int ea = Ep[a * 128 + row];
      const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16);
      double* out = p.Kpart + (part * p.ntile + tri_index(ra, b)) * TILE2 + static_cast<long>(r) * TILE;
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 16) {
        double v[16];
        join_groups16(lane_base + c0, v);
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          double w[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int eb = __ldg(Ep + b * 64 + c0 + j + h);
            w[h] = (ea == kNonFinite || eb == kNonFinite) ? __longlong_as_double(0x7ff8000000000000ll)
                                                          : scale2(v[j + h], 72 + ea + eb);
          }
          *reinterpret_cast<double2*>(out + c0 + j) = make_double2(w[0], w[1]);
        }
      }
    }
    if (!ok && lane == 0) {
      *abort = 1;
      atomicOr(p.err, DEVERR_TIMEOUT);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

int sm_count(int device) {
  static std::atomic<int> cached[64] = {};
  if (device < 0 || device >= 64) return 148;
  if (!cached[device]) {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
    cached[device] = v > 0 ? v : 148;
  }
  return cached[device];
}

}  // namespace

// Split-K parts of the int8 SYRK: chunk-aligned, at most kMaxPart k each; among up to four times the fewest
// parts (or parts for one wave), the count whose last wave of CTAs, one an SM, is fullest.
int syrk_i8_parts(long nt, long kdim, int device, long* kper_out) {
  const long nb = (nt + 1) / 2, ctas_per_part = nb * (nb + 1);
  const long sms = sm_count(device);
  const long nchunks = (kdim + kChunk - 1) / kChunk;
  const long min_parts = (kdim + kMaxPart - 1) / kMaxPart;
  const long want = std::max(min_parts, sms / ctas_per_part);
  long best = want;
  double best_eff = 0.0;
  for (long sp = want; sp <= 4 * want && sp <= std::max<long>(1, nchunks); ++sp) {
    const long ctas = ctas_per_part * sp, waves = (ctas + sms - 1) / sms;
    const double eff = static_cast<double>(ctas) / static_cast<double>(waves * sms);
    if (eff > best_eff + 0.02) {
      best_eff = eff;
      best = sp;
    }
  }
  long kper = round_up((kdim + best - 1) / best, kChunk);
  kper = std::min(kper, kMaxPart);
  *kper_out = kper;
  return static_cast<int>((kdim + kper - 1) / kper);
}

// K partials of the FP64 form from X^T (npad x kdim doubles) through its digits.
int syrk_i8(rijk_ctx* ctx, const double* XT, long npad, long nt, long kdim, int nparts, long kper, double* Kpart,
            cudaStream_t s) {
  const long npad2 = round_up(npad, 128);
  const long nblk = (kdim + kChunk - 1) / kChunk;
  int rc;
  if ((rc = ensure(ctx, ctx->Xs, static_cast<size_t>(npad2 / 128) * nblk * kBlockBytes, "int8 digits of X")) ||
      (rc = ensure(ctx, ctx->Xe, static_cast<size_t>(nparts) * npad2 * sizeof(int), "digit exponents")))
    return rc;
  uint8_t* Xs = static_cast<uint8_t*>(ctx->Xs.p);
  int* E = static_cast<int*>(ctx->Xe.p);
  k_slice_x<<<dim3(static_cast<unsigned>(npad2 / 8), static_cast<unsigned>(nparts)), kSliceThreads, 0, s>>>(
      XT, npad, npad2, kdim, kper, Xs, E);
  prof_mark(ctx, "slice_x");
  I8Params ip{};
  ip.Xs = Xs;
  ip.kdim = kdim;
  ip.kper = kper;
  ip.npad2 = static_cast<int>(npad2);
  ip.nt = static_cast<int>(nt);
  ip.Kpart = Kpart;
  ip.ntile = nt * (nt + 1) / 2;
  ip.E = E;
  ip.err = static_cast<int*>(ctx->err.p);
  const size_t smem = static_cast<size_t>(kI8Stages) * kI8Stage + 1024 + 256;
  ensure_smem_limit(reinterpret_cast<const void*>(k_syrk_i8), smem);
  const long nb = npad2 / 128;
  dim3 grid(static_cast<unsigned>(nb * (nb + 1)), static_cast<unsigned>(nparts));
  k_syrk_i8<<<grid, kI8Threads, smem, s>>>(ip);
  return cuda_check(ctx, cudaGetLastError(), "int8 SYRK launch");
}

}  // namespace rijk
