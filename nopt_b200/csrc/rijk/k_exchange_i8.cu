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

#include "i8_digits.cuh"
#include "i8_rule.h"
#include "rijk_internal.h"

namespace rijk {

int set_err(rijk_ctx* ctx, int code, const char* fmt, ...);
int cuda_check(rijk_ctx* ctx, cudaError_t e, const char* what);
int ensure(rijk_ctx* ctx, DeviceBuf& b, size_t bytes, const char* what);

namespace {

constexpr int kI8Threads = 192;                // warp 0 copies, warp 1 MMA, warps 2-5 epilogue
constexpr uint32_t kDigitB = 64 * kChunk;      // one digit of a 64-row panel: 2 KB
constexpr uint32_t kI8Stage = kDigits * (kDigitA + kDigitB);    // 42 KB
constexpr int kI8Stages = 5;

// Digits of X^T.  One CTA per (8 rows, part).  The rows' maxima over the part come with X (known: k_xform_i8
// leaves them in `tops`), or from a first sweep over it; then the digits are written, a lane per row and 16 k, so that 8
// lanes fill a 128-byte core matrix.  Rows at or past npad (the padding of the 128-row blocks), and k from
// kdim to the end of the last block, get zero digits.  HBM bounds it: 8 bytes read and 7 written per value.
constexpr int kSliceThreads = 256;

template <bool KNOWN>
__global__ void __launch_bounds__(kSliceThreads) k_slice_x(const double* __restrict__ XT, long npad, long npad2,
                                                           long kdim, long kper, const uint32_t* tops,
                                                           uint8_t* __restrict__ Xs, int* __restrict__ E) {
  __shared__ uint32_t top[8][kSliceThreads / 32];
  __shared__ int ex[8];
  const long r0 = static_cast<long>(blockIdx.x) * 8, part = blockIdx.y;
  const long k0 = part * kper, k1 = std::min(k0 + kper, kdim);
  const long kend = k1 == kdim ? (kdim + kChunk - 1) / kChunk * kChunk : k1;  // zero digits fill the last block
  const long nblk = (kdim + kChunk - 1) / kChunk;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool live = r0 < npad;  // npad is a multiple of 8
#pragma unroll 1
  for (int r = 0; r < 8 && !KNOWN; ++r) {
    uint32_t m = 0;
    if (live) {
      const double* x = XT + (r0 + r) * kdim;
      for (long k = k0 + 2L * t; k < k1; k += 2L * kSliceThreads) {  // kdim and kper are even
        const double2 a = *reinterpret_cast<const double2*>(x + k);
        m = max(m, max(magnitude(a.x), magnitude(a.y)));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) top[r][warp] = m;
  }
  __syncthreads();
  if (t < 8) {
    uint32_t m = 0;
    if (KNOWN)
      m = live ? tops[part * npad2 + r0 + t] : 0;
    else
      for (int w = 0; w < kSliceThreads / 32; ++w) m = max(m, top[t][w]);
    ex[t] = value_exponent(m);
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
struct I8Params {
  const uint8_t* Xs;
  long kdim, kper;
  int npad2, nt;
  double* Kpart;  // FP64 partials [part][ntile][64][64]
  long ntile;
  const int* E;   // row exponents [part][npad2]
  int* err;
};

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
        issue_digit_products<64, plain_desc_bits(128, 256), false>(tmem, sa, sa + kBlockBytes, c == 0);
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
      const double sa = value_scale(Ep[a * 128 + row]) * kJoined;
      const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16);
      double* out = p.Kpart + (part * p.ntile + tri_index(ra, b)) * TILE2 + static_cast<long>(r) * TILE;
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 16) {
        long long hi[16], lo[16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[4][16];
#pragma unroll
          for (int g = 0; g < 4; ++g) tmem_ld16_nowait(lane_base + (4 * h + g) * 64 + c0, v[g]);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) (h == 0 ? hi[j] : lo[j]) = join4(v[0][j], v[1][j], v[2][j], v[3][j]);
        }
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          double w[2];
#pragma unroll
          for (int h = 0; h < 2; ++h)
            w[h] = join8(hi[j + h], lo[j + h]) * sa * value_scale(__ldg(Ep + b * 64 + c0 + j + h));
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

// Split-K parts of the int8 SYRK: chunk-aligned, at most kMaxDigitSum k each; among up to four times the fewest
// parts (or parts for one wave), the count whose last wave of CTAs, one an SM, is fullest.
// Parts are whole aux functions (noccp k each) where a part can hold an even number of them, so that
// k_xform_i8 can keep each part's row maxima.
int syrk_i8_parts(long nt, long naux, long noccp, int device, long* kper_out) {
  const long kdim = naux * noccp;
  const long nb = (nt + 1) / 2, ctas_per_part = nb * (nb + 1);
  const long sms = sm_count(device);
  const long unit = noccp % kChunk == 0 ? noccp : 2 * noccp;  // aligned to chunks and aux functions
  const long grain = unit <= kMaxDigitSum ? unit : kChunk;
  const long max_part = kMaxDigitSum / grain * grain;
  const long min_parts = (kdim + max_part - 1) / max_part;
  const long want = std::max(min_parts, sms / ctas_per_part);
  long best = want;
  double best_eff = 0.0;
  for (long sp = want; sp <= 4 * want && sp <= std::max<long>(1, kdim / grain); ++sp) {
    const long ctas = ctas_per_part * sp, waves = (ctas + sms - 1) / sms;
    const double eff = static_cast<double>(ctas) / static_cast<double>(waves * sms);
    if (eff > best_eff + 0.02) {
      best_eff = eff;
      best = sp;
    }
  }
  const long kper = std::min(round_up((kdim + best - 1) / best, grain), max_part);
  *kper_out = kper;
  return static_cast<int>((kdim + kper - 1) / kper);
}

int syrk_i8_buffers(rijk_ctx* ctx, long npad, long kdim, int nparts) {
  const long npad2 = round_up(npad, 128), nblk = (kdim + kChunk - 1) / kChunk;
  const int rc = ensure(ctx, ctx->Xs, static_cast<size_t>(npad2 / 128) * nblk * kBlockBytes, "int8 digits of X");
  return rc ? rc : ensure(ctx, ctx->Xe, static_cast<size_t>(nparts) * npad2 * sizeof(int), "digit exponents");
}

// K partials of the FP64 form from X^T (npad x kdim doubles) through its digits.
// tops: the rows' largest magnitudes in every part (k_xform_i8), or null.
int syrk_i8(rijk_ctx* ctx, const double* XT, long npad, long nt, long kdim, int nparts, long kper,
            const uint32_t* tops, double* Kpart, cudaStream_t s) {
  const long npad2 = round_up(npad, 128);
  uint8_t* Xs = static_cast<uint8_t*>(ctx->Xs.p);
  int* E = static_cast<int*>(ctx->Xe.p);
  const dim3 sgrid(static_cast<unsigned>(npad2 / 8), static_cast<unsigned>(nparts));
  if (tops)
    k_slice_x<true><<<sgrid, kSliceThreads, 0, s>>>(XT, npad, npad2, kdim, kper, tops, Xs, E);
  else
    k_slice_x<false><<<sgrid, kSliceThreads, 0, s>>>(XT, npad, npad2, kdim, kper, tops, Xs, E);
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
