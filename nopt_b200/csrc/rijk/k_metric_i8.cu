// k_metric_i8.cu — K1, the metric contraction B^Q_{mu nu} = sum_P M_QP (P|mu nu) (k_metric.cu), on tcgen05 tensor
// cores with FP64 accuracy from exact int8 products (the digits and their error: k_exchange_i8.cu).
//
// The FP64 units bound k_metric_contract at 0.8 to 0.93 of DGEMM, most of a set-up's time.  Here both operands go in
// as digits along P: the rows of the raw integrals, one exponent each, gathered in the order of B's packed tile
// elements (k_slice_rows over blocks of 128 elements: two tile rows), and the rows of M, once per metric.
//
// k_metric_i8: persistent, one CTA per SM, over items (128 tile elements, 64 aux functions Q), the Q blocks of one
// element block next to each other so that its digits are read from HBM once.  Warp 0 copies stages of 32 P (28 KB
// of integrals, 14 KB of M), one thread of warp 1 issues the MMAs (digit s of the integrals against all digits
// of M side by side; eight groups of 64 columns fill the TMEM), eight epilogue warps join the groups,
// scale, and store: a lane holds one tile element, so each Q's 32 elements of a warp are 256 contiguous bytes of B.
// They also keep the largest |B^Q|, which the digits of B need.  Every digit sum is exact while naux is at most 18720.
// What bounds it: the int8 tensor pipe (34 products a value).  Against k_metric_contract, digits included: 4.5 instead of
// 11.7 ms at (H2O)8 cc-pVTZ (n 464, n_aux 1112), 7.1 instead of 18.0 at (H2O)16 cc-pVDZ, 0.69 instead of 2.13 s at
// (H2O)32 cc-pVTZ (n 1856, n_aux 4448: 102 TFLOP/s of the FP64 contraction, 3.5 POPS).
#include <algorithm>

#include "i8_digits.cuh"
#include "rijk_internal.h"

namespace rijk {
namespace {

constexpr int kQ = 64;         // aux functions of an item
constexpr int kMThreads = 320;  // warp 0 copies, warp 1 MMA, warps 2-9 epilogue
constexpr int kMStages = 5;
constexpr uint32_t kMStageB = kDigits * kQ * kChunk;  // 14 KB of M
constexpr uint32_t kMStage = kBlockBytes + kMStageB;
constexpr size_t kMSmem = static_cast<size_t>(kMStages) * kMStage + 1024 + 256;
constexpr long kMaxSum = 18720;  // 7 2^14 18720 < 2^31 - 1: every s32 sum exact
constexpr size_t kDigitRoom = 512ul << 20;  // digits of raw integrals in flight

// Where row i of a digitised matrix lies: i itself, or the pair row of a packed tile element (-1: none).
struct RowMap {
  int tiles;  // 0: identity
  int layout;
  long n, I0, pair_base, e0, count;
  __device__ long operator()(long i) const {
    if (i >= count) return -1;
    if (!tiles) return i;
    const long e = e0 + i;
    long I, J;
    tri_decode(e / TILE2, I, J);
    const long mu = I * TILE + (e % TILE2) / TILE, nu = J * TILE + e % TILE;
    if (mu >= n || nu >= n) return -1;
    if (layout == RIJK_LAYOUT_NOPT_FULL) return (mu - I0 * TILE) * n + nu;
    const long hi = mu > nu ? mu : nu, lo = mu > nu ? nu : mu;
    return hi * (hi + 1) / 2 + lo - pair_base;
  }
};

// Digits of rows of k values (a multiple of 32, pitch ld): blocks of `rows` (64 or 128) rows x 32 k as core-matrix
// images.  One CTA per 16 rows: a sweep for the rows' maxima, then the digits (re-read from L2), a lane per row and
// 16 k, so that 8 lanes fill a 128-byte core matrix.
__global__ void __launch_bounds__(256) k_slice_rows(const double* __restrict__ X, long ld, long k, int rows, RowMap map,
                                                    double* __restrict__ scale, uint8_t* __restrict__ out) {
  __shared__ uint32_t top[16];
  __shared__ long at[16];
  const long i0 = static_cast<long>(blockIdx.x) * 16;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t < 16) at[t] = map(i0 + t);
  __syncthreads();
  for (int r = 2 * warp; r < 2 * warp + 2; ++r) {
    uint32_t m = 0;
    if (at[r] >= 0)
      for (long j = 2L * lane; j < k; j += 64) {
        const double2 v = *reinterpret_cast<const double2*>(X + at[r] * ld + j);
        m = max(m, max(magnitude(v.x), magnitude(v.y)));
      }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) top[r] = m;
  }
  __syncthreads();
  if (t < 16) scale[i0 + t] = value_scale(value_exponent(top[t]));
  const int r = ((warp & 1) << 3) | (lane & 7);
  int e = value_exponent(top[r]);
  if (e == kNonFinite) e = 0;
  const long row = i0 + r, nk = k / kChunk;
  const uint32_t digit = static_cast<uint32_t>(rows) * kChunk;
  uint8_t* base = out + (row / rows) * nk * (kDigits * digit) + ((row % rows) >> 3) * 256 + (row & 7) * 16;
  for (long g = (warp >> 1) * 4 + (lane >> 3); g < 2 * nk; g += 16) {
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      double2 w = make_double2(0.0, 0.0);
      if (at[r] >= 0) w = *reinterpret_cast<const double2*>(X + at[r] * ld + g * 16 + j);
      v[j] = w.x;
      v[j + 1] = w.y;
    }
    uint4 d[kDigits];
    digits16(v, e, d);
    uint8_t* p = base + (g >> 1) * (kDigits * digit) + (g & 1) * 128;
#pragma unroll
    for (int s = 0; s < kDigits; ++s) *reinterpret_cast<uint4*>(p + s * digit) = d[s];
  }
}

struct MetricI8Params {
  const uint8_t* I3;      // digits of the integrals, [element block][chunk]
  const uint8_t* M;       // digits of M, [Q block][chunk]
  const double* scale3;   // per element
  const double* scaleM;   // per Q
  double* B;              // at the first element block
  uint32_t* top;
  long tile_elems;
  int nblk, nqb, nk, naux;
  int qb0;                // first Q block of the metric (an aux range may start inside it)
  int qoff;               // rows of that block before the range
  long tri;               // first Q of the range when M is lower triangular, else -1
  int* err;
};

// Chunks of one Q block: M's rows end at the diagonal in the Cholesky form.
__device__ __forceinline__ int chunks_of(const MetricI8Params& p, int qb) {
  if (p.tri < 0) return p.nk;
  return min(p.nk, (p.qb0 + qb + 1) * kQ / kChunk);
}

__global__ void __launch_bounds__(kMThreads, 1) k_metric_i8(MetricI8Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kMStages * kMStage);
  uint64_t* empty = full + kMStages;
  uint64_t* tfull = empty + kMStages;  // an item's groups are final
  uint64_t* tempty = tfull + 1;        // ... and have been read
  uint64_t* drain = tempty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kMStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, 8);
    mbar_init(drain, 1);
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
  const long nitems = static_cast<long>(p.nblk) * p.nqb;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (long item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
        const long blk = item / p.nqb;
        const int qb = static_cast<int>(item - blk * p.nqb);
        const uint8_t* pa = p.I3 + blk * p.nk * kBlockBytes;
        const uint8_t* pb = p.M + static_cast<long>(p.qb0 + qb) * p.nk * kMStageB;
        const int nk = chunks_of(p, qb);
        for (int c = 0; c < nk; ++c) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort)) {
            ok = false;
            break;
          }
          uint8_t* st = smem + stage * kMStage;
          mbar_expect_tx(&full[stage], kMStage);
          bulk_load(st, pa, kBlockBytes, &full[stage]);
          bulk_load(st + kBlockBytes, pb, kMStageB, &full[stage]);
          pa += kBlockBytes;
          pb += kMStageB;
          if (++stage == kMStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) {
        *abort = 1;
        atomicOr(p.err, DEVERR_TIMEOUT);
      }
      volatile int never = 0;  // every issued copy has landed before the CTA exits
      for (int i = 0; i < kMStages; ++i) {
        uint32_t par = (i < stage) ? phase : (phase ^ 1);
        mbar_wait(&full[i], par, &never);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, tph = 0;
      bool ok = true;
      for (long item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
        const int nk = chunks_of(p, static_cast<int>(item % p.nqb));
        if (!mbar_wait(tempty, tph ^ 1, abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        for (int c = 0; c < nk; ++c) {
          if (!mbar_wait(&full[stage], phase, abort)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * kMStage);
          issue_digit_products<kQ, plain_desc_bits(128, 256), false>(tmem, sa, sa + kBlockBytes, c == 0);
          umma_commit(&empty[stage]);
          if (++stage == kMStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        umma_commit(tfull);
        tph ^= 1;
      }
      if (!ok) {
        *abort = 1;
        atomicOr(p.err, DEVERR_TIMEOUT);
      }
      umma_commit(drain);  // every MMA issued ends before TMEM is freed
      volatile int never = 0;
      if (!mbar_wait(drain, 0, &never)) atomicOr(p.err, DEVERR_TIMEOUT);
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;  // TMEM lanes 32 q .., columns 32 half ..
    uint32_t tph = 0;
    for (long item = blockIdx.x; item < nitems; item += gridDim.x) {
      const long blk = item / p.nqb;
      const int qb = static_cast<int>(item - blk * p.nqb);
      if (!__all_sync(0xffffffffu, mbar_wait(tfull, tph, abort)) || __any_sync(0xffffffffu, *abort)) {
        if (lane == 0) {
          *abort = 1;
          atomicOr(p.err, DEVERR_TIMEOUT);
        }
        break;
      }
      tc_fence_after();
      const uint32_t t0 = tmem + (static_cast<uint32_t>(q * 32) << 16) + half * 32;
      long long hi[32], lo[32];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[4][16];
#pragma unroll
          for (int g = 0; g < 4; ++g) tmem_ld16_nowait(t0 + (4 * h + g) * kQ + u * 16, v[g]);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) (h == 0 ? hi : lo)[u * 16 + j] = join4(v[0][j], v[1][j], v[2][j], v[3][j]);
        }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty);
      tph ^= 1;
      const long e = blk * 128 + q * 32 + lane;
      const double se = p.scale3[e] * kJoined;
      const int j0 = (p.qb0 + qb) * kQ + half * 32;               // row of M
      const long q0 = static_cast<long>(qb) * kQ + half * 32 - p.qoff;  // aux function of the range, < 0 before it
      uint32_t mine = 0;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const double x = join8(hi[j], lo[j]) * se * __ldg(p.scaleM + j0 + j);
        const bool in = q0 + j >= 0 && q0 + j < p.naux;
        if (in) p.B[(q0 + j) * p.tile_elems + e] = x;
        const uint32_t m = __reduce_max_sync(0xffffffffu, magnitude(x));
        if (lane == j && in) mine = m;
      }
      if (q0 + lane >= 0 && q0 + lane < p.naux) atomicMax(p.top + q0 + lane, mine);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

long digit_bytes(long rows, long nk) { return rows * nk * kDigits * kChunk; }

// The digits of the metric factor, made on the first large contraction after rijk_set_metric.
bool mdig_prepare(rijk_ctx* ctx, long nauxp) {
  if (ctx->have_mdig) return true;
  const long rows = round_up(nauxp, kQ);
  const std::string keep = ctx->last_error;  // running out of room here is no error
  if (ensure(ctx, ctx->Mdig, rows * sizeof(double) + digit_bytes(rows, nauxp / kChunk), "int8 digits of M")) {
    ctx->last_error = keep;
    return false;
  }
  RowMap map{};
  map.count = nauxp;
  double* scale = static_cast<double*>(ctx->Mdig.p);
  k_slice_rows<<<static_cast<unsigned>(rows / 16), 256, 0, ctx->stream>>>(static_cast<const double*>(ctx->M.p), nauxp, nauxp, kQ,
                                                                        map, scale, reinterpret_cast<uint8_t*>(scale + rows));
  ctx->have_mdig = true;
  return true;
}

}  // namespace

void metric_contract(rijk_ctx* ctx, const double* raw, int layout, long n, long I0, long I1, DeviceBuf& digits) {
  const long naux = ctx->naux, nauxp = round_up(naux, kChunk), nq = ctx->nq, q0 = ctx->q0;
  const long nt = round_up(n, TILE) / TILE;
  const bool chol = ctx->metric_form == RIJK_METRIC_CHOLESKY;
  const long t0 = tri_index(I0, 0), t1 = tri_index(I1, 0), elems = (t1 - t0) * TILE2;
  double* B = static_cast<double*>(ctx->B.p);
  uint32_t* top = static_cast<uint32_t*>(ctx->Btop.p);
  const long nk = nauxp / kChunk;
  // elements of one round: whole blocks whose digits fit the room
  const long round = std::max<long>(128, std::min<long>(elems, static_cast<long>(kDigitRoom) / digit_bytes(1, nk) / 128 * 128));
  // below this the launches and the digits of M cost what is gained (0.1 ms of DMMA)
  const bool large = 2.0 * elems * nq * nauxp >= 2e9 && nauxp <= kMaxSum;
  const std::string keep = ctx->last_error;
  if (!large || !mdig_prepare(ctx, nauxp) ||
      ensure_tmp(ctx, digits, round * sizeof(double) + digit_bytes(round, nk), "int8 digits of the integrals")) {
    if (large) ctx->last_error = keep;
    launch_metric_contract_chunk(static_cast<const double*>(ctx->M.p) + q0 * nauxp, nauxp, nauxp - q0, raw, layout, n, nq, nt,
                                 I0, I1, B, top, ctx->stream, chol ? q0 : -1);
    return;
  }
  MetricI8Params p{};
  double* scale3 = static_cast<double*>(digits.p);
  uint8_t* d3 = reinterpret_cast<uint8_t*>(scale3 + round);
  const long mrows = round_up(nauxp, kQ);
  p.I3 = d3;
  p.scale3 = scale3;
  p.scaleM = static_cast<const double*>(ctx->Mdig.p);
  p.M = reinterpret_cast<const uint8_t*>(p.scaleM + mrows);
  p.top = top;
  p.tile_elems = nt * (nt + 1) / 2 * TILE2;
  p.nk = static_cast<int>(nk);
  p.naux = static_cast<int>(nq);
  p.qb0 = static_cast<int>(q0 / kQ);
  p.qoff = static_cast<int>(q0 % kQ);
  p.nqb = static_cast<int>((q0 + nq - 1) / kQ - q0 / kQ + 1);
  p.tri = chol ? q0 : -1;
  p.err = static_cast<int*>(ctx->err.p);
  ensure_smem_limit(reinterpret_cast<const void*>(k_metric_i8), kMSmem);
  RowMap map{};
  map.tiles = 1;
  map.layout = layout;
  map.n = n;
  map.I0 = I0;
  map.pair_base = I0 * TILE * (I0 * TILE + 1) / 2;
  for (long e = 0; e < elems; e += round) {
    const long cnt = std::min(round, elems - e);  // a multiple of 128
    map.e0 = t0 * TILE2 + e;
    map.count = cnt;
    k_slice_rows<<<static_cast<unsigned>(cnt / 16), 256, 0, ctx->stream>>>(raw, nauxp, nauxp, 128, map, scale3, d3);
    p.B = B + t0 * TILE2 + e;
    p.nblk = static_cast<int>(cnt / 128);
    const long items = static_cast<long>(p.nblk) * p.nqb;
    k_metric_i8<<<static_cast<unsigned>(std::min<long>(items, ctx->sms)), kMThreads, kMSmem, ctx->stream>>>(p);
  }
}

}  // namespace rijk
