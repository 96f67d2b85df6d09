// k_xform_i8.cu — the half-transform X^Q = C B^Q of the FP64 form on tcgen05 tensor cores, with FP64 accuracy
// from exact int8 products (the digits and their error: k_exchange_i8.cu).
//
// Digits of B, written once per fitted tensor (bdig_prepare): for every aux function Q, with one exponent
// x_Q, the 128 x 128 blocks (a, b), b <= a, of the symmetric B^Q, each as its seven digits' 128 x 128 bytes in
// 8-row x 16-byte core matrices, ordered [16-column group][8-row group].  Both ways to read a block are then
// one rectangular copy of 28 KB into the unswizzled canonical layouts:
//   rows as M   32 columns = 2 column groups of 2 KB             K-major:  SBO 128 (rows), LBO 2048 (columns)
//   columns as M  32 rows = 4 row groups of each column group     MN-major: SBO 512 (columns), LBO 128 (rows)
// so the stored lower triangle serves the full symmetric matrix, as in the other half-transforms.
//
// Row scales.  One exponent per Q (a block is read both ways) leaves every element an absolute rounding of 2^-55 of the
// largest of B^Q.  So that this means as much to every function, whatever the sizes of the functions, the digits are
// those of 2^-(e_mu + e_nu) B^Q_{mu nu}, with e_mu such that every row's largest element over all Q is about 1
// (k_balance, from the magnitudes the metric contraction keeps).  The factors are exact: those of the summed index go into
// the digits of C, those of the row nu into X.  The error of K_{mu nu} against sqrt(K_mu,mu K_nu,nu) is then the same for
// any scaling of the functions by powers of two: at the most 1.6e-15 for C12H26 cc-pVDZ (1.2e-15 on DMMA, 2.2e-5 without
// the scales when the functions' sizes spread over 2^20), 3e-16 for C24H50 (2.7e-14, 3.7e-6).  An element far below
// that size, of functions far apart, keeps fewer digits of its own than DMMA would leave it (5e-13 in the median for
// C24H50, against 8e-15).
// Where the rows' largest elements lie within a factor of 11, e = 0 serves as well (1.1e-15 for C12H26; 2.6e-15 at a
// factor of 16) and saves a pass over B: those of normalised functions in double- and triple-zeta bases lie
// within 3 to 10.
//
// k_xform_i8: persistent, one CTA per SM, over items (Q, 128 rows nu, batch of at most 64 orbitals), the batches of
// one (Q, rows) next to each other so that the later ones find B's digits in L2.  Warp 0 copies stages of
// 32 contraction indices (28 KB of B, 14 KB of orbitals), one thread of warp 1 issues the MMAs (digit s of B against
// all digits of C side by side, eight groups of up to 64 columns in the whole TMEM), and eight epilogue
// warps join each item's groups in 64-bit integers (TMEM is free again after about a thousand cycles), scale,
// write rows of XT through shared memory in 128-byte pieces, and keep each split part's row maxima for k_slice_x.
//
// What bounds it: the int8 tensor pipe at 34 products a value, and for few orbitals the copies from L2 (42 KB a
// stage of 1088 tensor clocks, a third less to do with 48 or 32 orbitals).  Against k_xform_f64: 17.8 instead of 52.1
// ms at C40H82 (n 970, n_aux 4686, n_c 161: 3.3 POPS of 34 products under the power cap), 3.3 instead of 8.4 at C25H52,
// 0.71 instead of 1.37 at (H2O)16 (n 384, n_c 80).  The first form of the epilogue (per-column exponents, 64-bit
// maxima, 8-byte stores) took 1.03 ms at (H2O)16: its eight warps, not the MMAs, set an item's time.
// K's error against extended precision, through this kernel and k_syrk_i8: 6e-17 of |K| at (H2O)16 where the DMMA
// kernels leave 1.3e-15, 1.1e-16 against 3e-16 from one to six waters.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "i8_digits.cuh"
#include "rijk_internal.h"

namespace rijk {
namespace {

constexpr long kSuper = 4L * kBlockBytes;  // a 128 x 128 block: 7 digits of 16 KB
constexpr int kXThreads = 320;             // warp 0 copies, warp 1 MMA, warps 2-9 epilogue
constexpr int kXStages = 4;
constexpr uint32_t kXStageC = kDigits * 64 * kChunk;  // orbitals of a stage, at most 14 KB
constexpr uint32_t kXStage = kBlockBytes + kXStageC;
constexpr int kOutLd = 18;  // doubles a row of the epilogue's transposing buffers (32 rows x 16 columns)
constexpr size_t kXSmem = static_cast<size_t>(kXStages) * kXStage + 8 * 32 * kOutLd * sizeof(double) + 1024 + 256;

// ------------------------------------------------------------------ digits of B ----
// top[e] = the largest magnitude over Q of element e, for a tensor that no metric contraction has left it for.
__global__ void __launch_bounds__(256) k_element_max(const double* __restrict__ B, long nq, long tile_elems, uint32_t* top) {
  const long e = static_cast<long>(blockIdx.x) * 256 + threadIdx.x;  // a double2; tile_elems / 2 is a multiple of 256
  const double2* b = reinterpret_cast<const double2*>(B) + e;
  uint32_t mx = 0, my = 0;
#pragma unroll 4
  for (long q = blockIdx.y; q < nq; q += gridDim.y) {
    const double2 v = ldg_stream(b + q * (tile_elems / 2));
    mx = max(mx, magnitude(v.x));
    my = max(my, magnitude(v.y));
  }
  atomicMax(top + 2 * e, mx);
  atomicMax(top + 2 * e + 1, my);
}

// log2 of a magnitude; nothing to balance where it is zero or not finite.  A row of nothing else has e = NaN, which the
// maxima below pass over.
__device__ __forceinline__ float log2_magnitude(uint32_t top) {
  if (top == 0 || top >= 0x7ff00000u) return -INFINITY;
  return static_cast<float>(static_cast<int>(top >> 20) - 1023) + __log2f(__uint_as_float(0x3f800000u | ((top & 0xfffffu) << 3)));
}

// Whether e = 0 will do (kPlain), from the first step's logarithms: half those of the rows' largest elements.  The
// aux functions' own maxima are then those of the metric contraction, if it has left any.
enum { kPlain = 0, kScaled = 1, kPlainNoTops = 2 };
__global__ void __launch_bounds__(256) k_spread(const float* __restrict__ e, long n, int have_tops, int* __restrict__ how) {
  __shared__ float lo[8], hi[8];
  float a = INFINITY, b = -INFINITY;
  for (long i = threadIdx.x; i < n; i += 256) {
    a = fminf(a, e[i]);
    b = fmaxf(b, e[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
    b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
  }
  if ((threadIdx.x & 31) == 0) {
    lo[threadIdx.x >> 5] = a;
    hi[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      a = fminf(a, lo[w]);
      b = fmaxf(b, hi[w]);
    }
    *how = b - a > 1.75f ? kScaled : have_tops ? kPlain : kPlainNoTops;
  }
}

// One step towards row scales: e_mu grows by half the logarithm of its row's largest scaled element, so that a pair
// of rows meets in the middle (Ruiz's scaling; it converges by halving, in one step where diagonals lead).  A warp a row.
__global__ void __launch_bounds__(256) k_balance(const uint32_t* __restrict__ top, long n, const int* how,
                                                 const float* __restrict__ e0, float* __restrict__ e1) {
  if (how && *how != kScaled) return;
  const long mu = static_cast<long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (mu >= n) return;
  const long I = mu / TILE, r = mu % TILE;
  float m = -INFINITY;
  for (long nu = threadIdx.x & 31; nu < n; nu += 32) {
    const long J = nu / TILE, c = nu % TILE;
    uint32_t t = top[I >= J ? tri_index(I, J) * TILE2 + r * TILE + c : tri_index(J, I) * TILE2 + c * TILE + r];
    if (I == J) t = max(t, top[tri_index(I, I) * TILE2 + c * TILE + r]);
    m = fmaxf(m, log2_magnitude(t) - e0[nu]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) e1[mu] = m == -INFINITY ? NAN : 0.5f * (e0[mu] + m);
}
constexpr int kBalanceSteps = 8;  // even: the result is where the first step read

// The scales as powers of two, down = 2^-e for B and up = 2^e for C and X; e0: the result, e1: any step's.  A function
// without any element has up = 0: its coefficients, whatever their size against the others', must not set the
// exponents of C.
__global__ void k_balance_scales(const float* __restrict__ e0, const float* __restrict__ e1, long n, long npad2,
                                 const int* how, double* __restrict__ down, double* __restrict__ up) {
  const long mu = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (mu >= npad2) return;
  const bool none = mu < n && isnan(e1[mu]);
  const int x = mu < n && !none && *how == kScaled ? static_cast<int>(rintf(fminf(fmaxf(e0[mu], -600.f), 600.f))) : 0;
  down[mu] = pow2i(-x);
  up[mu] = none ? 0.0 : pow2i(x);
}

// top[Q] = the largest magnitude of the scaled B^Q
__global__ void __launch_bounds__(256) k_bmax(const double* __restrict__ B, long ntile, const int* how,
                                              const double* __restrict__ down, uint32_t* top) {
  if (*how == kPlain) return;
  uint32_t m = 0;
  for (long t = blockIdx.x; t < ntile; t += gridDim.x) {
    long I, J;
    tri_decode(t, I, J);
    const double2* b = reinterpret_cast<const double2*>(B + (blockIdx.y * ntile + t) * TILE2);
    const int c = 2 * (threadIdx.x & 31);
    const double2 dc = __ldg(reinterpret_cast<const double2*>(down + J * TILE + c));
#pragma unroll
    for (int k = 0; k < TILE / 8; ++k) {
      const int r = (threadIdx.x >> 5) + 8 * k;
      const double dr = __ldg(down + I * TILE + r);
      const double2 v = ldg_stream(b + (r * TILE + c) / 2);
      m = max(m, max(magnitude(v.x * dr * dc.x), magnitude(v.y * dr * dc.y)));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(top + blockIdx.y, m);
}

// Their exponents, and the scales that go with the digits.
__global__ void k_exponents(const uint32_t* __restrict__ plain, const uint32_t* __restrict__ scaled, const int* how,
                            long count, int* __restrict__ ex, double* __restrict__ scale) {
  const uint32_t* top = *how == kPlain ? plain : scaled;
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    ex[i] = value_exponent(top[i]);
    scale[i] = value_scale(ex[i]);
  }
}

// One CTA per (128 x 128 block, Q): a lane per row and 16 columns, consecutive lanes on consecutive rows, so a
// warp writes 512 contiguous bytes of each digit.
__global__ void __launch_bounds__(256) k_slice_b(const double* __restrict__ B, long nt, long tile_elems, long nsb,
                                                 const int* __restrict__ ex, const double* __restrict__ down,
                                                 uint8_t* __restrict__ out) {
  long a, b;
  tri_decode(blockIdx.x, a, b);
  const long Q = blockIdx.y;
  const int e = ex[Q] == kNonFinite ? 0 : ex[Q];
  const double* BQ = B + Q * tile_elems;
  uint8_t* img = out + (Q * nsb + blockIdx.x) * kSuper;
  const int r = threadIdx.x & 127;
  const double dr = down[a * 128 + r];
  for (int cg = threadIdx.x >> 7; cg < 8; cg += 2) {
    const long I = 2 * a + (r >> 6), J = 2 * b + (cg >> 2);
    double v[16];
    if (I >= nt || J >= nt) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = 0.0;
    } else if (I >= J) {
      const double2* src = reinterpret_cast<const double2*>(BQ + tri_index(I, J) * TILE2 + (r & 63) * TILE + (cg & 3) * 16);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double2 w = src[j];
        v[2 * j] = w.x;
        v[2 * j + 1] = w.y;
      }
    } else {  // the tile above the diagonal of a diagonal block: the stored one's transpose
      const double* src = BQ + tri_index(J, I) * TILE2 + (cg & 3) * 16 * TILE + (r & 63);
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = src[j * TILE];
    }
    const double2* dc = reinterpret_cast<const double2*>(down + b * 128 + cg * 16);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const double2 f = __ldg(dc + j);
      v[2 * j] = v[2 * j] * dr * f.x;
      v[2 * j + 1] = v[2 * j + 1] * dr * f.y;
    }
    uint4 d[kDigits];
    digits16(v, e, d);
    uint8_t* p = img + cg * 2048 + r * 16;  // 8-row groups of 128 B
#pragma unroll
    for (int s = 0; s < kDigits; ++s) *reinterpret_cast<uint4*>(p + s * 16384) = d[s];
  }
}

// ------------------------------------------------------------------ digits of C ----
// Orbital batches: nbatch of them, of 16 (base + 1) or 16 base rows, the larger ones first.
struct Batches {
  int nbatch, base, extra;
  __host__ __device__ int first(int b) const { return 16 * (b * base + (b < extra ? b : extra)); }
  __host__ __device__ int rows(int b) const { return 16 * (base + (b < extra ? 1 : 0)); }
};

// One CTA per 16 orbital rows: their maxima over the n scaled columns, then digits, [chunk][digit][8-row group][2][8][16].
__global__ void __launch_bounds__(128) k_slice_c(const double* __restrict__ MOp, long n, long npad, long nk, Batches bt,
                                                 const double* __restrict__ up, double* __restrict__ scale,
                                                 uint8_t* __restrict__ out) {
  __shared__ uint32_t top[16];
  const int i0 = blockIdx.x * 16, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int r = warp; r < 16; r += 4) {
    uint32_t m = 0;
    for (long k = lane; k < n; k += 32) m = max(m, magnitude(MOp[(i0 + r) * npad + k] * up[k]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) top[r] = m;
  }
  __syncthreads();
  if (t < 16) scale[i0 + t] = value_scale(value_exponent(top[t]));
  int b = 0;
  while (b + 1 < bt.nbatch && bt.first(b + 1) <= i0) ++b;
  const long nb = bt.rows(b), row0 = i0 - bt.first(b);
  uint8_t* img = out + static_cast<long>(bt.first(b)) * kDigits * kChunk * nk;
  const int r = t & 15;
  int e = value_exponent(top[r]);
  if (e == kNonFinite) e = 0;
  for (long g = t >> 4; g < 2 * nk; g += 8) {  // 16 columns; the rows are zero from n to npad
    double v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = MOp[(i0 + r) * npad + g * 16 + j] * up[g * 16 + j];
    uint4 d[kDigits];
    digits16(v, e, d);
    const long row = row0 + r;
    uint8_t* p = img + (g >> 1) * (kDigits * nb * kChunk) + (row >> 3) * 256 + (g & 1) * 128 + (row & 7) * 16;
#pragma unroll
    for (int s = 0; s < kDigits; ++s) *reinterpret_cast<uint4*>(p + s * nb * kChunk) = d[s];
  }
}

// ------------------------------------------------------------------ half-transform ----
struct XformI8Params {
  const uint8_t* C;
  const double* scaleB;
  const double* scaleC;
  const double* up;          // row scales of B's digits
  double* XT;
  uint32_t* tops;            // [part][npad2]
  long qper;                 // aux functions of a part
  long kdim, npad, nsb;
  int naux, nb, nk, noccp;   // 128-row blocks, 32-wide chunks
  Batches bt;
  int* err;
};

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::
          "r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

// The MMAs of one item: blocks K <= M of B^Q read by rows, the others by columns.
template <int NB>
__device__ __forceinline__ bool item_mmas(int nk, int M, uint32_t tmem, uint8_t* smem, uint64_t* full, uint64_t* empty,
                                          int& stage, uint32_t& phase, volatile int* abort) {
  for (int c = 0; c < nk; ++c) {
    if (!mbar_wait(&full[stage], phase, abort)) return false;
    tc_fence_after();
    const uint32_t sa = smem_u32(smem + stage * kXStage);
    if ((c >> 2) <= M)
      issue_digit_products<NB, plain_desc_bits(2048, 128), false>(tmem, sa, sa + kBlockBytes, c == 0);
    else  // never an item's first chunk
      issue_digit_products<NB, plain_desc_bits(128, 512), true>(tmem, sa, sa + kBlockBytes, false);
    umma_commit(&empty[stage]);
    if (++stage == kXStages) {
      stage = 0;
      phase ^= 1;
    }
  }
  return true;
}

__global__ void __launch_bounds__(kXThreads, 1)
    k_xform_i8(const __grid_constant__ CUtensorMap map_rows, const __grid_constant__ CUtensorMap map_cols, XformI8Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  double* outb = reinterpret_cast<double*>(smem + kXStages * kXStage);
  uint64_t* full = reinterpret_cast<uint64_t*>(outb + 8 * 32 * kOutLd);
  uint64_t* empty = full + kXStages;
  uint64_t* tfull = empty + kXStages;  // an item's groups are final
  uint64_t* tempty = tfull + 1;        // ... and have been read
  uint64_t* drain = tempty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kXStages; ++i) {
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
  const int per_q = p.nb * p.bt.nbatch;
  const long nitems = static_cast<long>(p.naux) * per_q;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&map_rows);
      tma_prefetch_desc(&map_cols);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (long item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
        const int Q = static_cast<int>(item / per_q), rest = static_cast<int>(item - static_cast<long>(Q) * per_q);
        const int M = rest / p.bt.nbatch, b = rest - M * p.bt.nbatch;
        const uint32_t cbytes = static_cast<uint32_t>(p.bt.rows(b)) * kDigits * kChunk;
        const uint8_t* pc = p.C + static_cast<long>(p.bt.first(b)) * kDigits * kChunk * p.nk;
        const long qs = static_cast<long>(Q) * p.nsb;
        for (int c = 0; c < p.nk; ++c) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort)) {
            ok = false;
            break;
          }
          uint8_t* st = smem + stage * kXStage;
          mbar_expect_tx(&full[stage], kBlockBytes + cbytes);
          const int K = c >> 2, part = c & 3;
          if (K <= M)
            tma_load_4d(st, &map_rows, &full[stage], 0, 2 * part, 0, static_cast<int>(qs + tri_index(M, K)));
          else
            tma_load_4d(st, &map_cols, &full[stage], 64 * part, 0, 0, static_cast<int>(qs + tri_index(K, M)));
          bulk_load(st + kBlockBytes, pc, cbytes, &full[stage]);
          pc += cbytes;
          if (++stage == kXStages) {
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
      for (int i = 0; i < kXStages; ++i) {
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
        const int rest = static_cast<int>(item % per_q);
        const int M = rest / p.bt.nbatch, nbr = p.bt.rows(rest - M * p.bt.nbatch);
        if (!mbar_wait(tempty, tph ^ 1, abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        switch (nbr) {
          case 16: ok = item_mmas<16>(p.nk, M, tmem, smem, full, empty, stage, phase, abort); break;
          case 32: ok = item_mmas<32>(p.nk, M, tmem, smem, full, empty, stage, phase, abort); break;
          case 48: ok = item_mmas<48>(p.nk, M, tmem, smem, full, empty, stage, phase, abort); break;
          default: ok = item_mmas<64>(p.nk, M, tmem, smem, full, empty, stage, phase, abort); break;
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
    const int q = warp & 3, half = (warp - 2) >> 2;  // TMEM lanes 32 q .., the lower or upper half of the columns
    double* mine = outb + (warp - 2) * 32 * kOutLd;
    uint32_t tph = 0;
    for (long item = blockIdx.x; item < nitems; item += gridDim.x) {
      const int Q = static_cast<int>(item / per_q), rest = static_cast<int>(item - static_cast<long>(Q) * per_q);
      const int M = rest / p.bt.nbatch, b = rest - M * p.bt.nbatch;
      const int nbr = p.bt.rows(b), units = nbr / 16;  // 8-column units of this half
      if (!__all_sync(0xffffffffu, mbar_wait(tfull, tph, abort)) || __any_sync(0xffffffffu, *abort)) {
        if (lane == 0) {
          *abort = 1;
          atomicOr(p.err, DEVERR_TIMEOUT);
        }
        break;
      }
      tc_fence_after();
      const uint32_t t0 = tmem + (static_cast<uint32_t>(q * 32) << 16) + half * units * 8;
      long long hi[4][8], lo[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (u < units) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t v[4][8];
#pragma unroll
            for (int g = 0; g < 4; ++g) tmem_ld8_nowait(t0 + (4 * h + g) * nbr + u * 8, v[g]);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) (h == 0 ? hi : lo)[u][j] = join4(v[0][j], v[1][j], v[2][j], v[3][j]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty);
      tph ^= 1;
      // rows nu0 .. nu0 + 31, columns i0 .. of XT
      const long nu0 = static_cast<long>(M) * 128 + q * 32;
      const int i0 = p.bt.first(b) + half * units * 8;
      if (nu0 >= p.npad) continue;  // npad is a multiple of 64: the whole warp
      const double sb = p.scaleB[Q] * kJoined * p.up[nu0 + lane];
      double* out = p.XT + (nu0 + (lane >> 3)) * p.kdim + static_cast<long>(Q) * p.noccp + i0 + 2 * (lane & 7);
      const long step = 4 * p.kdim;
      const double2* sc = reinterpret_cast<const double2*>(p.scaleC + i0);
      uint32_t m = 0;
#pragma unroll
      for (int u = 0; u < 4; u += 2) {
        if (u < units) {
          const int w = units - u >= 2 ? 16 : 8;  // columns of this turn
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            if (j < w) {
              const double2 c = __ldg(sc + (u * 8 + j) / 2);
              const double x = join8(hi[u + j / 8][j % 8], lo[u + j / 8][j % 8]) * sb * c.x;
              const double y = join8(hi[u + j / 8][j % 8 + 1], lo[u + j / 8][j % 8 + 1]) * sb * c.y;
              m = max(m, max(magnitude(x), magnitude(y)));
              *reinterpret_cast<double2*>(mine + lane * kOutLd + j) = make_double2(x, y);
            }
          }
          __syncwarp();
          if (2 * (lane & 7) < w) {
            double* o = out + u * 8;
            const double* from = mine + (lane >> 3) * kOutLd + 2 * (lane & 7);
#pragma unroll
            for (int r = 0; r < 8; ++r, o += step, from += 4 * kOutLd)
              *reinterpret_cast<double2*>(o) = *reinterpret_cast<const double2*>(from);
          }
          __syncwarp();
        }
      }
      atomicMax(p.tops + (Q / p.qper) * (static_cast<long>(p.nb) * 128) + nu0 + lane, m);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  // looked up once (thread-safe static initialisation: contexts may live on several host threads)
  static const EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeTiledFn>(f);
    return static_cast<EncodeTiledFn>(nullptr);
  }();
  return fn;
}

// The digits of B as 8-byte words [block of any Q][digit][column group][256 words = 16 row groups], box x * y * 7.
bool map_digits(CUtensorMap* m, const void* base, uint64_t blocks, uint32_t x, uint32_t y) {
  const EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  cuuint64_t dims[4] = {256, 8, kDigits, blocks};
  cuuint64_t strides[3] = {2048, 16384, static_cast<cuuint64_t>(kSuper)};
  cuuint32_t box[4] = {x, y, kDigits, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// What Bexp holds.
struct BScales {
  double *scale, *down, *up;  // of the aux functions (value_scale), of the orbital functions
  int* ex;                    // exponents of the aux functions
  uint32_t* top;
  int* how;                   // kPlain, kScaled, kPlainNoTops
  float *e0, *e1;             // the balancing's logarithms
};
static size_t scales_bytes(long nq, long npad2) {
  return (round_up(nq, 2) + 2 * npad2) * sizeof(double) + (2 * nq + 1 + 2 * npad2) * sizeof(int);
}
static BScales scales_of(void* p, long nq, long npad2) {
  BScales s{};
  s.scale = static_cast<double*>(p);
  s.down = s.scale + round_up(nq, 2);  // read 16 bytes at a time
  s.up = s.down + npad2;
  s.ex = reinterpret_cast<int*>(s.up + npad2);
  s.top = reinterpret_cast<uint32_t*>(s.ex + nq);
  s.how = reinterpret_cast<int*>(s.top + nq);
  s.e0 = reinterpret_cast<float*>(s.how + 1);
  s.e1 = s.e0 + npad2;
  return s;
}

static size_t bdig_bytes(long nq, long nt) {
  const long nb = (nt + 1) / 2;
  return static_cast<size_t>(nq) * (nb * (nb + 1) / 2) * kSuper;
}

bool bdig_prepare(rijk_ctx* ctx) {
  // A recorded build reads B itself: digits formed in it would not be there before its replay, and digits formed
  // before it would be those of an earlier tensor in a replay after the next set-up.
  if (recording(ctx)) return false;
  if (ctx->have_bdig) return true;
  if (ctx->no_bdig || !encode_tiled()) return false;
  const long nb = (ctx->nt + 1) / 2, nsb = nb * (nb + 1) / 2;
  const size_t bytes = bdig_bytes(ctx->nq, ctx->nt);
  const std::string keep = ctx->last_error;  // running out of room here is no error
  auto no_room = [&]() {
    ctx->last_error = keep;
    drop_bdig(ctx, true);
    ctx->no_bdig = true;
    return false;
  };
  const long te = ctx->ntile * TILE2, npad2 = nb * 128;
  // The small buffers first: short of memory, `ensure` gives Bdig's back (drop_bdig) and still succeeds.
  if (ensure(ctx, ctx->Bexp, scales_bytes(ctx->nq, npad2), "digit scales of B") ||
      ensure(ctx, ctx->Btop, (te + ctx->nq) * sizeof(uint32_t), "magnitudes of B"))
    return no_room();
  if (ctx->Bdig.bytes < bytes) {
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    if (free_b + ctx->Bdig.bytes < bytes + total_b / 24) return no_room();
  }
  if (ensure(ctx, ctx->Bdig, bytes, "int8 digits of B")) return no_room();
  cudaStream_t s = ctx->stream;
  const BScales sc = scales_of(ctx->Bexp.p, ctx->nq, npad2);
  uint32_t* top = static_cast<uint32_t*>(ctx->Btop.p);
  const double* B = static_cast<const double*>(ctx->B.p);
  const unsigned q = static_cast<unsigned>(ctx->nq);
  if (!ctx->have_btop) {  // a tensor read from a file
    cudaMemsetAsync(top, 0, te * sizeof(uint32_t), s);
    k_element_max<<<dim3(static_cast<unsigned>(te / 512), static_cast<unsigned>(std::min<long>(ctx->nq, 16))), 256, 0, s>>>(
        B, ctx->nq, te, top);
  }
  const unsigned rows = static_cast<unsigned>((ctx->n + 7) / 8);
  cudaMemsetAsync(sc.e0, 0, ctx->n * sizeof(float), s);
  k_balance<<<rows, 256, 0, s>>>(top, ctx->n, nullptr, sc.e0, sc.e1);
  k_spread<<<1, 256, 0, s>>>(sc.e1, ctx->n, ctx->have_btop, sc.how);
  for (int i = 1; i < kBalanceSteps; ++i)
    k_balance<<<rows, 256, 0, s>>>(top, ctx->n, sc.how, i & 1 ? sc.e1 : sc.e0, i & 1 ? sc.e0 : sc.e1);
  k_balance_scales<<<static_cast<unsigned>(nb), 128, 0, s>>>(sc.e0, sc.e1, ctx->n, npad2, sc.how, sc.down, sc.up);
  cudaMemsetAsync(sc.top, 0, ctx->nq * sizeof(uint32_t), s);
  k_bmax<<<dim3(static_cast<unsigned>(std::min<long>(ctx->ntile, 8)), q), 256, 0, s>>>(B, ctx->ntile, sc.how, sc.down, sc.top);
  k_exponents<<<static_cast<unsigned>((ctx->nq + 255) / 256), 256, 0, s>>>(top + te, sc.top, sc.how, ctx->nq, sc.ex, sc.scale);
  k_slice_b<<<dim3(static_cast<unsigned>(nsb), q), 256, 0, s>>>(B, ctx->nt, te, nsb, sc.ex, sc.down,
                                                                 static_cast<uint8_t*>(ctx->Bdig.p));
  ctx->have_bdig = true;
  return true;
}

void drop_bdig(rijk_ctx* ctx, bool for_good) {
  ctx->no_bdig = ctx->no_bdig || (for_good && ctx->have_bdig);  // (without them it is memory of an earlier tensor)
  ctx->have_bdig = false;
  cudaStreamSynchronize(ctx->stream);
  release(ctx->Bdig);
}

void forget_bdig(rijk_ctx* ctx, long nq, long nt) {
  ctx->have_bdig = ctx->no_bdig = ctx->no_i8k = false;
  if (ctx->Bdig.p && ctx->Bdig.bytes != bdig_bytes(nq, nt)) drop_bdig(ctx, false);
}

int xform_i8_buffers(rijk_ctx* ctx, long noccp, long parts) {
  const long nk = (ctx->n + kChunk - 1) / kChunk, npad2 = round_up(ctx->npad, 128);
  int rc = ensure(ctx, ctx->Cdig, static_cast<size_t>(noccp) * kDigits * kChunk * nk + noccp * sizeof(double), "int8 digits of C");
  if (!rc) rc = ensure(ctx, ctx->Xtop, static_cast<size_t>(parts) * npad2 * sizeof(uint32_t), "part maxima");
  return rc;
}

int xform_i8(rijk_ctx* ctx, const double* MOp, long noccp, double* XT, long qper, long parts, cudaStream_t s) {
  const long nk = (ctx->n + kChunk - 1) / kChunk, nb = (ctx->nt + 1) / 2, nsb = nb * (nb + 1) / 2;
  const long units = noccp / 16;
  Batches bt;
  bt.nbatch = static_cast<int>((units + 3) / 4);
  bt.base = static_cast<int>(units / bt.nbatch);
  bt.extra = static_cast<int>(units % bt.nbatch);
  double* scaleC = static_cast<double*>(ctx->Cdig.p);  // the scales, then the digits
  uint8_t* C = reinterpret_cast<uint8_t*>(scaleC + noccp);
  uint32_t* tops = static_cast<uint32_t*>(ctx->Xtop.p);
  cudaMemsetAsync(tops, 0, static_cast<size_t>(parts) * nb * 128 * sizeof(uint32_t), s);
  const BScales sc = scales_of(ctx->Bexp.p, ctx->nq, nb * 128);
  k_slice_c<<<static_cast<unsigned>(units), 128, 0, s>>>(MOp, ctx->n, ctx->npad, nk, bt, sc.up, scaleC, C);
  CUtensorMap rows, cols;
  const uint64_t blocks = static_cast<uint64_t>(ctx->nq) * nsb;
  if (!map_digits(&rows, ctx->Bdig.p, blocks, 256, 2) || !map_digits(&cols, ctx->Bdig.p, blocks, 64, 8))
    return set_err(ctx, RIJK_ERR_CUDA, "tensor map encoding failed (digits of B)");
  XformI8Params p{};
  p.C = C;
  p.scaleB = sc.scale;
  p.scaleC = scaleC;
  p.up = sc.up;
  p.XT = XT;
  p.tops = tops;
  p.qper = qper;
  p.kdim = ctx->nq * noccp;
  p.npad = ctx->npad;
  p.nsb = nsb;
  p.naux = static_cast<int>(ctx->nq);
  p.nb = static_cast<int>(nb);
  p.nk = static_cast<int>(nk);
  p.noccp = static_cast<int>(noccp);
  p.bt = bt;
  p.err = static_cast<int*>(ctx->err.p);
  ensure_smem_limit(reinterpret_cast<const void*>(k_xform_i8), kXSmem);
  const long items = ctx->nq * nb * bt.nbatch;
  k_xform_i8<<<static_cast<unsigned>(std::min<long>(items, ctx->sms)), kXThreads, kXSmem, s>>>(rows, cols, p);
  return cuda_check(ctx, cudaGetLastError(), "int8 half-transform launch");
}

}  // namespace rijk
