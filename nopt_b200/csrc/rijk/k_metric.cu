// k_metric.cu — K1, the metric contraction B^Q_{mu nu} = sum_P M_QP (P|mu nu).
//
// Replaces the reference's per-iteration metric products (V^-1/2 applied to RI_J twice,
// src/RI.cpp:128-138, and to the half-transformed tensor, src/RI.cpp:152-156): the metric
// factor M (V^-1/2 or L^-1) is applied once per geometry and B is kept in HBM.
//
// GEMM: rows Q (64 per CTA), columns = 64 of the pairs that are stored, contraction over P in 32-wide chunks.  M is
// zero-padded to nauxp x nauxp and the raw integrals carry row pitch nauxp, so chunks never straddle.
// The raw integrals arrive in row-blocks of whole tile rows (I in [I0, I1)); the columns are counted through them:
// packed layout, all pairs mu >= nu, each a raw row, the diagonal tiles' other halves written from the same sums;
// NOPT full-square layout, all nu of the tiles up to the diagonal one, each from its own raw row.
//
// What bounds it: the FP64 tensor pipe, 35.5 TFLOP/s here.  Columns were once the rows of the stored tiles, which
// also multiplied the padding past n and the upper halves of the diagonal tiles: a third of the work at n = 464
// (147,456 columns against 107,880 pairs), 3 % at n = 1856.  Measured, packed: (H2O)8
// cc-pVTZ 11.7 -> 8.75 ms, (H2O)6 cc-pVDZ 0.79 -> 0.38 ms.
#include <algorithm>

#include "gemm_f64.cuh"
#include "i8_digits.cuh"
#include "rijk_internal.h"

namespace rijk {

constexpr int K1_THREADS = 128;

// Column c of the tile rows from I0 on -> (mu, nu).
__device__ __forceinline__ void k1_column(long c, int layout, long n, long I0, long& mu, long& nu) {
  if (layout == RIJK_LAYOUT_NOPT_FULL) {
    // tile row I has 64 rows of min(n, 64 (I + 1)) columns, so those before it have 64 x 64 a tile
    long I, J;
    tri_decode(c / TILE2 + I0 * (I0 + 1) / 2, I, J);
    const long rem = c - (I * (I + 1) / 2 - I0 * (I0 + 1) / 2) * TILE2;
    const long w = n < (I + 1) * TILE ? n : (I + 1) * TILE;
    mu = I * TILE + rem / w;
    nu = rem % w;
  } else {
    tri_decode(c + I0 * TILE * (I0 * TILE + 1) / 2, mu, nu);
  }
}

__global__ void __launch_bounds__(K1_THREADS)
    k_metric_contract(const double* __restrict__ M, long nauxp, long mrows, const double* __restrict__ I3, int layout,
                      long n, long naux, long I0, long ncol, double* __restrict__ B, long tile_elems, long tri,
                      uint32_t* __restrict__ top) {
  extern __shared__ __align__(16) double smem_k1[];
  double* sA[2] = {smem_k1, smem_k1 + 64 * LDK};
  double* sB[2] = {smem_k1 + 2 * 64 * LDK, smem_k1 + 3 * 64 * LDK};
  __shared__ long rowoff[64];  // raw row of each column, -1 past the last
  __shared__ long dst[64];     // its element of a tile set
  __shared__ long mirror[64];  // and the transposed one, where the column stands for both; -1 otherwise

  const long q0 = static_cast<long>(blockIdx.y) * 64;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;

  if (tid < 64) {
    const long c = static_cast<long>(blockIdx.x) * 64 + tid;
    long off = -1, d = -1, m = -1;
    if (c < ncol) {
      long mu, nu;
      k1_column(c, layout, n, I0, mu, nu);
      const long I = mu / TILE, J = nu / TILE, r = mu % TILE, q = nu % TILE, t = I * (I + 1) / 2 + J;
      d = t * TILE2 + r * TILE + q;
      if (layout == RIJK_LAYOUT_NOPT_FULL) {
        off = (mu - I0 * TILE) * n + nu;
      } else {
        off = c;
        if (I == J && r != q) m = t * TILE2 + q * TILE + r;
      }
    }
    rowoff[tid] = off;
    dst[tid] = d;
    mirror[tid] = m;
  }
  __syncthreads();

  auto load = [&](int stage, long p0) {
    // A: M rows q0..q0+63, cols p0..p0+31 ; B: raw rows rowoff[c], cols p0..p0+31
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      int idx = tid + it * K1_THREADS;  // 0..1023
      int row = idx >> 4, seg = idx & 15;
      long q = q0 + row;
      const double* src = M + q * nauxp + p0 + seg * 2;
      cp_async16(&sA[stage][row * LDK + seg * 2], q < mrows ? src : M, q < mrows);
      long ro = rowoff[row];
      const double* srcb = I3 + (ro >= 0 ? ro : 0) * nauxp + p0 + seg * 2;
      cp_async16(&sB[stage][row * LDK + seg * 2], srcb, ro >= 0);
    }
  };

  double acc[4][4][2];
  zero_acc(acc);
  // tri >= 0: M is lower triangular (the Cholesky factor's inverse), its rows starting at global row
  // tri, so rows q0 .. q0 + 63 hold zeros past column tri + q0 + 63 and the chunks beyond add nothing
  const long nk = tri < 0 ? nauxp / KC : std::min(nauxp / KC, (tri + q0 + 64 + KC - 1) / KC);
  load(0, 0);
  cp_async_commit();
  for (long kc = 0; kc < nk; ++kc) {
    if (kc + 1 < nk) {
      load(static_cast<int>((kc + 1) & 1), (kc + 1) * KC);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    warp_mma_chunk<4, 4, true>(acc, sA[kc & 1], sB[kc & 1], wm * 32, wn * 32, lane);
    __syncthreads();
  }

  const int g = lane >> 2, tq = lane & 3;
  uint32_t m[4][2] = {};  // of this thread's 8 columns
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    long q = q0 + wm * 32 + i * 8 + g;
    uint32_t mq = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = wn * 32 + j * 8 + 2 * tq + e;
        const double x = acc[i][j][e];
        if (q < naux && dst[c] >= 0) {
          B[q * tile_elems + dst[c]] = x;
          if (mirror[c] >= 0) B[q * tile_elems + mirror[c]] = x;
          m[j][e] = max(m[j][e], magnitude(x));
          mq = max(mq, magnitude(x));
        }
      }
    }
    mq = max(mq, __shfl_xor_sync(0xffffffffu, mq, 1));
    mq = max(mq, __shfl_xor_sync(0xffffffffu, mq, 2));
    if (tq == 0 && q < naux) atomicMax(top + tile_elems + q, mq);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) m[j][e] = max(m[j][e], __shfl_xor_sync(0xffffffffu, m[j][e], o));
      const long d = dst[wn * 32 + j * 8 + 2 * tq + e];
      if (g == 0 && d >= 0) atomicMax(top + d, m[j][e]);
    }
}

// I3 holds the tile rows I in [I0, I1): full layout rows (mu - I0*64)*n + nu, packed layout
// pair rows starting at pair_base = (I0*64)(I0*64+1)/2.
void launch_metric_contract_chunk(const double* M, long nauxp, long mrows, const double* I3, int layout, long n,
                                  long naux, long nt, long I0, long I1, double* B, uint32_t* top, cudaStream_t s,
                                  long tri) {
  const long ntile = nt * (nt + 1) / 2;
  const long mu0 = I0 * TILE, mu1 = std::min(I1 * TILE, n);
  long ncol;
  if (layout == RIJK_LAYOUT_NOPT_FULL) {
    const long whole = n / TILE < I1 ? n / TILE : I1;  // tile rows of 64 rows; a last one may have fewer
    ncol = (tri_index(std::max(whole, I0), 0) - tri_index(I0, 0)) * TILE2 + (mu1 - std::max(whole, I0) * TILE) * n;
  } else {
    ncol = mu1 * (mu1 + 1) / 2 - mu0 * (mu0 + 1) / 2;
  }
  dim3 grid(static_cast<unsigned>((ncol + 63) / 64), static_cast<unsigned>((naux + 63) / 64));
  const size_t smem = 4 * 64 * LDK * sizeof(double);
  ensure_smem_limit(reinterpret_cast<const void*>(k_metric_contract), smem);
  k_metric_contract<<<grid, K1_THREADS, smem, s>>>(M, nauxp, mrows, I3, layout, n, naux, I0, ncol, B, ntile * TILE2, tri,
                                                   top);
}

}  // namespace rijk
