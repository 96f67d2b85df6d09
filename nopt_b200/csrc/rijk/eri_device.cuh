// eri_device.cuh — what the integral kernels share: shell records, the launch's arguments, index helpers.
#pragma once
#include <cuda_runtime.h>

#include "gto_tables.h"
#include "rijk_internal.h"

namespace rijk {
namespace eri {

using gto_tab::LMAX;
constexpr int LTOT = 3 * LMAX;
constexpr int TET_MAX = (LTOT + 1) * (LTOT + 2) * (LTOT + 3) / 6;  // 455 entries with t+u+v <= 12
constexpr int NSPH = 245;            // sum over l <= 4 of (2l+1) ncart(l)
constexpr int TERM_KEYS = 2 * (LMAX + 1);
constexpr int TERM_STRIDE = 16;      // per key: offsets of m = 0 .. 15 (ncart(4) = 15) and the end

struct EriShell {
  double x, y, z;
  int l, nprim, prim0, off;
  int nfunc, pure, pad0, pad1;
};

// A bra function as Cartesian terms: spherical rows (at most 6 terms for l <= 4), or one Cartesian.
constexpr int SPH_ROWS = (LMAX + 1) * 15;  // row l * 15 + function; the Cartesian rows follow
struct SphRow {
  int n;
  int cart[6];  // lx | ly << 4 | lz << 8
  double c[6];
};

struct EriTerm {
  short t, u, v, j;  // Hermite index of the term and the power j of (2 gamma)^-1
  int pad;
  double d;
};

struct EriLaunch {
  const EriShell* bra;
  const double* bexp;
  const double* bcoef;
  const int2* pairs;
  long npair;
  const EriShell* ket;
  const double* kexp;
  const double* kcoef;
  const int* kets;
  long nket;
  int la, lb, lc, G;
  int gsize;        // doubles of shared memory per group
  int mode;         // 0 packed rows (hi(hi+1)/2 + lo), 1 full rows (mu n + nu), 2 square (P, Q)
  long mu0, mu1;    // rows written (modes 0, 1)
  long rowbase;     // row index subtracted before storing
  long n;           // orbital functions (mode 1 row pitch in pairs)
  long ld;          // element pitch between stored rows
  double* out;
  const double* boys;
  const double* sph;
  const EriTerm* terms;
  const int* term_off;
  const int* tuv;
  const int* cart;
  const SphRow* sph_rows;   // [spherical, Cartesian][SPH_ROWS]
  const double* harm_norm;  // [l][9]: norms of the integer harmonics (harm in eri_thread.cuh)
  int e1size, esize;        // k_eri_thread: doubles of its 1-D and pair expansions in shared memory
  int tile;                 // k_eri_thread: aux shells of a CTA, a power of two up to its 64 threads
};

__host__ __device__ inline int tet(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
__host__ __device__ inline int ncart_d(int l) { return (l + 1) * (l + 2) / 2; }
__device__ __forceinline__ int tet_index(int t, int u, int v) {
  const int s = t + u + v, w = u + v;
  return s * (s + 1) * (s + 2) / 6 + w * (w + 1) / 2 + v;
}
__host__ __device__ inline int sph_off(int l) {
  int o = 0;
  for (int k = 0; k < l; ++k) o += (2 * k + 1) * ncart_d(k);
  return o;
}

}  // namespace eri
}  // namespace rijk
