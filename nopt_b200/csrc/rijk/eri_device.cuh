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
constexpr int LEX_STRIDE = 84;       // entries with t+u+v <= 6
constexpr int TERM_STRIDE = 16;      // per key: offsets of m = 0 .. 15 (ncart(4) = 15) and the end

struct EriShell {
  double x, y, z;
  int l, nprim, prim0, off;
  int nfunc, pure, pad0, pad1;
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
  const int* lex;           // [la + lb][LEX_STRIDE]: (t, u, v) in k_eri_thread's order, t | u << 4 | v << 8
  int e1size, esize;        // k_eri_thread: doubles of its 1-D and pair expansions in shared memory
  bool thread_terms;        // k_eri_thread may run (its compiled-in term lists are the table's)
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

// F_m(T), m = 0 .. L, exactly as the host engine evaluates it (Taylor about the nearest grid
// point, downward recursion; F_0 and upward recursion past the grid).
__device__ __forceinline__ void boys_eval(int L, double T, const double* __restrict__ tab, double* F) {
  constexpr double TMAX = gto_tab::BOYS_TMAX;
  constexpr int NPER = gto_tab::BOYS_NPER, MTAB = gto_tab::BOYS_MTAB;
  if (T < TMAX - 0.5 / NPER) {
    const int i = static_cast<int>(T * NPER + 0.5);
    const double dt = static_cast<double>(i) / NPER - T;
    const double* row = tab + static_cast<long>(i) * MTAB;
    double f = __ldg(row + L + 6);
    f = __ldg(row + L + 5) + f * dt / 6.0;
    f = __ldg(row + L + 4) + f * dt / 5.0;
    f = __ldg(row + L + 3) + f * dt / 4.0;
    f = __ldg(row + L + 2) + f * dt / 3.0;
    f = __ldg(row + L + 1) + f * dt / 2.0;
    f = __ldg(row + L) + f * dt;
    F[L] = f;
    const double e = exp(-T);
    for (int m = L; m > 0; --m) F[m - 1] = (2.0 * T * F[m] + e) / (2 * m - 1);
  } else {
    const double e = exp(-T);
    F[0] = 0.5 * sqrt(gto_tab::PI / T);
    for (int m = 0; m < L; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) / (2.0 * T);
  }
}

// The same with L a template parameter, F in registers.
template <int L>
__device__ __forceinline__ void boys_eval_l(double T, const double* __restrict__ tab, double* F) {
  constexpr double TMAX = gto_tab::BOYS_TMAX;
  constexpr int NPER = gto_tab::BOYS_NPER, MTAB = gto_tab::BOYS_MTAB;
  if (T < TMAX - 0.5 / NPER) {
    const int i = static_cast<int>(T * NPER + 0.5);
    const double dt = static_cast<double>(i) / NPER - T;
    const double* row = tab + static_cast<long>(i) * MTAB;
    double f = __ldg(row + L + 6);
    f = __ldg(row + L + 5) + f * dt / 6.0;
    f = __ldg(row + L + 4) + f * dt / 5.0;
    f = __ldg(row + L + 3) + f * dt / 4.0;
    f = __ldg(row + L + 2) + f * dt / 3.0;
    f = __ldg(row + L + 1) + f * dt / 2.0;
    f = __ldg(row + L) + f * dt;
    F[L] = f;
    const double e = exp(-T);
#pragma unroll
    for (int m = L; m > 0; --m) F[m - 1] = (2.0 * T * F[m] + e) / (2 * m - 1);
  } else {
    const double e = exp(-T);
    F[0] = 0.5 * sqrt(gto_tab::PI / T);
#pragma unroll
    for (int m = 0; m < L; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) / (2.0 * T);
  }
}

// 1-D Hermite expansion E[i][j][t] of a primitive product, i <= la, j <= lb, t < ts (= la+lb+2).
__device__ __forceinline__ void hermite_1d_dev(int la, int lb, double p, double xpa, double xpb, double k0, double* E, int ts) {
  const double o2p = 0.5 / p;
  auto at = [&](int i, int j, int t) -> double& { return E[(i * (lb + 1) + j) * ts + t]; };
  for (int k = 0; k < (la + 1) * (lb + 1) * ts; ++k) E[k] = 0.0;
  at(0, 0, 0) = k0;
  for (int i = 0; i < la; ++i)
    for (int t = 0; t <= i + 1; ++t) {
      double v = xpa * at(i, 0, t) + (t + 1) * at(i, 0, t + 1);
      if (t > 0) v += o2p * at(i, 0, t - 1);
      at(i + 1, 0, t) = v;
    }
  for (int i = 0; i <= la; ++i)
    for (int j = 0; j < lb; ++j)
      for (int t = 0; t <= i + j + 1; ++t) {
        double v = xpb * at(i, j, t) + (t + 1) * at(i, j, t + 1);
        if (t > 0) v += o2p * at(i, j, t - 1);
        at(i, j + 1, t) = v;
      }
}

}  // namespace eri
}  // namespace rijk
