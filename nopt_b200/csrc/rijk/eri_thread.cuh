// eri_thread.cuh — the three-centre integral kernel for spherical aux shells: a thread per aux shell.
//
// The Hermite expansion of a solid-harmonic Gaussian r^l Y_lm exp(-gamma r^2) about its own centre is the
// harmonic polynomial itself in the derivatives, times (2 gamma)^-l: every lower term cancels, because the
// polynomial's Laplacian vanishes.  An integral over one bra primitive pair p is then
//     (ab|m) = sum_tuv E^ab_tuv W_m[tuv],   W_m[tuv] = c (-1/2gamma)^l s_m sum_c q_mc R[tuv + c]
// with q_mc the integer coefficients of the polynomial, s_m its norm and E^ab the bra's spherical (or
// Cartesian) functions in Hermite Gaussians.
//
// One CTA of 64 threads takes a bra shell pair and a tile of 8 to 64 aux shells of one l (eri_tile); with fewer
// than 64, several threads share an aux shell and divide the bra functions between them (each forms R and W
// again, which costs no time on lanes that would idle).  The threads form E for each bra primitive
// pair in shared memory once, for all those aux shells; each thread then runs its aux shell: the Boys
// values, the R recursion in place in registers (entries in falling order: a layer's entry of order k reads
// only entries of order k - 1 and k - 2, not yet overwritten; local memory from total order 7 on), W, and
// the product with E, whose entries all threads read as 16-byte broadcasts.  la + lb and lc are template
// parameters, so the recursion and the harmonic sums are straight-line code without index tables.
//
// What bounds it: the FP64 pipe and its latency at 8 to 16 warps per SM.  Measured against a group of lanes per
// shell triple with everything in shared memory (k_eri, kept for (P|Q), Cartesian aux shells and la + lb > 6), whose
// Boys values one lane formed while the others waited and whose E was formed again for every aux shell: at
// (H2O)8 cc-pVTZ/cc-pVTZ-JKFIT all of (P|Q) and (mu nu|P) 31.8 -> 4.0 ms, (H2O)16
// cc-pVDZ/cc-pVDZ-JKFIT 32.7 -> 3.1 ms, (H2O)32 cc-pVTZ 1.02 -> 0.130 s.
#pragma once
#include <utility>

#include "eri_device.cuh"

namespace rijk {
namespace eri {

constexpr int NT = 64;        // threads of a CTA
constexpr int LAB_MAX = 6;    // la + lb handled here (f f)

// Hermite index -> (t, u, v), the order of tet_index
constexpr int dec_s(int e) {
  int s = 0;
  while ((s + 1) * (s + 2) * (s + 3) / 6 <= e) ++s;
  return s;
}
constexpr int dec_w(int e) {
  const int s = dec_s(e);
  int r = e - s * (s + 1) * (s + 2) / 6, w = 0;
  while ((w + 1) * (w + 2) / 2 <= r) ++w;
  return w;
}
constexpr int dec_v(int e) {
  const int s = dec_s(e), w = dec_w(e);
  return e - s * (s + 1) * (s + 2) / 6 - w * (w + 1) / 2;
}
constexpr int dec_t(int e) { return dec_s(e) - dec_w(e); }
constexpr int dec_u(int e) { return dec_w(e) - dec_v(e); }
constexpr int tetc(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
constexpr int tix(int t, int u, int v) {
  const int s = t + u + v, w = u + v;
  return s * (s + 1) * (s + 2) / 6 + w * (w + 1) / 2 + v;
}

// Integer coefficient of x^t y^u z^v in the real solid harmonic (l, m), m = -l .. l as row m + l (the standard
// Cartesian forms; Helgaker, Jorgensen, Olsen, Molecular Electronic-Structure Theory, table 6.3).
constexpr int harm(int l, int row, int t, int u, int v) {
  const int k = t * 100 + u * 10 + v;
  switch (l * 10 + row) {
    case 0: return 1;
    case 10: return k == 10 ? 1 : 0;
    case 11: return k == 1 ? 1 : 0;
    case 12: return k == 100 ? 1 : 0;
    case 20: return k == 110 ? 1 : 0;
    case 21: return k == 11 ? 1 : 0;
    case 22: return k == 2 ? 2 : (k == 200 || k == 20) ? -1 : 0;
    case 23: return k == 101 ? 1 : 0;
    case 24: return k == 200 ? 1 : k == 20 ? -1 : 0;
    case 30: return k == 210 ? 3 : k == 30 ? -1 : 0;
    case 31: return k == 111 ? 1 : 0;
    case 32: return k == 12 ? 4 : (k == 210 || k == 30) ? -1 : 0;
    case 33: return k == 3 ? 2 : (k == 201 || k == 21) ? -3 : 0;
    case 34: return k == 102 ? 4 : (k == 300 || k == 120) ? -1 : 0;
    case 35: return k == 201 ? 1 : k == 21 ? -1 : 0;
    case 36: return k == 300 ? 1 : k == 120 ? -3 : 0;
    case 40: return k == 310 ? 1 : k == 130 ? -1 : 0;
    case 41: return k == 211 ? 3 : k == 31 ? -1 : 0;
    case 42: return k == 112 ? 6 : (k == 310 || k == 130) ? -1 : 0;
    case 43: return k == 13 ? 4 : (k == 211 || k == 31) ? -3 : 0;
    case 44: return k == 4 ? 8 : (k == 202 || k == 22) ? -24 : (k == 400 || k == 40) ? 3 : k == 220 ? 6 : 0;
    case 45: return k == 103 ? 4 : (k == 301 || k == 121) ? -3 : 0;
    case 46: return k == 202 ? 6 : k == 22 ? -6 : k == 400 ? -1 : k == 40 ? 1 : 0;
    case 47: return k == 301 ? 1 : k == 121 ? -3 : 0;
    case 48: return (k == 400 || k == 40) ? 1 : k == 220 ? -6 : 0;
    default: return 0;
  }
}

template <int E>
__device__ __forceinline__ void r_entry(double* R, double X, double Y, double Z) {
  constexpr int t = dec_t(E), u = dec_u(E), v = dec_v(E);
  if constexpr (t > 0) {
    if constexpr (t > 1)
      R[E] = fma(X, R[tix(t - 1, u, v)], (t - 1) * R[tix(t - 2, u, v)]);
    else
      R[E] = X * R[tix(t - 1, u, v)];
  } else if constexpr (u > 0) {
    if constexpr (u > 1)
      R[E] = fma(Y, R[tix(t, u - 1, v)], (u - 1) * R[tix(t, u - 2, v)]);
    else
      R[E] = Y * R[tix(t, u - 1, v)];
  } else {
    if constexpr (v > 1)
      R[E] = fma(Z, R[tix(t, u, v - 1)], (v - 1) * R[tix(t, u, v - 2)]);
    else
      R[E] = Z * R[tix(t, u, v - 1)];
  }
}

template <int CNT, int... E>
__device__ __forceinline__ void r_layer(double* R, double X, double Y, double Z, std::integer_sequence<int, E...>) {
  (r_entry<CNT - 1 - E>(R, X, Y, Z), ...);  // entries CNT - 1 .. 1
}

// R_tuv of t + u + v <= L from G[n] = (-2 alpha)^n F_n(T)
template <int L, int N = L>
__device__ __forceinline__ void r_layers(double* R, const double* G, double X, double Y, double Z) {
  constexpr int CNT = tetc(L - N);
  if constexpr (CNT > 1) r_layer<CNT>(R, X, Y, Z, std::make_integer_sequence<int, CNT - 1>());
  R[0] = G[N];
  if constexpr (N > 0) r_layers<L, N - 1>(R, G, X, Y, Z);
}

// sum_c q_c R[h + c] over the Cartesians c of l
template <int H, int LC, int ROW, int C = 0>
__device__ __forceinline__ double w_entry(const double* R) {
  constexpr int NC = (LC + 1) * (LC + 2) / 2;
  // Cartesian C of l: the Hermite entries of order LC in tet order
  constexpr int e = LC == 0 ? 0 : tetc(LC - 1) + C;
  constexpr int q = harm(LC, ROW, dec_t(e), dec_u(e), dec_v(e));
  constexpr int at = tix(dec_t(H) + dec_t(e), dec_u(H) + dec_u(e), dec_v(H) + dec_v(e));
  double s = 0.0;
  if constexpr (C + 1 < NC) s = w_entry<H, LC, ROW, C + 1>(R);
  if constexpr (q != 0) s = fma(static_cast<double>(q), R[at], s);
  return s;
}
template <int LC, int ROW, int... H>
__device__ __forceinline__ void w_all(const double* R, double f, double* W, std::integer_sequence<int, H...>) {
  ((W[H] = f * w_entry<H, LC, ROW>(R)), ...);
}

// F_0 .. F_L of T into F
template <int L>
__device__ __forceinline__ void boys(double T, const double* __restrict__ tab, double* F) {
  constexpr double TMAX = gto_tab::BOYS_TMAX;
  constexpr int NPER = gto_tab::BOYS_NPER, MTAB = gto_tab::BOYS_MTAB;
  const double e = exp(-T);
  if (T < TMAX - 0.5 / NPER) {
    const int i = static_cast<int>(T * NPER + 0.5);
    const double dt = static_cast<double>(i) / NPER - T;
    const double* row = tab + static_cast<long>(i) * MTAB + L;
    double f = __ldg(row + 6) * (1.0 / 720.0);
    f = fma(f, dt, __ldg(row + 5) * (1.0 / 120.0));
    f = fma(f, dt, __ldg(row + 4) * (1.0 / 24.0));
    f = fma(f, dt, __ldg(row + 3) * (1.0 / 6.0));
    f = fma(f, dt, __ldg(row + 2) * 0.5);
    f = fma(f, dt, __ldg(row + 1));
    f = fma(f, dt, __ldg(row));
    F[L] = f;
#pragma unroll
    for (int m = L; m > 0; --m) F[m - 1] = fma(2.0 * T, F[m], e) * (1.0 / (2 * m - 1));
  } else {
    const double it = 0.5 / T;
    F[0] = 0.5 * sqrt(gto_tab::PI / T);
#pragma unroll
    for (int m = 0; m < L; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) * it;
  }
}

// v[m] = sum_h E[ab][h] W[h] for one aux function: two partial sums
template <int NH>
__device__ __forceinline__ double dot_row(const double* __restrict__ E, const double* W) {
  double a = 0.0, b = 0.0;
#pragma unroll
  for (int h = 0; h + 1 < NH; h += 2) {
    const double2 e = *reinterpret_cast<const double2*>(E + h);
    a = fma(e.x, W[h], a);
    b = fma(e.y, W[h + 1], b);
  }
  if (NH & 1) a = fma(E[NH - 1], W[NH - 1], a);
  return a + b;
}

// The aux functions ROW .. 2 LC of one thread: out(ab, m, value) for its bra function pairs ab0, ab0 + dab, ..
template <int LAB, int LC, int ROW, typename Out>
__device__ __forceinline__ void rows(const double* R, double f, const double* __restrict__ norm,
                                     const double* __restrict__ E, int ab0, int dab, int nab, Out out) {
  constexpr int NH = tetc(LAB), NHP = (NH + 1) & ~1;
  double W[NH];
  w_all<LC, ROW>(R, f * __ldg(norm + ROW), W, std::make_integer_sequence<int, NH>());
#pragma unroll 1
  for (int ab = ab0; ab < nab; ab += dab) out(ab, ROW, dot_row<NH>(E + ab * NHP, W));
  if constexpr (ROW < 2 * LC) rows<LAB, LC, ROW + 1>(R, f, norm, E, ab0, dab, nab, out);
}

// s s: every aux function of the thread, added to acc
template <int LC, int ROW>
__device__ __forceinline__ void sums(const double* R, double f, const double* __restrict__ norm, double* acc) {
  acc[ROW] = fma(f * __ldg(norm + ROW), w_entry<0, LC, ROW>(R), acc[ROW]);
  if constexpr (ROW < 2 * LC) sums<LC, ROW + 1>(R, f, norm, acc);
}

template <int LAB, int LC>
__global__ void __launch_bounds__(NT) k_eri_thread(const EriLaunch P) {
  constexpr int L = LAB + LC, NR = tetc(L), NH = tetc(LAB), NHP = (NH + 1) & ~1, NF = 2 * LC + 1;
  extern __shared__ __align__(16) double sm[];
  double* E1 = sm;                      // 3 x (la+1)(lb+1)(LAB+1)
  double* E = sm + P.e1size;            // nab x NHP
  const int tid = threadIdx.x;
  const int tile = P.tile, kt = tid & (tile - 1), part = tid / tile, parts = NT / tile;
  double* acc = E + P.esize;            // nab x tile NF, contracted pairs only
  const int arow = tile * NF;
  const long ntile = (P.nket + tile - 1) / tile;
  const long ip = blockIdx.x / ntile;
  const long k0 = (blockIdx.x - ip * ntile) * tile;
  const int2 pair = P.pairs[ip];
  const EriShell A = P.bra[pair.x];
  const EriShell B = P.bra[pair.y];
  const bool live = k0 + kt < P.nket;
  const EriShell C = P.ket[P.kets[live ? k0 + kt : P.nket - 1]];
  const int la = A.l, lb = B.l, nfb = B.nfunc, nab = A.nfunc * nfb;
  // the tile's largest primitive count: the aux shells are sorted by it
  const int nprim_k = P.ket[P.kets[min(k0 + tile, P.nket) - 1]].nprim;
  const bool direct = A.nprim * B.nprim * nprim_k == 1;
  const double* norm = P.harm_norm + LC * 9;
  const double two_pi_25 = 2.0 * 17.493418327624862;  // 2 pi^(5/2)

  // one value of the thread's aux function m and the bra functions ab to its place
  auto store = [&](int ab, long col, double v) {
    const int fa = ab / nfb, fb = ab - fa * nfb;
    const long mu = A.off + fa, nu = B.off + fb;
    if (P.mode == 0) {
      if (pair.x == pair.y && nu > mu) return;
      const long hi = mu > nu ? mu : nu, lo = mu > nu ? nu : mu;
      if (hi < P.mu0 || hi >= P.mu1) return;
      P.out[(hi * (hi + 1) / 2 + lo - P.rowbase) * P.ld + col] = v;
    } else {
      if (mu >= P.mu0 && mu < P.mu1) P.out[((mu - P.rowbase) * P.n + nu) * P.ld + col] = v;
      if (pair.x != pair.y && nu >= P.mu0 && nu < P.mu1) P.out[((nu - P.rowbase) * P.n + mu) * P.ld + col] = v;
    }
  };

  double racc[NF] = {};  // LAB = 0: the sums stay in registers, E is one number
  if (LAB > 0 && !direct) {
    for (int o = tid; o < nab * arow; o += NT) acc[o] = 0.0;
    __syncthreads();
  }
  const double ABx = A.x - B.x, ABy = A.y - B.y, ABz = A.z - B.z;
  const double r2 = ABx * ABx + ABy * ABy + ABz * ABz;
  bool any = false;
  for (int ij = 0; ij < A.nprim * B.nprim; ++ij) {
    const int i = ij / B.nprim, j = ij - i * B.nprim;
    const double a = P.bexp[A.prim0 + i], b = P.bexp[B.prim0 + j];
    const double cc = P.bcoef[A.prim0 + i] * P.bcoef[B.prim0 + j];
    const double p = a + b, ip1 = 1.0 / p;
    const double K = exp(-(a * b * ip1) * r2);
    if (fabs(cc * K) < 1e-22) continue;  // contributes below double precision (host rule); the same for all threads
    any = true;
    const double Px = (a * A.x + b * B.x) * ip1, Py = (a * A.y + b * B.y) * ip1, Pz = (a * A.z + b * B.z) * ip1;
    if constexpr (LAB > 0) {
      // E1[d][i][j][t]: 1-D Hermite expansion of the primitive product
      const int ts = LAB + 1, n1 = (la + 1) * (lb + 1) * ts;
      __syncthreads();  // the previous primitive pair's readers of E are done
      if (tid < 3) {
        const double pd = tid == 0 ? Px : (tid == 1 ? Py : Pz);
        const double ad = tid == 0 ? A.x : (tid == 1 ? A.y : A.z);
        const double bd = tid == 0 ? B.x : (tid == 1 ? B.y : B.z);
        const double xpa = pd - ad, xpb = pd - bd, o2p = 0.5 * ip1;
        double* e1 = E1 + tid * n1;
        e1[0] = tid == 0 ? K * cc : 1.0;
        for (int q = 0; q <= la; ++q)
          for (int r = 0; r <= lb; ++r) {
            if (q + r == 0) continue;
            const double* src = e1 + (r > 0 ? (q * (lb + 1) + r - 1) : ((q - 1) * (lb + 1))) * ts;
            double* dst = e1 + (q * (lb + 1) + r) * ts;
            const double x = r > 0 ? xpb : xpa;
            const int o = q + r;  // the source has entries t <= o - 1
            for (int t = 0; t <= o; ++t) {
              double v = t < o ? x * src[t] : 0.0;
              if (t + 1 < o) v += (t + 1) * src[t + 1];
              if (t > 0) v += o2p * src[t - 1];
              dst[t] = v;
            }
          }
      }
      __syncthreads();
      // E[ab][tuv] over the spherical (or Cartesian) functions of the pair
      for (int o = tid; o < nab * NH; o += NT) {
        const int ab = o / NH, h = o - ab * NH;
        const int c = __ldg(P.tuv + h);
        const int t = c & 0xff, u = (c >> 8) & 0xff, v = c >> 16;
        const int fa = ab / nfb, fb = ab - fa * nfb;
        const SphRow& ra = P.sph_rows[(A.pure ? 0 : 1) * SPH_ROWS + la * 15 + fa];
        const SphRow& rb = P.sph_rows[(B.pure ? 0 : 1) * SPH_ROWS + lb * 15 + fb];
        double s = 0.0;
        for (int x = 0; x < ra.n; ++x) {
          const int ka = ra.cart[x];
          const int ax = ka & 15, ay = (ka >> 4) & 15, az = ka >> 8;
          for (int y = 0; y < rb.n; ++y) {
            const int kb = rb.cart[y];
            const int bx = kb & 15, by = (kb >> 4) & 15, bz = kb >> 8;
            if (t > ax + bx || u > ay + by || v > az + bz) continue;
            s += ra.c[x] * rb.c[y] * E1[(ax * (lb + 1) + bx) * ts + t] * E1[n1 + (ay * (lb + 1) + by) * ts + u] *
                 E1[2 * n1 + (az * (lb + 1) + bz) * ts + v];
          }
        }
        E[ab * NHP + h] = s;
      }
      __syncthreads();
    }
    const double X = Px - C.x, Y = Py - C.y, Z = Pz - C.z;
    const double d2 = X * X + Y * Y + Z * Z;
#pragma unroll 1
    for (int k = 0; k < nprim_k; ++k) {
      const bool has = k < C.nprim;
      const double gam = has ? P.kexp[C.prim0 + k] : 1.0, ck = has ? P.kcoef[C.prim0 + k] : 0.0;
      const double rs = rsqrt(p + gam), al = p * gam * rs * rs, ig = 1.0 / gam;
      double f = two_pi_25 * ip1 * ig * rs * ck;
      if (LAB == 0) f *= K * cc;
      const double o2g = -0.5 * ig;
#pragma unroll
      for (int q = 0; q < LC; ++q) f *= o2g;
      double G[L + 1];
      boys<L>(al * d2, P.boys, G);
      const double m2a = -2.0 * al;
      double pw = 1.0;
#pragma unroll
      for (int m = 1; m <= L; ++m) {
        pw *= m2a;
        G[m] *= pw;
      }
      double R[NR];
      r_layers<L>(R, G, X, Y, Z);
      if constexpr (LAB == 0) {
        sums<LC, 0>(R, f, norm, racc);
      } else if (direct) {
        rows<LAB, LC, 0>(R, f, norm, E, part, parts, nab, [&](int ab, int m, double v) {
          if (live) store(ab, C.off + m, v);
        });
      } else {
        double* mine = acc + kt * NF;
        rows<LAB, LC, 0>(R, f, norm, E, part, parts, nab, [&](int ab, int m, double v) { mine[ab * arow + m] += v; });
      }
    }
  }
  if (!live) return;
  if constexpr (LAB == 0) {
    if (part == 0)
#pragma unroll
      for (int m = 0; m < NF; ++m) store(0, C.off + m, racc[m]);
  } else if (!direct) {
    for (int ab = part; ab < nab; ab += parts)
#pragma unroll
      for (int m = 0; m < NF; ++m) store(ab, C.off + m, acc[ab * arow + kt * NF + m]);
  } else if (!any) {  // every primitive pair is below double precision
    for (int ab = part; ab < nab; ab += parts)
#pragma unroll
      for (int m = 0; m < NF; ++m) store(ab, C.off + m, 0.0);
  }
}

}  // namespace eri
}  // namespace rijk

namespace rijk {
namespace eri {

// One launch of the class (la + lb = LAB, LC) over P.npair bra pairs and P.nket aux shells.
template <int LAB, int LC>
cudaError_t launch(const EriLaunch& P, size_t smem, cudaStream_t s) {
  const void* fn = reinterpret_cast<const void*>(k_eri_thread<LAB, LC>);
  const cudaError_t e = ensure_smem_limit(fn, smem);
  if (e != cudaSuccess) return e;
  // P.npair * tiles is far below 2^31: a call's row block holds at most 2 GiB of integrals
  const long blocks = P.npair * ((P.nket + P.tile - 1) / P.tile);
  k_eri_thread<LAB, LC><<<static_cast<unsigned>(blocks), NT, smem, s>>>(P);
  return cudaGetLastError();
}

template <int LC>
cudaError_t launch_lc(int lab, const EriLaunch& P, size_t smem, cudaStream_t s) {
  switch (lab) {
    case 0: return launch<0, LC>(P, smem, s);
    case 1: return launch<1, LC>(P, smem, s);
    case 2: return launch<2, LC>(P, smem, s);
    case 3: return launch<3, LC>(P, smem, s);
    case 4: return launch<4, LC>(P, smem, s);
    case 5: return launch<5, LC>(P, smem, s);
    default: return launch<6, LC>(P, smem, s);
  }
}

}  // namespace eri
}  // namespace rijk
