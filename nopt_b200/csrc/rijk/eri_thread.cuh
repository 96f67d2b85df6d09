// eri_thread.cuh — the three-centre integral kernel for uncontracted spherical aux shells: a thread per aux shell.
//
// One CTA of 64 threads takes a bra shell pair and a tile of 8 to 64 aux shells of one l (eri_tile); with fewer
// than 64, several threads share an aux shell and divide the bra functions between them (each forms R and W
// again, which costs no time on lanes that would idle).  For each bra primitive pair the threads form the products
// of its Hermite expansions, [Cartesian pair][tuv], in shared memory once for all those aux shells; each thread
// then runs its aux shell: the Boys values, the R recursion in place in registers (entries in falling order: a
// layer's entry of order k reads only entries of order k - 1 and k - 2, not yet overwritten; local memory from
// total order 7 on), the aux Hermite sums W, and their product with the expansions, whose entries all threads
// read as 16-byte broadcasts.  la + lb and lc are template parameters, so the recursion and the aux sums are
// straight-line code without index tables.
//
// The operations on one integral and their order are k_eri's, so both give the same bits: the split-BF16 copy of
// the fitted tensor rounds it, and integrals that differ in their last bits moved single elements of mixed J and K
// by 1e-7.  What k_eri spent its time on was not these operations: one lane of a group formed the Boys values while
// the others waited, every stage ran through shared memory with a barrier, and the bra's expansion was formed
// again for every aux shell.  (P|Q), Cartesian or contracted aux shells and la + lb > 6 stay there.
// What bounds this kernel: the FP64 pipe and its latency at 8 to 16 warps per SM.  Measured, all classes of one
// build: (H2O)8 cc-pVTZ 31.8 -> 6.5 ms, (H2O)32 cc-pVTZ 1.02 -> 0.234 s.
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

// The aux Hermite terms of a spherical function, in the order of the term table (t, then u, then v rising): the
// harmonic itself, and the places where the table's lower terms cancel to a last bit instead of to zero.
constexpr bool is_term(int l, int row, int t, int u, int v) {
  if (t + u + v == l) return harm(l, row, t, u, v) != 0;
  const int k = t * 100 + u * 10 + v;
  switch (l * 10 + row) {
    case 32: return k == 10;
    case 34: return k == 100;
    case 42: return k == 110;
    case 43: return k == 11;
    case 45: return k == 101;
    case 46: return k == 20 || k == 200;
    default: return false;
  }
}
constexpr int nterm(int l, int row) {
  int n = 0;
  for (int t = 0; t <= l; ++t)
    for (int u = 0; u <= l - t; ++u)
      for (int v = 0; v <= l - t - u; ++v) n += is_term(l, row, t, u, v);
  return n;
}
// term i of the list as t | u << 4 | v << 8
constexpr int term_at(int l, int row, int i) {
  for (int t = 0; t <= l; ++t)
    for (int u = 0; u <= l - t; ++u)
      for (int v = 0; v <= l - t - u; ++v)
        if (is_term(l, row, t, u, v) && i-- == 0) return t | (u << 4) | (v << 8);
  return 0;
}
// the h-th (t, u, v), t + u + v <= L, in that order, packed likewise
__host__ __device__ constexpr int lex_at(int L, int h) {
  for (int t = 0; t <= L; ++t)
    for (int u = 0; u <= L - t; ++u) {
      const int n = L - t - u + 1;
      if (h < n) return t | (u << 4) | (h << 8);
      h -= n;
    }
  return 0;
}

// X r1 + k r2 of the recursion; as intrinsics, so that no other contraction is chosen
template <int K>
__device__ __forceinline__ double r_step(double X, double r1, double r2) {
  if constexpr (K == 0)
    return __dmul_rn(X, r1);
  else if constexpr (K == 1)
    return __dadd_rn(r2, __dmul_rn(X, r1));
  else
    return __fma_rn(static_cast<double>(K), r2, __dmul_rn(X, r1));
}

template <int E>
__device__ __forceinline__ void r_entry(double* R, double X, double Y, double Z) {
  constexpr int t = dec_t(E), u = dec_u(E), v = dec_v(E);
  if constexpr (t > 0)
    R[E] = r_step<t - 1>(X, R[tix(t - 1, u, v)], R[tix(t > 1 ? t - 2 : 0, u, v)]);
  else if constexpr (u > 0)
    R[E] = r_step<u - 1>(Y, R[tix(t, u - 1, v)], R[tix(t, u > 1 ? u - 2 : 0, v)]);
  else
    R[E] = r_step<v - 1>(Z, R[tix(t, u, v - 1)], R[tix(t, u, v > 1 ? v - 2 : 0)]);
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

// sum over the terms I .. of the aux function: s + sum dp[i] R[h + term i], in order
template <int T, int U, int V, int LC, int ROW, int I = 0>
__device__ __forceinline__ double w_entry(const double* R, const double* dp, double s) {
  constexpr int k = term_at(LC, ROW, I);
  s = fma(dp[I], R[tix(T + (k & 15), U + ((k >> 4) & 15), V + (k >> 8))], s);
  if constexpr (I + 1 < nterm(LC, ROW)) return w_entry<T, U, V, LC, ROW, I + 1>(R, dp, s);
  return s;
}
template <int LAB, int LC, int ROW, int... H>
__device__ __forceinline__ void w_all(const double* R, const double* dp, double* W, std::integer_sequence<int, H...>) {
  ((W[H] = w_entry<lex_at(LAB, H) & 15, (lex_at(LAB, H) >> 4) & 15, (lex_at(LAB, H) >> 8), LC, ROW>(R, dp, 0.0)), ...);
}

// acc[ab] += sum_h E[ab][h] W[h] for the thread's Cartesian pairs, h in order; four pairs at a time, whose chains
// of FMAs hide each other's latency
template <int NH>
__device__ __forceinline__ void add_rows(const double* __restrict__ E, const double* W, int ab0, int dab, int nab, int stride,
                                         double* acc) {
  constexpr int NHP = (NH + 1) & ~1;
#pragma unroll 1
  for (int ab = ab0; ab < nab; ab += 4 * dab) {
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    const double* e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = E + (ab + i * dab < nab ? ab + i * dab : ab) * NHP;
#pragma unroll
    for (int h = 0; h < NH; h += 2) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double2 c = *reinterpret_cast<const double2*>(e[i] + h);
        v[i] = fma(c.x, W[h], v[i]);
        if (h + 1 < NH) v[i] = fma(c.y, W[h + 1 < NH ? h + 1 : h], v[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (ab + i * dab < nab) acc[(ab + i * dab) * stride] += v[i];
  }
}

// The aux functions ROW .. 2 LC of one thread.  terms, toff: the term table and its offsets for this l; pw: the
// prefactor times powers of 1 / 2 gamma
template <int LAB, int LC, int ROW>
__device__ __forceinline__ void rows(const double* R, const double* pw, const EriTerm* __restrict__ terms,
                                     const int* __restrict__ toff, const double* __restrict__ E, int ab0, int dab, int nab,
                                     int stride, double* acc) {
  constexpr int NH = tetc(LAB), NT_ = nterm(LC, ROW);
  double dp[NT_];
  const EriTerm* q = terms + __ldg(toff + ROW);
#pragma unroll
  for (int i = 0; i < NT_; ++i) {
    const int k = term_at(LC, ROW, i);
    dp[i] = __dmul_rn(q[i].d, pw[(LC + (k & 15) + ((k >> 4) & 15) + (k >> 8)) / 2]);
  }
  double W[NH];
  w_all<LAB, LC, ROW>(R, dp, W, std::make_integer_sequence<int, NH>());
  if constexpr (LAB == 0)
    acc[ROW] += __dmul_rn(E[0], W[0]);
  else
    add_rows<NH>(E, W, ab0, dab, nab, stride, acc + ROW);
  if constexpr (ROW < 2 * LC) rows<LAB, LC, ROW + 1>(R, pw, terms, toff, E, ab0, dab, nab, stride, acc);
}

template <int LAB, int LC>
__global__ void __launch_bounds__(NT) k_eri_thread(const EriLaunch P) {
  constexpr int L = LAB + LC, NR = tetc(L), NH = tetc(LAB), NHP = (NH + 1) & ~1, NF = 2 * LC + 1, ts = LAB + 2;
  extern __shared__ __align__(16) double sm[];
  double* E1 = sm;                // 3 x (la+1)(lb+1) ts: 1-D expansions
  double* E = sm + P.e1size;      // nab x NHP: their products
  double* acc = E + P.esize;      // nab x tile NF: Cartesian integrals
  const int tid = threadIdx.x;
  const int tile = P.tile, kt = tid & (tile - 1), part = tid / tile, parts = NT / tile;
  const int arow = tile * NF;
  const long ntile = (P.nket + tile - 1) / tile;
  const long ip = blockIdx.x / ntile;
  const long k0 = (blockIdx.x - ip * ntile) * tile;
  const int2 pair = P.pairs[ip];
  const EriShell A = P.bra[pair.x];
  const EriShell B = P.bra[pair.y];
  const bool live = k0 + kt < P.nket;
  const EriShell C = P.ket[P.kets[live ? k0 + kt : P.nket - 1]];
  const int la = A.l, lb = B.l, nca = ncart_d(la), ncb = ncart_d(lb), nab = nca * ncb;
  const double gam = P.kexp[C.prim0], ck = P.kcoef[C.prim0];
  const int* toff = P.term_off + (LMAX + 1 + LC) * (TERM_STRIDE + 1);
  const double sgn = (LC & 1) ? -1.0 : 1.0;
  const double two_pi_25 = 2.0 * 17.493418327624862;  // 2 pi^(5/2)

  double racc[NF] = {};  // LAB = 0: the sums stay in registers
  if (LAB > 0) {
    for (int o = tid; o < nab * arow; o += NT) acc[o] = 0.0;
    __syncthreads();
  }
  const double ABx = A.x - B.x, ABy = A.y - B.y, ABz = A.z - B.z;
  const double r2 = fma(ABz, ABz, fma(ABx, ABx, __dmul_rn(ABy, ABy)));
  for (int ij = 0; ij < A.nprim * B.nprim; ++ij) {
    const int i = ij / B.nprim, j = ij - i * B.nprim;
    const double a = P.bexp[A.prim0 + i], ca = P.bcoef[A.prim0 + i];
    const double b = P.bexp[B.prim0 + j], cb = P.bcoef[B.prim0 + j];
    const double p = a + b, mu = a * b / p;
    const double K = exp(-mu * r2);
    const double cc = ca * cb;
    if (fabs(cc * K) < 1e-22) continue;  // contributes below double precision (host rule); the same for all threads
    const double Px = fma(b, B.x, __dmul_rn(a, A.x)) / p, Py = fma(b, B.y, __dmul_rn(a, A.y)) / p;
    const double Pz = fma(b, B.z, __dmul_rn(a, A.z)) / p;
    if constexpr (LAB > 0) {
      const int n1 = (la + 1) * (lb + 1) * ts;
      __syncthreads();  // the previous primitive pair's readers of E are done
      if (tid < 3) {
        const double pd = tid == 0 ? Px : (tid == 1 ? Py : Pz);
        const double ad = tid == 0 ? A.x : (tid == 1 ? A.y : A.z);
        const double bd = tid == 0 ? B.x : (tid == 1 ? B.y : B.z);
        hermite_1d_dev(la, lb, p, pd - ad, pd - bd, tid == 0 ? K : 1.0, E1 + tid * n1, ts);
      }
      __syncthreads();
      // E[ab][tuv] = Ex Ey Ez, zero beyond the pair's orders
      for (int o = tid; o < nab * NH; o += NT) {
        const int ab = o / NH, h = o - ab * NH;
        const int c = __ldg(P.lex + LAB * LEX_STRIDE + h);
        const int t = c & 15, u = (c >> 4) & 15, v = c >> 8;
        const int ka = __ldg(P.cart + la * 16 + ab / ncb), kb = __ldg(P.cart + lb * 16 + ab % ncb);
        const int ax = ka & 15, ay = (ka >> 4) & 15, az = ka >> 8;
        const int bx = kb & 15, by = (kb >> 4) & 15, bz = kb >> 8;
        double e = 0.0;
        if (t <= ax + bx && u <= ay + by && v <= az + bz) {
          const double et = E1[(ax * (lb + 1) + bx) * ts + t];
          const double eu = __dmul_rn(et, E1[n1 + (ay * (lb + 1) + by) * ts + u]);
          e = __dmul_rn(eu, E1[2 * n1 + (az * (lb + 1) + bz) * ts + v]);
        }
        E[ab * NHP + h] = e;
      }
      __syncthreads();
    }
    const double al = p * gam / (p + gam);
    const double X = Px - C.x, Y = Py - C.y, Z = Pz - C.z;
    const double T = al * fma(Z, Z, fma(X, X, __dmul_rn(Y, Y)));
    double G[L + 1];
    boys_eval_l<L>(T, P.boys, G);
    const double pref = two_pi_25 / (p * gam * sqrt(p + gam)) * cc * ck * sgn;
    const double i2g = 1.0 / (2.0 * gam);
    double pw[LC + 1];
    pw[0] = pref;
#pragma unroll
    for (int q = 1; q <= LC; ++q) pw[q] = pw[q - 1] * i2g;
    const double m2a = -2.0 * al;
    double pwn = 1.0;
#pragma unroll
    for (int m = 1; m <= L; ++m) {
      pwn *= m2a;
      G[m] *= pwn;
    }
    double R[NR];
    r_layers<L>(R, G, X, Y, Z);
    if constexpr (LAB == 0)
      rows<0, LC, 0>(R, pw, P.terms, toff, &K, 0, 1, 1, 0, racc);
    else
      rows<LAB, LC, 0>(R, pw, P.terms, toff, E, part, parts, nab, arow, acc + kt * NF);
  }
  if (LAB > 0) __syncthreads();  // the other parts' integrals
  if (!live) return;
  // bra Cartesian -> spherical, then store
  const int nfb = B.nfunc, nfab = A.nfunc * nfb;
  const double* ta = P.sph + sph_off(la);
  const double* tb = P.sph + sph_off(lb);
  for (int f = part; f < nfab; f += parts) {
    const int fa = f / nfb, fb = f - fa * nfb;
    const int ia0 = A.pure ? 0 : fa, ia1 = A.pure ? nca : fa + 1;
    const int ib0 = B.pure ? 0 : fb, ib1 = B.pure ? ncb : fb + 1;
    double v[NF] = {};
    if constexpr (LAB == 0) {
#pragma unroll
      for (int m = 0; m < NF; ++m) v[m] = racc[m];  // the s function's coefficient is 1
    } else {
      for (int ia = ia0; ia < ia1; ++ia) {
        const double wa = A.pure ? __ldg(ta + fa * nca + ia) : 1.0;
        if (wa == 0.0) continue;
        double sb[NF] = {};
        for (int ib = ib0; ib < ib1; ++ib) {
          const double wb = B.pure ? __ldg(tb + fb * ncb + ib) : 1.0;
#pragma unroll
          for (int m = 0; m < NF; ++m) sb[m] = fma(wb, acc[(ia * ncb + ib) * arow + kt * NF + m], sb[m]);
        }
#pragma unroll
        for (int m = 0; m < NF; ++m) v[m] = fma(wa, sb[m], v[m]);
      }
    }
    const long mu = A.off + fa, nu = B.off + fb;
    double *o0 = nullptr, *o1 = nullptr;
    if (P.mode == 0) {
      if (pair.x == pair.y && nu > mu) continue;
      const long hi = mu > nu ? mu : nu, lo = mu > nu ? nu : mu;
      if (hi < P.mu0 || hi >= P.mu1) continue;
      o0 = P.out + (hi * (hi + 1) / 2 + lo - P.rowbase) * P.ld + C.off;
    } else {
      if (mu >= P.mu0 && mu < P.mu1) o0 = P.out + ((mu - P.rowbase) * P.n + nu) * P.ld + C.off;
      if (pair.x != pair.y && nu >= P.mu0 && nu < P.mu1) o1 = P.out + ((nu - P.rowbase) * P.n + mu) * P.ld + C.off;
    }
#pragma unroll
    for (int m = 0; m < NF; ++m) {
      if (o0) o0[m] = v[m];
      if (o1) o1[m] = v[m];
    }
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
