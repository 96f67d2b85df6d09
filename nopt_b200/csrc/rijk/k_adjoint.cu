// k_adjoint.cu — the adjoint of the Fock build (rijk_grad).  No reference counterpart: the
// reference has no analytic gradient and differentiates by finite differences
// (src/QM_calc.cpp:142).
//
// With D = C^T C over the n_c occupied rows of MO (src/SCF.cpp:63-73), the fitted tensor
// B^Q = sum_P M_QP (P|.), w_Q = <B^Q, D> and Y^Q = C B^Q C^T (n_c x n_c), the energy of the
// reference's RHF (src/SCF.cpp:134) is
//     E = 2 tr(H D) + 2 sum_Q w_Q^2 - sum_Q |Y^Q|^2 + e_nuc ,
// and its derivatives are
//     dE/dC        = 4 C F,  F = H + 2J - K                          (orbital gradient)
//     Gamma^Q      = dE/dB^Q = 4 w_Q D - 2 C^T Y^Q C                 (full-square derivative)
//     dE/d(P|mu nu) = sum_Q M_QP Gamma^Q_{mu nu}                    (times 2 for mu != nu when the
//                                                                      pair is stored once)
//     dE/d(P|Q)    = -(M^T G M)_PQ,  G_QR = (1/2) sum_{mu nu} Gamma^Q_{mu nu} B^R_{mu nu}
// (E depends on the metric only through V^-1 = M^T M, for either metric form).
//
// Gamma^Q depends on Q only through w_Q and the n_c x n_c matrix Y^Q.  With the metric factor applied to those,
// u_P = sum_Q M_QP w_Q and Z^P = sum_Q M_QP Y^Q,
//     dE/d(P|mu nu) = 4 u_P D_{mu nu} - 2 (C^T Z^P C)_{mu nu} :
// the contraction with the metric runs over n_c (n_c + 1) / 2 values per aux function instead of the n (n + 1) / 2
// of Gamma.  dE/d(P|Q) could be had from Z^P as well, sum_ij Z^P_ij Z^Q_ij - 2 u_P u_Q, and is formed from Gamma
// all the same: M^T G M multiplies the rounding of G by |M|^2, 3e-10 of the whole and up to 7e-8 of single
// elements for C10H22, so G keeps its sums, to the order of their terms (as close to 64 bits by either way), and
// the build before it the DMMA half-transform.
//
// Device work, FP64 throughout, every contraction on hand-written DMMA kernels: one FP64 Fock build
// (which leaves w and the half-transformed XT in the context), Y^Q = X^Q C^T over chunks of aux functions,
// Z and u by one GEMM with M (the pairs i >= j packed, u as one more row), the first index of C^T Z C by one
// GEMM, and the second by one GEMM per orbital row mu, whose epilogue writes the packed pair rows.  Those rows
// leave in blocks: the copy of one block to the host runs while the next is formed, so the device never holds
// the whole derivative.  Behind the copies, which take longest (or with each chunk of Y, where Y of all aux functions
// does not fit or nothing is copied), dE/d(P|Q) over chunks of aux functions: T^Q = Y^Q C (k_gemm_f64), the packed Gamma tiles
// (k_gamma_f64), their rows of G by one GEMM with B, and at the end M^T G M; the blocks' GEMMs take the
// high-priority stream beside it.
// (H2O)8 cc-pVDZ, 151 MB out: 15.5 to 18.7 ms a call with Gamma for both derivatives and the copies at the end, 7.6 to 8.5
// now (medians of 20 to 30 calls in many runs, output arrays reused; with new arrays, whose pages the copies
// touch first, 38.5 to 39.1 and 29.2 to 30.2); (H2O)16, 126 and 59 to 71.
#include <algorithm>
#include <cmath>
#include <vector>

#include "gemm_f64.cuh"
#include "rijk_internal.h"

#define RIJK_API extern "C" __attribute__((visibility("default")))

namespace rijk {
namespace {

constexpr int G_THREADS = 128;

// Gamma[Q][t][r][c] = 4 w_Q D[mu][nu] - 2 sum_i T^Q[mu][i] Ct[nu][i], tile t = (I, J), I >= J; half of that in the
// diagonal tiles, so that a product with B over the stored elements is half the one over the full squares.
// Tt: [(Q, i)][npad] = T^Q transposed (row (Q, i), mu contiguous); Ct: [npad][noccp]; D: n x n.
constexpr int G_ASTAGE = (64 * LDK > KC * LDM) ? 64 * LDK : KC * LDM;
__global__ void __launch_bounds__(G_THREADS)
    k_gamma_f64(const double* __restrict__ Tt, const double* __restrict__ Ct, const double* __restrict__ D,
                const double* __restrict__ w, long n, long npad, long noccp, long tile_elems,
                double* __restrict__ Gamma) {
  extern __shared__ __align__(16) double smem_g[];
  double* sA[2] = {smem_g, smem_g + G_ASTAGE};
  double* sB[2] = {smem_g + 2 * G_ASTAGE, smem_g + 2 * G_ASTAGE + 64 * LDK};
  const long t = blockIdx.x, Q = blockIdx.y;
  long I, J;
  tri_decode(t, I, J);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  const double* Ar = Tt + Q * noccp * npad + I * TILE;  // A(mu, i) = Ar[i * npad + mu]: staged [i][mu]
  const double* Br = Ct + J * TILE * noccp;
  auto load = [&](int stage, long k0) {
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      int idx = tid + it * G_THREADS;
      int ka = idx >> 5, pa = idx & 31;  // A: k row (i) 0..31, mu pair 0..31
      bool oka = k0 + ka < noccp;
      cp_async16(&sA[stage][ka * LDM + pa * 2], oka ? Ar + (k0 + ka) * npad + pa * 2 : Tt, oka);
      int row = idx >> 4, seg = idx & 15;  // B: row nu 0..63, i pair 0..15
      long k = k0 + seg * 2;
      bool ok = k < noccp;
      cp_async16(&sB[stage][row * LDK + seg * 2], ok ? Br + row * noccp + k : Ct, ok);
    }
  };
  double acc[4][4][2];
  zero_acc(acc);
  const long nk = (noccp + KC - 1) / KC;
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
    warp_mma_chunk<4, 4, false>(acc, sA[kc & 1], sB[kc & 1], wm * 32, wn * 32, lane);
    __syncthreads();
  }
  const int g = lane >> 2, tq = lane & 3;
  const double wq4 = 4.0 * w[Q];
  const double f = I == J ? 0.5 : 1.0;
  double* out = Gamma + Q * tile_elems + t * TILE2;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = wm * 32 + i * 8 + g;
    const long mu = I * TILE + r;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = wn * 32 + j * 8 + 2 * tq;
      const long nu = J * TILE + c;
      double d0 = (mu < n && nu < n) ? D[mu * n + nu] : 0.0;
      double d1 = (mu < n && nu + 1 < n) ? D[mu * n + nu + 1] : 0.0;
      *reinterpret_cast<double2*>(out + r * TILE + c) =
          make_double2(f * (wq4 * d0 - 2.0 * acc[i][j][0]), f * (wq4 * d1 - 2.0 * acc[i][j][1]));
    }
  }
}

// Ct[nu][i] = C_{i nu} from the padded MOp[i][nu]
__global__ void k_transpose_mo(const double* __restrict__ MOp, long noccp, long npad, double* __restrict__ Ct) {
  long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; idx < noccp * npad; idx += static_cast<long>(gridDim.x) * blockDim.x) {
    long nu = idx / noccp, i = idx % noccp;
    Ct[idx] = MOp[i * npad + nu];
  }
}

// Yp[Q][p] = Y[(Q, i)][j] for the pairs p = (i, j), i >= j, of aux functions q0 .. q0 + nq; Yp[Q][np] = w_Q.
__global__ void k_pack_pairs(const double* __restrict__ Y, const double* __restrict__ w, long q0, long nq, long nocc,
                             long noccp, long np, long ldp, double* __restrict__ Yp) {
  for (long p = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; p < ldp;
       p += static_cast<long>(gridDim.x) * blockDim.x) {
    long i, j;
    tri_decode(p, i, j);
    for (long q = blockIdx.y; q < nq; q += gridDim.y)
      Yp[(q0 + q) * ldp + p] = p < np ? Y[(q * noccp + i) * nocc + j] : p == np ? w[q0 + q] : 0.0;
  }
}

// From Z[p][P] (rows p = (i, j), i >= j) the full square Zf[j][i][P] with zeros from naux to the even pitch ldP.
__global__ void k_expand_pairs(const double* __restrict__ Z, long nocc, long np, long naux, long ldP,
                               double* __restrict__ Zf) {
  for (long p = blockIdx.y; p < np; p += gridDim.y) {
    long i, j;
    tri_decode(p, i, j);
    for (long P = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; P < ldP;
         P += static_cast<long>(gridDim.x) * blockDim.x) {
      const double z = P < naux ? Z[p * ldP + P] : 0.0;
      Zf[(j * nocc + i) * ldP + P] = z;
      if (i != j) Zf[(i * nocc + j) * ldP + P] = z;
    }
  }
}

__global__ void k_fock_sym(const double* __restrict__ H, const double* __restrict__ J, const double* __restrict__ K,
                           long nn, double* __restrict__ F) {
  long idx = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; idx < nn; idx += static_cast<long>(gridDim.x) * blockDim.x) F[idx] = H[idx] + 2.0 * J[idx] - K[idx];
}

// partial[b], partial[512 + b]: compensated sum of D (F + H) over a grid-stride slice
__global__ void k_energy_partial(const double* __restrict__ D, const double* __restrict__ F,
                                 const double* __restrict__ H, long nn, double* __restrict__ partial) {
  double s = 0.0, c = 0.0;
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < nn; i += static_cast<long>(gridDim.x) * blockDim.x)
    neumaier_add(s, c, D[i] * (F[i] + H[i]));
  warp_sum_comp(s, c);
  __shared__ double sh[2][8];
  if ((threadIdx.x & 31) == 0) {
    sh[0][threadIdx.x >> 5] = s;
    sh[1][threadIdx.x >> 5] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0, u = 0.0;
    for (int i = 0; i < 8; ++i) {
      neumaier_add(t, u, sh[0][i]);
      u += sh[1][i];
    }
    partial[blockIdx.x] = t;
    partial[512 + blockIdx.x] = u;
  }
}

// Device time per stage of rijk_grad when profiling is on: mark(k) records an event on the stream,
// and the interval since the previous mark counts for stage k (k < 0: not counted).
struct GradTimer {
  bool on = false;
  cudaStream_t s = nullptr;
  std::vector<std::pair<int, cudaEvent_t>> ev;
  void mark(int stage) {
    if (!on) return;
    cudaEvent_t e;
    cudaEventCreate(&e);
    cudaEventRecord(e, s);
    ev.emplace_back(stage, e);
  }
  // after the stream has drained
  void collect(rijk_stats_t& st) {
    for (double& v : st.ms_grad_stage) v = 0.0;
    st.ms_grad_total = 0.0;
    for (size_t i = 1; i < ev.size(); ++i) {
      if (ev[i].first < 0) continue;
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, ev[i - 1].second, ev[i].second);
      st.ms_grad_stage[ev[i].first] += ms;
      st.ms_grad_total += ms;
    }
  }
  ~GradTimer() {
    for (auto& e : ev) cudaEventDestroy(e.second);
  }
};

unsigned grid_of(long total) {
  long b = (total + 255) / 256;
  if (b > 148L * 16) b = 148L * 16;
  return static_cast<unsigned>(b < 1 ? 1 : b);
}

}  // namespace
}  // namespace rijk

using namespace rijk;

RIJK_API int rijk_set_grad_chunk(rijk_ctx* ctx, long q_per_chunk) {
  if (!ctx) return RIJK_ERR_ARG;
  if (q_per_chunk < 0) return set_err(ctx, RIJK_ERR_ARG, "rijk_set_grad_chunk: negative chunk");
  ctx->grad_qchunk = q_per_chunk;
  return RIJK_OK;
}

RIJK_API int rijk_grad(rijk_ctx* ctx, const double* MO, long nocc, const double* H, double e_nuc, double* E,
                       double* dEdC, double* dEdI3, double* dEdPQ) {
  if (!ctx) return RIJK_ERR_ARG;
  if (!MO || !H || !E || !dEdC) return set_err(ctx, RIJK_ERR_ARG, "rijk_grad: null pointer");
  int rc = check_fock_args(ctx, nocc, RIJK_PREC_FP64);
  if (rc) return rc;
  if (nocc < 1) return set_err(ctx, RIJK_ERR_ARG, "rijk_grad: n_c must be at least 1");
  NvtxRange range("rijk_grad");
  if (ctx->nq != ctx->naux)
    return set_err(ctx, RIJK_ERR_STATE, "rijk_grad needs all aux functions in one context (no aux range)");
  cudaSetDevice(ctx->device);
  cudaStream_t s = ctx->stream;
  const long n = ctx->n, naux = ctx->naux, npad = ctx->npad, ntile = ctx->ntile;
  const long nn = n * n, te = ntile * TILE2, noccp = round_up(nocc, 16), nauxp = round_up(naux, KC);
  const size_t b_nn = nn * sizeof(double);
  DeviceBuf dMO, dH, dD, dJ, dK, dF, dG, red, Y, Yp, Z, Zf, Ct, Gam, Gm, T1, out[2];
  auto cleanup = [&]() {
    DeviceBuf* all[] = {&dMO, &dH, &dD, &dJ, &dK, &dF, &dG, &red, &Y, &Yp, &Z, &Zf, &Ct, &Gam, &Gm, &T1, &out[0], &out[1]};
    for (DeviceBuf* b : all) release(*b);
  };
  auto chk = [&](int r) {
    if (r) cleanup();
    return r;
  };
  if ((rc = chk(ensure_tmp(ctx, dMO, nocc * n * sizeof(double), "grad MO"))) || (rc = chk(ensure_tmp(ctx, dH, b_nn, "grad H"))) ||
      (rc = chk(ensure_tmp(ctx, dD, b_nn, "grad D"))) || (rc = chk(ensure_tmp(ctx, dJ, b_nn, "grad J"))) ||
      (rc = chk(ensure_tmp(ctx, dK, b_nn, "grad K"))) || (rc = chk(ensure_tmp(ctx, dF, b_nn, "grad F"))) ||
      (rc = chk(ensure_tmp(ctx, dG, nocc * n * sizeof(double), "grad dEdC"))) ||
      (rc = chk(ensure_tmp(ctx, red, 1024 * sizeof(double), "grad reduce"))))
    return rc;
  double* pMO = static_cast<double*>(dMO.p);
  double* pD = static_cast<double*>(dD.p);
  double* pF = static_cast<double*>(dF.p);
  cudaMemcpyAsync(pMO, MO, nocc * n * sizeof(double), cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(dH.p, H, b_nn, cudaMemcpyHostToDevice, s);
  GradTimer tm;
  tm.on = ctx->profiling;
  tm.s = s;
  tm.mark(-1);
  {  // D[mu][nu] = sum_i C[i][mu] C[i][nu]
    GemmF64Args g;
    g.M = n, g.N = n, g.K = nocc;
    g.A = pMO, g.lda = n, g.a_kmajor = false;
    g.B = pMO, g.ldb = n, g.b_kmajor = false;
    g.C = pD, g.ldc = n;
    gemm_f64(g, 1, s);
  }
  if ((rc = chk(fock_device_impl(ctx, pD, pMO, nocc, static_cast<double*>(dJ.p), static_cast<double*>(dK.p),
                                 RIJK_PREC_FP64, nullptr, nullptr, dEdPQ != nullptr))))
    return rc;
  k_fock_sym<<<grid_of(nn), 256, 0, s>>>(static_cast<const double*>(dH.p), static_cast<const double*>(dJ.p),
                                         static_cast<const double*>(dK.p), nn, pF);
  k_energy_partial<<<512, 256, 0, s>>>(pD, pF, static_cast<const double*>(dH.p), nn, static_cast<double*>(red.p));
  {  // dE/dC[i][mu] = 4 sum_nu C[i][nu] F[nu][mu]
    GemmF64Args g;
    g.M = nocc, g.N = n, g.K = n;
    g.A = pMO, g.lda = n, g.a_kmajor = true;
    g.B = pF, g.ldb = n, g.b_kmajor = false;
    g.C = static_cast<double*>(dG.p), g.ldc = n;
    g.alpha = 4.0;
    gemm_f64(g, 1, s);
  }
  tm.mark(0);
  std::vector<double> part(1024);
  cudaMemcpyAsync(part.data(), red.p, 1024 * sizeof(double), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(dEdC, dG.p, nocc * n * sizeof(double), cudaMemcpyDeviceToHost, s);
  tm.mark(-1);
  if ((rc = chk(cuda_check(ctx, cudaStreamSynchronize(s), "rijk_grad energy"))) || (rc = chk(check_device_error(ctx))))
    return rc;
  double es = 0.0, ec = 0.0;  // compensated: the 512 block sums, their compensations, then e_nuc
  for (int b = 0; b < 512; ++b) {
    neumaier_add(es, ec, part[b]);
    ec += part[512 + b];
  }
  neumaier_add(es, ec, e_nuc);
  *E = es + ec;
  if (!dEdI3 && !dEdPQ) {
    tm.collect(ctx->stats);
    cleanup();
    return RIJK_OK;
  }
  // Y^Q over chunks of aux functions (rijk_set_grad_chunk; all at once by default), from the X the FP64 build
  // left in XT.
  const long kdim = naux * noccp;
  const long np = nocc * (nocc + 1) / 2, ldp = round_up(np + 1, 2), ldP = round_up(naux, 2);
  const double* MOp = static_cast<const double*>(ctx->MOp.p);
  const double* pM = static_cast<const double*>(ctx->M.p);  // row-major [Q][P], ld nauxp
  long qc = ctx->grad_qchunk > 0 ? std::min(ctx->grad_qchunk, naux) : naux;
  const size_t b_pairs = static_cast<size_t>(np + 1) * ldP * sizeof(double);
  // blocks of orbital rows of dE/d(P|mu nu), about 64 MB each and at least one row
  const long blk = std::max<long>(n * naux, (64L << 20) / 8);
  // With both derivatives wanted Y stays for all aux functions while that fits, beside Z, which does whatever the chunk:
  // G then follows the first copies out instead of Y's chunks (C40H82 in chunks of 1200: 1.4 against 2.7 s).
  long qy = dEdPQ && dEdI3 ? naux : qc;
  while ((rc = ensure_tmp(ctx, Y, static_cast<size_t>(qy) * noccp * nocc * sizeof(double), "grad Y"))) {
    if (qy == 1 || ctx->fail_alloc_after == 0) return chk(rc);
    qy = qy > qc ? qc : (qy + 1) / 2;
  }
  qc = std::min(qc, qy);
  const bool behind = dEdPQ && dEdI3 && qy == naux;
  // aux functions per chunk of T and Gamma, in whole tiles of G's rows and no more than the chunk: 1 GiB, less if that cannot
  // be had (asking for the free memory first took 7 ms a call)
  const long per_q = te + npad * noccp;
  long gq = std::max<long>(1, std::min<long>(naux, (1L << 30) / (8 * per_q)));
  if (gq < naux && gq >= 64) gq -= gq % 64;
  gq = std::min(gq, qc);
  if (dEdPQ && ((rc = chk(ensure_tmp(ctx, Ct, static_cast<size_t>(npad) * noccp * sizeof(double), "grad Ct"))) ||
                (rc = chk(ensure_tmp(ctx, Gm, static_cast<size_t>(naux) * naux * sizeof(double), "grad G"))) ||
                (rc = chk(ensure_tmp(ctx, T1, static_cast<size_t>(naux) * naux * sizeof(double), "grad T1")))))
    return rc;
  while (dEdPQ && (rc = ensure_tmp(ctx, Gam, static_cast<size_t>(gq) * per_q * sizeof(double), "grad Gamma"))) {
    if (gq == 1 || ctx->fail_alloc_after == 0) return chk(rc);
    gq = (gq + 1) / 2;
  }
  if (dEdI3 && ((rc = chk(ensure_tmp(ctx, Yp, static_cast<size_t>(naux) * ldp * sizeof(double), "grad Y pairs"))) ||
                (rc = chk(ensure_tmp(ctx, Z, b_pairs, "grad Z"))) ||
                (rc = chk(ensure_tmp(ctx, Zf, static_cast<size_t>(nocc) * nocc * ldP * sizeof(double), "grad Z square"))) ||
                (rc = chk(ensure_tmp(ctx, out[0], blk * sizeof(double), "grad dI3 block"))) ||
                (rc = chk(ensure_tmp(ctx, out[1], blk * sizeof(double), "grad dI3 block")))))
    return rc;
  double* pY = static_cast<double*>(Y.p);
  const size_t gsmem = (2 * G_ASTAGE + 2 * 64 * LDK) * sizeof(double);
  if (dEdPQ) {
    ensure_smem_limit(reinterpret_cast<const void*>(k_gamma_f64), gsmem);
    k_transpose_mo<<<grid_of(noccp * npad), 256, 0, s>>>(MOp, noccp, npad, static_cast<double*>(Ct.p));
  }
  // rows q0 .. q0 + nq of G, from Y^q0 .. at y
  auto g_rows = [&](long q0, long nq, const double* y) {
    double* pGam = static_cast<double*>(Gam.p);
    double* pT = pGam + gq * te;
    for (long g0 = 0; g0 < nq; g0 += gq) {
      const long ng = std::min(gq, nq - g0);
      {  // T^Q transposed, Tt[(Q, i)][mu] = sum_j Y^Q[i][j] C_{j mu}, one GEMM for the chunk
        GemmF64Args g;
        g.M = ng * noccp, g.N = npad, g.K = nocc;
        g.A = y + g0 * noccp * nocc, g.lda = nocc, g.a_kmajor = true;
        g.B = MOp, g.ldb = npad, g.b_kmajor = false;
        g.C = pT, g.ldc = npad;
        gemm_f64(g, 1, s);
      }
      k_gamma_f64<<<dim3(static_cast<unsigned>(ntile), static_cast<unsigned>(ng)), G_THREADS, gsmem, s>>>(
          pT, static_cast<const double*>(Ct.p), pD, static_cast<const double*>(ctx->w.p) + q0 + g0, n, npad, noccp, te,
          pGam);
      {  // G_QR = 1/2 sum_{mu nu} Gamma^Q B^R over the full squares
        GemmF64Args g;
        g.M = ng, g.N = naux, g.K = te;
        g.A = pGam, g.lda = te, g.a_kmajor = true;
        g.B = static_cast<const double*>(ctx->B.p), g.ldb = te, g.b_kmajor = true;
        g.C = static_cast<double*>(Gm.p) + (q0 + g0) * naux, g.ldc = naux;
        gemm_f64(g, 1, s);
      }
      tm.mark(5);
    }
  };
  // dE/d(P|Q) = -M^T G M
  auto queue_dpq = [&]() {
    double* pG = static_cast<double*>(Gm.p);
    // T1[Q][P'] = sum_R G[Q][R] M[R][P'];  out[P][P'] = -sum_Q M[Q][P] T1[Q][P']
    GemmF64Args g;
    g.M = naux, g.N = naux, g.K = naux;
    g.A = pG, g.lda = naux, g.a_kmajor = true;
    g.B = pM, g.ldb = nauxp, g.b_kmajor = false;
    g.C = static_cast<double*>(T1.p), g.ldc = naux;
    gemm_f64(g, 1, s);
    GemmF64Args h;
    h.M = naux, h.N = naux, h.K = naux;
    h.A = pM, h.lda = nauxp, h.a_kmajor = false;
    h.B = static_cast<const double*>(T1.p), h.ldb = naux, h.b_kmajor = false;
    h.C = pG, h.ldc = naux;
    h.alpha = -1.0;
    gemm_f64(h, 1, s);
    tm.mark(6);
  };
  for (long q0 = 0; q0 < naux; q0 += qy) {
    const long nq = std::min(qy, naux - q0);
    // Y^Q[i][j] = sum_nu X^Q_{i nu} C_{j nu} (= C B^Q C^T), every Q of the chunk in one product: rows (Q, i)
    // of X^T's columns are contiguous
    GemmF64Args g;
    g.M = nq * noccp, g.N = nocc, g.K = npad;
    g.A = static_cast<const double*>(ctx->XT.p) + q0 * noccp, g.lda = kdim, g.a_kmajor = false;
    g.B = MOp, g.ldb = npad, g.b_kmajor = true;
    g.C = pY, g.ldc = nocc;
    gemm_f64(g, 1, s);
    if (dEdI3) {
      dim3 grid(static_cast<unsigned>((ldp + 255) / 256), static_cast<unsigned>(std::min<long>(nq, 1024)));
      k_pack_pairs<<<grid, 256, 0, s>>>(pY, static_cast<const double*>(ctx->w.p), q0, nq, nocc, noccp, np, ldp,
                                        static_cast<double*>(Yp.p));
    }
    tm.mark(2);
    if (dEdPQ && !behind) g_rows(q0, nq, pY);
  }
  if (dEdPQ && !behind) queue_dpq();
  if (dEdI3) {
    // Z[p][P] = sum_Q Y[Q][p] M_QP, the last row u_P = sum_Q w_Q M_QP
    double* pZ = static_cast<double*>(Z.p);
    GemmF64Args z;
    z.M = np + 1, z.N = naux, z.K = naux;
    z.A = static_cast<const double*>(Yp.p), z.lda = ldp, z.a_kmajor = false;
    z.B = pM, z.ldb = nauxp, z.b_kmajor = false;
    z.C = pZ, z.ldc = ldP;
    gemm_f64(z, 1, s);
    k_expand_pairs<<<dim3(static_cast<unsigned>(std::min<long>((ldP + 255) / 256, 64)), static_cast<unsigned>(std::min<long>(np, 32768))),
                     256, 0, s>>>(pZ, nocc, np, naux, ldP, static_cast<double*>(Zf.p));
    // T[mu][i][P] = sum_j C_{j mu} Z[j][i][P], in XT's memory (X is not needed any more)
    const long row = nocc * ldP;
    if ((rc = chk(ensure(ctx, ctx->XT, static_cast<size_t>(n) * row * sizeof(double), "grad T")))) return rc;
    double* pT = static_cast<double*>(ctx->XT.p);
    GemmF64Args g;
    g.M = n, g.N = row, g.K = nocc;
    g.A = MOp, g.lda = npad, g.a_kmajor = false;
    g.B = static_cast<const double*>(Zf.p), g.ldb = row, g.b_kmajor = false;
    g.C = pT, g.ldc = row;
    gemm_f64(g, 1, s);
    tm.mark(3);
    // rows mu of dE/d(P|mu nu) in blocks, each on its way to the host while the next one is formed; on the
    // high-priority stream, so that dE/d(P|Q) fills what they and the copies leave (not under per-stage timing)
    cudaStream_t sb = ctx->profiling ? s : ctx->j_stream;
    cudaEventRecord(ctx->ev_pk, s);
    cudaStreamWaitEvent(sb, ctx->ev_pk, 0);
    const double* pu = pZ + np * ldP;
    auto tri = [](long m) { return m * (m + 1) / 2; };
    long prev0 = -1, prev1 = -1;
    int slot = 0;
    auto copy_out = [&](long m0, long m1, int b) -> int {
      cudaStreamWaitEvent(ctx->copy_stream, ctx->ev_blk[b], 0);
      const int r = cuda_check(ctx, cudaMemcpyAsync(dEdI3 + tri(m0) * naux, out[b].p,
                                                    static_cast<size_t>(tri(m1) - tri(m0)) * naux * sizeof(double),
                                                    cudaMemcpyDeviceToHost, ctx->copy_stream), "D2H dI3 block");
      cudaEventRecord(ctx->ev_out[b], ctx->copy_stream);
      return r;
    };
    for (long m0 = 0; m0 < n && !rc; slot ^= 1) {
      long m1 = m0 + 1;
      while (m1 < n && (tri(m1 + 1) - tri(m0)) * naux <= blk) ++m1;
      if (prev0 >= 0) cudaStreamWaitEvent(sb, ctx->ev_out[slot], 0);  // the copy of the block before the last
      GemmF64Args h;
      h.M = m1, h.N = naux, h.K = nocc;
      h.A = MOp, h.lda = npad, h.a_kmajor = false;
      h.B = pT + m0 * row, h.ldb = ldP, h.sB = row, h.b_kmajor = false;
      h.C = static_cast<double*>(out[slot].p), h.ldc = naux;
      h.mode = GEMM_DPAIRS;
      h.mu0 = m0, h.n_ao = n, h.D = pD, h.u = pu;
      gemm_f64(h, m1 - m0, sb);
      cudaEventRecord(ctx->ev_blk[slot], sb);
      if (m0 == 0 && behind) {  // before the first copy, which pageable memory makes the host wait for
        tm.mark(4);
        g_rows(0, naux, pY);
        queue_dpq();
      }
      if (prev0 >= 0) rc = copy_out(prev0, prev1, slot ^ 1);
      prev0 = m0;
      prev1 = m1;
      m0 = m1;
    }
    tm.mark(4);
    if (!rc) rc = copy_out(prev0, prev1, slot ^ 1);
  }
  if (dEdPQ && !rc)
    rc = cuda_check(ctx, cudaMemcpyAsync(dEdPQ, Gm.p, static_cast<size_t>(naux) * naux * sizeof(double),
                                         cudaMemcpyDeviceToHost, s), "D2H dPQ");
  ctx->stats.grad_qchunk = qc;
  const int rc_s = cuda_check(ctx, cudaStreamSynchronize(s), "rijk_grad");
  const int rc_j = cuda_check(ctx, cudaStreamSynchronize(ctx->j_stream), "rijk_grad blocks");
  const int rc_c = cuda_check(ctx, cudaStreamSynchronize(ctx->copy_stream), "rijk_grad copies");
  if (!rc) rc = rc_s ? rc_s : rc_j ? rc_j : rc_c;
  if (!rc) tm.collect(ctx->stats);
  cleanup();
  return rc;
}
