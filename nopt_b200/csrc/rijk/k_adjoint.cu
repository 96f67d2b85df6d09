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
// Gamma^Q depends on Q only through w_Q and the n_c x n_c matrix Y^Q, so neither derivative needs Gamma
// itself.  With the metric factor applied to those, u_P = sum_Q M_QP w_Q and Z^P = sum_Q M_QP Y^Q,
//     dE/d(P|mu nu) = 4 u_P D_{mu nu} - 2 (C^T Z^P C)_{mu nu}
//     dE/d(P|Q)     = sum_ij Z^P_ij Z^Q_ij - 2 u_P u_Q
// (from G_QR = 2 w_Q w_R - sum_ij Y^Q_ij Y^R_ij, as <D, B^R> = w_R and C B^R C^T = Y^R).  The contractions with
// the metric then run over n_c (n_c + 1) / 2 values per aux function instead of the n (n + 1) / 2 of Gamma.
//
// Device work, FP64 throughout, every contraction on the hand-written DMMA GEMM: one FP64 Fock build
// (which leaves w and the half-transformed XT in the context), Y^Q = X^Q C^T over chunks of aux functions,
// Z and u by one GEMM with M (the pairs i >= j packed, u as one more row), dE/d(P|Q) by one GEMM over the
// packed pairs, the first index of C^T Z C by one GEMM, and the second by one GEMM per orbital row mu, whose
// epilogue writes the packed pair rows.  Those rows leave in blocks: the copy of one block to the host runs
// while the next is formed, so the device never holds the whole derivative.
#include <algorithm>
#include <cmath>
#include <vector>

#include "gemm_f64.cuh"
#include "rijk_internal.h"

#define RIJK_API extern "C" __attribute__((visibility("default")))

namespace rijk {
namespace {

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

// From Z[p][P] (rows p = (i, j), i >= j, then u): the weighted rows Zw (1 on the diagonal i = j, 2 off it, -2 for
// u), and the full square Zf[j][i][P] with zeros from naux to the even pitch ldP.
__global__ void k_expand_pairs(const double* __restrict__ Z, long nocc, long np, long naux, long ldP,
                               double* __restrict__ Zw, double* __restrict__ Zf) {
  for (long p = blockIdx.y; p <= np; p += gridDim.y) {
    long i, j;
    tri_decode(p, i, j);
    const double f = p == np ? -2.0 : i == j ? 1.0 : 2.0;
    for (long P = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; P < ldP;
         P += static_cast<long>(gridDim.x) * blockDim.x) {
      const double z = P < naux ? Z[p * ldP + P] : 0.0;
      if (Zw) Zw[p * ldP + P] = f * z;
      if (Zf && p < np) {
        Zf[(j * nocc + i) * ldP + P] = z;
        if (i != j) Zf[(i * nocc + j) * ldP + P] = z;
      }
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
  const long n = ctx->n, naux = ctx->naux, npad = ctx->npad;
  const long nn = n * n, noccp = round_up(nocc, 16), nauxp = round_up(naux, KC);
  const size_t b_nn = nn * sizeof(double);
  DeviceBuf dMO, dH, dD, dJ, dK, dF, dG, red, Y, Yp, Z, Zw, Zf, dV, out[2];
  auto cleanup = [&]() {
    DeviceBuf* all[] = {&dMO, &dH, &dD, &dJ, &dK, &dF, &dG, &red, &Y, &Yp, &Z, &Zw, &Zf, &dV, &out[0], &out[1]};
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
                                 RIJK_PREC_FP64))))
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
  const long qc = ctx->grad_qchunk > 0 ? std::min(ctx->grad_qchunk, naux) : naux;
  const size_t b_pairs = static_cast<size_t>(np + 1) * ldP * sizeof(double);
  // blocks of orbital rows of dE/d(P|mu nu), about 64 MB each and at least one row
  const long blk = std::max<long>(n * naux, (64L << 20) / 8);
  if ((rc = chk(ensure_tmp(ctx, Y, static_cast<size_t>(qc) * noccp * nocc * sizeof(double), "grad Y"))) ||
      (rc = chk(ensure_tmp(ctx, Yp, static_cast<size_t>(naux) * ldp * sizeof(double), "grad Y pairs"))) ||
      (rc = chk(ensure_tmp(ctx, Z, b_pairs, "grad Z"))))
    return rc;
  if (dEdPQ && ((rc = chk(ensure_tmp(ctx, Zw, b_pairs, "grad weighted Z"))) ||
                (rc = chk(ensure_tmp(ctx, dV, static_cast<size_t>(naux) * naux * sizeof(double), "grad dPQ")))))
    return rc;
  if (dEdI3 && ((rc = chk(ensure_tmp(ctx, Zf, static_cast<size_t>(nocc) * nocc * ldP * sizeof(double), "grad Z square"))) ||
                (rc = chk(ensure_tmp(ctx, out[0], blk * sizeof(double), "grad dI3 block"))) ||
                (rc = chk(ensure_tmp(ctx, out[1], blk * sizeof(double), "grad dI3 block")))))
    return rc;
  double* pY = static_cast<double*>(Y.p);
  double* pZ = static_cast<double*>(Z.p);
  for (long q0 = 0; q0 < naux; q0 += qc) {
    const long nq = std::min(qc, naux - q0);
    // Y^Q[i][j] = sum_nu X^Q_{i nu} C_{j nu} (= C B^Q C^T), every Q of the chunk in one product: rows (Q, i)
    // of X^T's columns are contiguous
    GemmF64Args g;
    g.M = nq * noccp, g.N = nocc, g.K = npad;
    g.A = static_cast<const double*>(ctx->XT.p) + q0 * noccp, g.lda = kdim, g.a_kmajor = false;
    g.B = MOp, g.ldb = npad, g.b_kmajor = true;
    g.C = pY, g.ldc = nocc;
    gemm_f64(g, 1, s);
    dim3 grid(static_cast<unsigned>((ldp + 255) / 256), static_cast<unsigned>(std::min<long>(nq, 1024)));
    k_pack_pairs<<<grid, 256, 0, s>>>(pY, static_cast<const double*>(ctx->w.p), q0, nq, nocc, noccp, np, ldp,
                                      static_cast<double*>(Yp.p));
  }
  tm.mark(2);
  {  // Z[p][P] = sum_Q Y[Q][p] M_QP, the last row u_P = sum_Q w_Q M_QP
    GemmF64Args g;
    g.M = np + 1, g.N = naux, g.K = naux;
    g.A = static_cast<const double*>(Yp.p), g.lda = ldp, g.a_kmajor = false;
    g.B = pM, g.ldb = nauxp, g.b_kmajor = false;
    g.C = pZ, g.ldc = ldP;
    gemm_f64(g, 1, s);
    k_expand_pairs<<<dim3(static_cast<unsigned>(std::min<long>((ldP + 255) / 256, 64)), static_cast<unsigned>(std::min<long>(np + 1, 32768))),
                     256, 0, s>>>(pZ, nocc, np, naux, ldP, static_cast<double*>(Zw.p), static_cast<double*>(Zf.p));
  }
  tm.mark(3);
  if (dEdPQ) {  // dE/d(P|Q) = sum_p Zw[p][P] Z[p][Q]
    GemmF64Args g;
    g.M = naux, g.N = naux, g.K = np + 1;
    g.A = static_cast<const double*>(Zw.p), g.lda = ldP, g.a_kmajor = false;
    g.B = pZ, g.ldb = ldP, g.b_kmajor = false;
    g.C = static_cast<double*>(dV.p), g.ldc = naux;
    gemm_f64(g, 1, s);
    tm.mark(6);
  }
  if (dEdI3) {
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
    // rows mu of dE/d(P|mu nu) in blocks, each on its way to the host while the next one is formed
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
      if (prev0 >= 0) cudaStreamWaitEvent(s, ctx->ev_out[slot], 0);  // the copy of the block before the last
      GemmF64Args h;
      h.M = m1, h.N = naux, h.K = nocc;
      h.A = MOp, h.lda = npad, h.a_kmajor = false;
      h.B = pT + m0 * row, h.ldb = ldP, h.sB = row, h.b_kmajor = false;
      h.C = static_cast<double*>(out[slot].p), h.ldc = naux;
      h.mode = GEMM_DPAIRS;
      h.mu0 = m0, h.n_ao = n, h.D = pD, h.u = pu;
      gemm_f64(h, m1 - m0, s);
      cudaEventRecord(ctx->ev_blk[slot], s);
      if (prev0 >= 0) rc = copy_out(prev0, prev1, slot ^ 1);
      prev0 = m0;
      prev1 = m1;
      m0 = m1;
    }
    tm.mark(4);
    if (!rc) rc = copy_out(prev0, prev1, slot ^ 1);
  }
  if (dEdPQ && !rc)
    rc = cuda_check(ctx, cudaMemcpyAsync(dEdPQ, dV.p, static_cast<size_t>(naux) * naux * sizeof(double),
                                         cudaMemcpyDeviceToHost, s), "D2H dPQ");
  ctx->stats.grad_qchunk = qc;
  const int rc_s = cuda_check(ctx, cudaStreamSynchronize(s), "rijk_grad");
  const int rc_c = cuda_check(ctx, cudaStreamSynchronize(ctx->copy_stream), "rijk_grad copies");
  if (!rc) rc = rc_s ? rc_s : rc_c;
  if (!rc) tm.collect(ctx->stats);
  cleanup();
  return rc;
}
