// Screening that feeds the direct interaction Hd, in FP64 on the GPU.
//
//   rpa_epsilon            RPA::calculate_epsilon_r (xtp/src/libxtp/gwbse/rpa.cc:145-200):
//                          eps = 1 - 2 sum_m M_m^T diag(chi_m) M_m over occupied m, unoccupied c,
//                          chi = (w - dE)/((w - dE)^2 + (wi + eta)^2) - (w + dE)/((w + dE)^2 + (wi - eta)^2)
//                          as one weighted SYRK-shaped GEMM over the (m, c) pairs.
//   cholesky_inverse       eps^-1 = L^-T L^-1 with eps = L L^T: the dense screening W that
//                          bse_op_create_dense_screening folds into the vv block.  It replaces
//                          the host eigen-decomposition of BSE::SetupDirectInteractionOperator
//                          (bse.cc:188-204, eigenvectors rotate Mmn, epsilon_0_inv = 1/lambda):
//                          sum_PQ M^P (eps^-1)_PQ M^Q equals the rotated-diagonal form.
//   mmn_multiply_right     TCMatrix_gwbse::MultiplyRightWithAuxMatrix (threecenter.cc:54-65):
//                          every slice M[m] <- M[m] U.
#include <cmath>
#include <vector>

#include "dgemm.cuh"
#include "fast_fp64.cuh"
#include "host_eig.hpp"

namespace vgb {

namespace {

constexpr int NB = 64;  // Cholesky block

unsigned g1d(int64_t n) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), 16LL * 152));
}

// -2 chi of the (m, c) pairs: two divisions each, once per pair and not once per (pair, P)
__global__ void rpa_chi_kernel(const double *energies, int64_t n_occ_chunk, int64_t m0, int64_t n_unocc,
                               int64_t lumo_idx, double wr, double wi, double eta, double *chi2) {
  pdl_wait();
  const int64_t total = n_occ_chunk * n_unocc;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const QuotRem x = quot_rem(t, n_unocc);
    const int64_t c = x.r, mi = x.q;
    const double dE = energies[lumo_idx + c] - energies[m0 + mi];
    const double dm = wr - dE, dp = wr + dE;
    const double s1 = (wi + eta) * (wi + eta), s2 = (wi - eta) * (wi - eta);
    const double chi = dm / (dm * dm + s1) - dp / (dp * dp + s2);
    chi2[t] = -2.0 * chi;
  }
}

// B[(m, c)][P] = M(rpamin+m, lumo+c, P), and the same scaled by -2 chi_{m,c} (Bw); one grid row
// per (m, P), so that no thread divides an index.  Bound: HBM, 24 bytes an element (v32 c256
// Naux1000: 359 us with the divisions inside, 40 us).
__global__ void rpa_weights_kernel(const double *raw, int64_t n_unocc, int64_t naux, int64_t nsize, int64_t row0,
                                   const double *chi2, double *B, double *Bw, int64_t ldb, int64_t rows) {
  pdl_wait();
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {  // r = mi * naux + P
    const QuotRem x = quot_rem(r, naux);
    const int64_t mi = x.q, P = x.r;
    const double *src = raw + r * nsize + row0, *w = chi2 + mi * n_unocc;
    double *b = B + mi * n_unocc + ldb * P, *bw = Bw + mi * n_unocc + ldb * P;
    for (int64_t c = threadIdx.x; c < n_unocc; c += blockDim.x) {
      const double x = src[c];
      b[c] = x;
      bw[c] = w[c] * x;
    }
  }
}

__global__ void add_identity_kernel(double *A, int64_t n) {
  pdl_wait();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    A[i + n * i] += 1.0;
}

// Cholesky factor L and its inverse of the nb x nb (<= 64) diagonal block at A (lda), one CTA: the
// factorisation of [A | I] in registers, so that column k of L and row k of L^-1 come out
// together.  L: lower triangle, zeros above, at Lo (ldl); L^-1 likewise at Li (ldi).
// An element (i, j) holds A's until step j and L^-1's from then on, and every step is one FMA of
// column k with row k for the rows below.  Bound: the FP64 pipe (64 clocks of an SM quarter per
// warp instruction) and the pivot's chain; a warp has 8 rows, the two warps of a quarter rows q
// and 7 - q of eight, which have 18 instructions a step together whatever q (columns past the
// diagonal are left out).  64 x 64: 263 us as two kernels with divisions, 100 us from shared
// memory, 87 us.
__global__ void __launch_bounds__(256) chol_block_kernel(const double *A, int64_t lda, int nb, double *Lo,
                                                         int64_t ldl, double *Li, int64_t ldi, int *info,
                                                         int64_t j0) {
  pdl_wait();
  __shared__ double colk[NB], rowk[NB], l[NB], rk[NB];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int blk = warp < 4 ? warp : 11 - warp;  // rows 8 blk ..
  const int i = 8 * blk + (lane & 7), c = lane >> 3;  // columns c, c + 4, ..
  double v[16];
#pragma unroll
  for (int s = 0; s < 16; ++s) {
    const int j = c + 4 * s;
    v[s] = j > i ? 0.0 : (i < nb ? A[i + lda * j] : (i == j ? 1.0 : 0.0));
  }
#pragma unroll
  for (int sk = 0; sk < 16; ++sk) {
#pragma unroll 1
    for (int ck = 0; ck < 4; ++ck) {
      const int k = 4 * sk + ck;
      if (c == ck && i >= k) colk[i] = v[sk];
      if (i == k) {
#pragma unroll
        for (int s = 0; s <= sk; ++s) rowk[c + 4 * s] = v[s];
      }
      __syncthreads();
      if (warp < 4) {  // one warp per quarter: column k of L (warps 0, 1), row k of L^-1 (warps 2, 3)
        const double d = colk[k];
        const long long b = __double_as_longlong(d);  // an FP64 comparison costs what an FMA does
        const bool ok = b > 0 && b <= 0x7FF0000000000000ll;
        const double y = ok ? rsqrt64(d) : 1.0;
        const int e = (warp & 1) * 32 + lane;
        if (warp < 2) {
          const double x = e > k ? colk[e] : ok ? d : 1.0;
          const double lv = x * y;
          if (e >= k) {
            if (e > k) { l[e] = lv; rk[e] = lv; }
            if (e < nb) Lo[e + ldl * k] = lv;
          } else if (e < nb && k < nb) {
            Lo[e + ldl * k] = 0.0;
          }
          if (e == k && !ok && *info == 0) *info = (int)(j0 + k + 1);
        } else if (e <= k) {
          rk[e] = (e < k ? rowk[e] : 1.0) * y;
        }
      }
      __syncthreads();
      if (i == k) {  // row k of L^-1 is final
#pragma unroll
        for (int s = 0; s <= sk; ++s)
          if (c + 4 * s <= k) v[s] = rk[c + 4 * s];
      }
      if (8 * blk + 7 > k) {  // the warp has rows below k
        const double li = i > k ? l[i] : 0.0;
        if (c == ck && i > k) v[sk] = 0.0;
#pragma unroll
        for (int s = 0; s < 16; ++s)
          if (s <= 2 * blk + 1) v[s] = fma(-li, rk[c + 4 * s], v[s]);
      }
    }
  }
#pragma unroll
  for (int s = 0; s < 16; ++s) {
    const int j = c + 4 * s;
    if (i < nb && j < nb) Li[i + ldi * j] = j <= i ? v[s] : 0.0;
  }
}

}  // namespace

void rpa_epsilon(const bse_mmn_desc &desc, const double *const *slices, const double *energies,
                 int64_t rpatotal, int64_t homo, int64_t rpamin, int64_t rpamax, double wr, double wi,
                 double eta, double *eps_host, cudaStream_t s) {
  const int64_t naux = desc.auxsize;
  const int64_t lumo = homo + 1;
  const int64_t n_occ = lumo - rpamin, n_unocc = rpamax - lumo + 1;
  const int64_t nsize = desc.nmax - desc.nmin + 1;
  VGB_REQUIRE(n_occ >= 1 && n_unocc >= 1, "rpa_epsilon: empty occupied or unoccupied range");
  VGB_REQUIRE(rpatotal == rpamax - rpamin + 1, "rpa_epsilon: energies must cover rpamin..rpamax");
  VGB_REQUIRE(desc.mmin <= rpamin && desc.mmax >= homo, "rpa_epsilon: Mmn m-range misses occupied levels");
  VGB_REQUIRE(nsize >= n_unocc, "rpa_epsilon: Mmn n-range shorter than the unoccupied range");
  DeviceBuffer<double> dE(rpatotal), eps(naux * naux);
  VGB_CUDA(cudaMemcpyAsync(dE.get(), energies, rpatotal * sizeof(double), cudaMemcpyHostToDevice, s));
  // occupied levels in chunks so that the pair matrices stay below ~1 GB
  const int64_t per_m = n_unocc * naux;
  const int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(n_occ, (64LL << 20) / std::max<int64_t>(per_m, 1)));
  DeviceBuffer<double> raw(chunk * naux * nsize), B(chunk * per_m), Bw(chunk * per_m), chi(chunk * n_unocc);
  GemmWorkspace ws;
  for (int64_t m0 = 0; m0 < n_occ; m0 += chunk) {
    const int64_t cnt = std::min(chunk, n_occ - m0);
    for (int64_t i = 0; i < cnt; ++i) {
      const double *src = slices[rpamin + m0 + i - desc.mmin];
      VGB_REQUIRE(src != nullptr, "rpa_epsilon: null Mmn slice");
      VGB_CUDA(cudaMemcpyAsync(raw.get() + i * naux * nsize, src, naux * nsize * sizeof(double),
                               cudaMemcpyHostToDevice, s));
    }
    const int64_t rows = cnt * n_unocc;
    // Mmn_[m].bottomRows(n_unocc), as the reference reads it
    launch_pdl(rpa_chi_kernel, g1d(rows), 256, 0, s, dE.get(), cnt, m0, n_unocc, lumo - rpamin, wr, wi, eta,
               chi.get());
    VGB_LAUNCH_CHECK();
    launch_pdl(rpa_weights_kernel, (unsigned)std::min<int64_t>(cnt * naux, 64LL * sm_count()), 128, 0, s,
               raw.get(), n_unocc, naux, nsize, nsize - n_unocc, chi.get(), B.get(), Bw.get(), rows,
               cnt * naux);
    VGB_LAUNCH_CHECK();
    GemmDesc g;  // eps (+)= B^T Bw
    g.M = naux; g.N = naux; g.K = rows;
    g.a_colmajor(B.get(), rows, true).b_colmajor(Bw.get(), rows, false).c_colmajor(eps.get(), naux);
    g.beta = m0 > 0 ? 1.0 : 0.0;
    dgemm(g, s, &ws);
    VGB_CUDA(cudaStreamSynchronize(s));
  }
  launch_pdl(add_identity_kernel, g1d(naux), 256, 0, s, eps.get(), naux);
  VGB_LAUNCH_CHECK();
  VGB_CUDA(cudaMemcpyAsync(eps_host, eps.get(), naux * naux * sizeof(double), cudaMemcpyDeviceToHost, s));
  VGB_CUDA(cudaStreamSynchronize(s));
  ws.check();
}

void cholesky_inverse(int64_t n, const double *a_host, int64_t lda, double *inv_host, int64_t ldi,
                      cudaStream_t s, bool in_place) {
  VGB_REQUIRE(n >= 1 && lda >= n && ldi >= n, "cholesky_inverse: bad size");
  // Y = L^-1; L beside A, so that the panel product needs no copy, or where there is no room for a third
  // matrix in place of A's lower triangle, through a panel
  DeviceBuffer<double> A(n * n), Y(n * n), Lbeside, panel;
  if (!in_place) {
    try {
      Lbeside.resize((size_t)(n * n));
    } catch (const Error &e) {
      if (e.code != BSE_ERR_OUT_OF_MEMORY) throw;
      cudaGetLastError();
      in_place = true;
    }
  }
  if (in_place) panel.resize((size_t)(n * NB));
  double *const L = in_place ? A.get() : Lbeside.get();
  DeviceBuffer<int> info(1);
  GemmWorkspace ws;
  VGB_CUDA(cudaMemcpy2DAsync(A.get(), n * sizeof(double), a_host, lda * sizeof(double),
                             n * sizeof(double), n, cudaMemcpyHostToDevice, s));
  VGB_CUDA(cudaMemsetAsync(info.get(), 0, sizeof(int), s));
  VGB_CUDA(cudaMemsetAsync(Y.get(), 0, n * n * sizeof(double), s));
  // right-looking blocked Cholesky: A = L L^T (lower), the diagonal blocks' inverses into Y
  for (int64_t j = 0; j < n; j += NB) {
    const int nb = (int)std::min<int64_t>(NB, n - j);
    launch_pdl(chol_block_kernel, 1, 256, 0, s, A.get() + j + n * j, n, nb, L + j + n * j, n,
               Y.get() + j + n * j, n, info.get(), j);
    VGB_LAUNCH_CHECK();
    const int64_t rest = n - j - nb;
    if (rest > 0) {
      double *A21 = A.get() + (j + nb) + n * j, *L21 = in_place ? panel.get() : L + (j + nb) + n * j;
      const int64_t ld = in_place ? rest : n;
      GemmDesc t;  // L21 = A21 L11^-T
      t.M = rest; t.N = nb; t.K = nb;
      t.a_colmajor(A21, n, false).b_colmajor(Y.get() + j + n * j, n, true).c_colmajor(L21, ld);
      dgemm(t, s, &ws);
      if (in_place)
        VGB_CUDA(cudaMemcpy2DAsync(A21, n * sizeof(double), L21, ld * sizeof(double), rest * sizeof(double), nb,
                                   cudaMemcpyDeviceToDevice, s));
      GemmDesc u;  // A22 -= L21 L21^T
      u.M = rest; u.N = rest; u.K = nb;
      u.a_colmajor(L21, ld, false).b_colmajor(L21, ld, true).c_colmajor(A.get() + (j + nb) + n * (j + nb), n);
      u.alpha = -1.0; u.beta = 1.0;
      dgemm(u, s, &ws);
    }
  }
  int hinfo = 0;
  VGB_CUDA(cudaMemcpyAsync(&hinfo, info.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
  VGB_CUDA(cudaStreamSynchronize(s));
  if (hinfo != 0)
    fail(BSE_ERR_NUMERICAL, "cholesky_inverse: matrix is not positive definite (pivot " +
                                std::to_string(hinfo) + ")");
  // Y = L^-1 by doubling: of [L11 0; L21 L22] with the inverses of both diagonal blocks of h rows,
  // Y21 = -Y22 (L21 Y11), all pairs of a level at once: 2 log2(n / 64) launches of large products
  // in place of 5 small ones per block row.  T lies in A, which is free beside L; with L in place in the
  // upper triangle, transposed.
  for (int64_t h = NB; h < n; h *= 2) {
    const int64_t full = n / (2 * h);  // pairs of two whole blocks
    const int64_t i0 = full * 2 * h, last = n - i0 - h;  // a last pair whose second block is short
    for (int r = 0; r < 2; ++r) {
      const int64_t np = r == 0 ? full : (last > 0 ? 1 : 0), h2 = r == 0 ? h : last, o = r == 0 ? 0 : i0;
      if (np == 0) continue;
      const int64_t step = 2 * h * (n + 1);
      double *T = A.get() + (in_place ? o + n * (o + h) : o + h + n * o);
      const int64_t t_rs = in_place ? n : 1, t_cs = in_place ? 1 : n;
      GemmDesc t;  // T = L21 Y11
      t.M = h2; t.N = h; t.K = h;
      t.a_colmajor(L + o + h + n * o, n, false).b_colmajor(Y.get() + o + n * o, n, false);
      t.C = T; t.c_rs = t_rs; t.c_cs = t_cs;
      t.nb1 = np; t.a_b1 = step; t.b_b1 = step; t.c_b1 = step;
      dgemm(t, s, &ws);
      GemmDesc u;  // Y21 = -Y22 T
      u.M = h2; u.N = h; u.K = h2;
      u.a_colmajor(Y.get() + (o + h) * (n + 1), n, false).c_colmajor(Y.get() + o + h + n * o, n);
      u.B = T; u.b_rs = t_rs; u.b_cs = t_cs;
      u.alpha = -1.0;
      u.nb1 = np; u.a_b1 = step; u.b_b1 = step; u.c_b1 = step;
      dgemm(u, s, &ws);
    }
  }
  // A^-1 = L^-T L^-1 = Y^T Y
  GemmDesc f;
  f.M = n; f.N = n; f.K = n;
  f.a_colmajor(Y.get(), n, true).b_colmajor(Y.get(), n, false).c_colmajor(A.get(), n);
  dgemm(f, s, &ws);
  VGB_CUDA(cudaMemcpy2DAsync(inv_host, ldi * sizeof(double), A.get(), n * sizeof(double),
                             n * sizeof(double), n, cudaMemcpyDeviceToHost, s));
  VGB_CUDA(cudaStreamSynchronize(s));
  ws.check();
}

void mmn_multiply_right(const bse_mmn_desc &desc, double *const *slices, const double *U_host,
                        int64_t ldu, cudaStream_t s) {
  const int64_t naux = desc.auxsize, nsize = desc.nmax - desc.nmin + 1;
  const int64_t msize = desc.mmax - desc.mmin + 1;
  VGB_REQUIRE(naux >= 1 && nsize >= 1 && msize >= 1 && ldu >= naux, "mmn_multiply_right: bad sizes");
  DeviceBuffer<double> U(naux * naux);
  VGB_CUDA(cudaMemcpy2DAsync(U.get(), naux * sizeof(double), U_host, ldu * sizeof(double),
                             naux * sizeof(double), naux, cudaMemcpyHostToDevice, s));
  const int64_t per = nsize * naux;
  const int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(msize, (64LL << 20) / per));
  DeviceBuffer<double> in(chunk * per), out(chunk * per);
  GemmWorkspace ws;
  for (int64_t m0 = 0; m0 < msize; m0 += chunk) {
    const int64_t cnt = std::min(chunk, msize - m0);
    for (int64_t i = 0; i < cnt; ++i)
      VGB_CUDA(cudaMemcpyAsync(in.get() + i * per, slices[m0 + i], per * sizeof(double),
                               cudaMemcpyHostToDevice, s));
    GemmDesc g;  // out[m] = in[m] U  (each nsize x naux column-major)
    g.M = nsize; g.N = naux; g.K = naux;
    g.a_colmajor(in.get(), nsize, false).b_colmajor(U.get(), naux, false).c_colmajor(out.get(), nsize);
    g.nb1 = cnt; g.a_b1 = per; g.c_b1 = per;
    dgemm(g, s, &ws);
    for (int64_t i = 0; i < cnt; ++i)
      VGB_CUDA(cudaMemcpyAsync(slices[m0 + i], out.get() + i * per, per * sizeof(double),
                               cudaMemcpyDeviceToHost, s));
    VGB_CUDA(cudaStreamSynchronize(s));
    ws.check();
  }
}

// W = U diag(w) U^T with A = U diag(lambda) U^T and w = 1/lambda for lambda > cutoff, else 0:
// the screening of BSE::SetupDirectInteractionOperator (bse.cc:188-204: eigen-decomposition of
// eps, modes with lambda <= 1e-8 dropped) as one dense matrix.  The symmetric eigenproblem is
// solved on the host (as the reference does), the product U diag(w) U^T on the device.
void positive_inverse(int64_t n, const double *a_host, int64_t lda, double cutoff, double *inv_host,
                      int64_t ldi, cudaStream_t s) {
  VGB_REQUIRE(n >= 1 && lda >= n && ldi >= n, "positive_inverse: bad size");
  std::vector<double> A(n * n);
  for (int64_t j = 0; j < n; ++j)
    for (int64_t i = 0; i < n; ++i) A[i + n * j] = a_host[i + lda * j];
  std::vector<double> lam, U;
  if (!sym_eig(n, A.data(), lam, U)) fail(BSE_ERR_NUMERICAL, "positive_inverse: eigenvalue problem failed");
  std::vector<double> UW(n * n);
  for (int64_t j = 0; j < n; ++j) {
    const double w = lam[j] > cutoff ? 1.0 / lam[j] : 0.0;
    for (int64_t i = 0; i < n; ++i) UW[i + n * j] = U[i + n * j] * w;
  }
  DeviceBuffer<double> dU(n * n), dUW(n * n), dW(n * n);
  VGB_CUDA(cudaMemcpyAsync(dU.get(), U.data(), n * n * sizeof(double), cudaMemcpyHostToDevice, s));
  VGB_CUDA(cudaMemcpyAsync(dUW.get(), UW.data(), n * n * sizeof(double), cudaMemcpyHostToDevice, s));
  GemmDesc g;  // W = (U diag(w)) U^T
  g.M = n; g.N = n; g.K = n;
  g.A = dUW.get(); g.a_rs = 1; g.a_cs = n;
  g.B = dU.get(); g.b_rs = n; g.b_cs = 1;
  g.C = dW.get(); g.c_rs = 1; g.c_cs = n;
  GemmWorkspace ws;
  dgemm(g, s, &ws);
  VGB_CUDA(cudaMemcpy2DAsync(inv_host, ldi * sizeof(double), dW.get(), n * sizeof(double), n * sizeof(double), n,
                             cudaMemcpyDeviceToHost, s));
  VGB_CUDA(cudaStreamSynchronize(s));
  ws.check();
}

}  // namespace vgb
