// The harmonic-Ritz problem of the HAM Davidson on the device (FP64), one CTA per problem.
//
// DavidsonSolver::getHarmonicRitz (xtp/src/libxtp/davidsonsolver.cc:241-332) solves the
// generalized eigenproblem T u = theta B u of the projected matrices T = V^T A V and
// B = V^T A A V (Eigen::GeneralizedEigenSolver there), drops the second member of every complex
// conjugate pair, keeps the eigenvectors' real parts (normalised), takes the needed pairs with
// the largest real parts and returns lambda = diag(U^T T U).  Here, with published textbook
// steps and no library code:
//   1. B = P L U (LU with partial pivoting), C = B^-1 T;
//   2. Householder reduction of C to upper Hessenberg form H = Q^T C Q, reflectors kept;
//   3. eigenvalues of H by the Francis double-shift QR iteration with deflation (the classical
//      real-arithmetic algorithm), four warps: every warp runs the scalar recurrence, the row and
//      column updates of each bulge step are split over their lanes;
//   4. the selection of the reference (complex partners, largest real parts first);
//   5. for the selected eigenvalues only: inverse iteration on the Hessenberg matrix in complex
//      arithmetic (Hessenberg LU with partial pivoting, three steps, vectors of eigenvalues
//      closer than 1e-8 (|C| + 1) projected out of each other), back-transformation x = Q z,
//      phase fixed so that the largest component is real and positive, real part normalised.
//      Real eigenvalues apart from the others (all of them, in a stable BSE) run in real
//      arithmetic, all at once: the factorisations a warp each, the serial chains of the
//      solves a lane each, everything elementwise on the whole block.
// The matrices stay in shared memory up to m = 97.  m = 44, 10 pairs: 11.4 ms before the lane-wise
// divisions and scans and the parallel inverse iteration, 4.4 ms with them; the bits are the same.
#include "fast_fp64.cuh"
#include "small_eig.cuh"

#include <algorithm>
#include <memory>
#include <mutex>

namespace vgb {

namespace {

constexpr int kGenThreads = 256;
constexpr int kGenWarps = kGenThreads / 32;
constexpr int kGenJobs = 256;

struct GenEigGroup {
  GenEigJob j[kGenJobs];
  int n;
  int64_t smem_doubles;
};

__device__ inline double sgn_of(double a, double b) { return b >= 0.0 ? fabs(a) : -fabs(a); }

struct cplx {
  double re, im;
};
__device__ inline cplx cmul(cplx a, cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ inline cplx csub(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }
__device__ inline double cabs2(cplx a) { return a.re * a.re + a.im * a.im; }
__device__ inline cplx cdiv(cplx a, cplx b) {
  // Smith's division
  if (fabs(b.re) >= fabs(b.im)) {
    const double r = b.im / b.re, d = b.re + r * b.im;
    return {(a.re + r * a.im) / d, (a.im - r * a.re) / d};
  }
  const double r = b.re / b.im, d = b.im + r * b.re;
  return {(a.re * r + a.im) / d, (a.im * r - a.re) / d};
}

__device__ double gsum(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < kGenWarps; ++w) t += red[w];
  return t;
}
__device__ double gmax(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = red[0];
  for (int w = 1; w < kGenWarps; ++w) t = fmax(t, red[w]);
  return t;
}
__device__ double wsum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Barrier of the warps that run the QR iteration.
constexpr int kQrThreads = 128;
__device__ __forceinline__ void qr_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kQrThreads) : "memory"); }

__device__ __forceinline__ int max_exponent(double p, double q, double r) {
  auto ex = [](double x) { return (__double2hiint(x) >> 20) & 0x7FF; };
  return max(ex(p), max(ex(q), ex(r)));
}
// x 2^-sh for a normal result (else 0), in integers
__device__ __forceinline__ double scale_down(double x, int sh) {
  const int h = __double2hiint(x), e = ((h >> 20) & 0x7FF) - sh;
  return e > 0 ? __hiloint2double(h - (sh << 20), __double2loint(x)) : 0.0;
}
__device__ __forceinline__ double scale_up(double x, int sh) {
  const int h = __double2hiint(x), e = ((h >> 20) & 0x7FF) + sh;
  return e > 0 && e < 0x7FF ? __hiloint2double(h + (sh << 20), __double2loint(x)) : scalbn(x, sh);
}

// Francis double-shift QR iteration on the upper Hessenberg a (n x n, leading dimension ld),
// eigenvalues only, by the first four warps.  Returns false when an eigenvalue needs more than 60
// steps.  An FP64 instruction holds its SM quarter for 64 clocks whatever its active lanes, a
// division 565 and a square root 700, so the scalar recurrence (which every warp runs, one per
// quarter) is what it costs: independent divisions run as one instruction in different lanes,
// and the scans for a small subdiagonal and for the start of the bulge test 32 rows at once
// (one row after another they cost as much as the bulge itself).  FAST: the reflectors are scaled by
// a power of two instead of their 1-norm and built with fast_rsqrt and fast_rcp, with differences in
// the last bits (split-precision solves keep the divisions: their iterations amplify one bit).  m 44
// with 10 vectors: 4.4 ms with divisions, 3.2 ms; a bulge step is 2.8k clocks of dependent FP64
// instructions (75 each), half of them the reflector.
template <bool FAST>
__device__ __forceinline__ bool hqr_block(double *a_, int ld, int n, double *wr, double *wi) {
  const int tid = threadIdx.x, lane = tid & 31;
  auto A = [&](int r, int c) -> double & { return a_[r + ld * c]; };
  double an = 0.0;
  for (int i = 0; i < n; ++i)
    for (int j = max(0, i - 1) + lane; j < n; j += 32) an += fabs(A(i, j));
  const double anorm = wsum(an);
  int nn = n - 1;
  double t = 0.0;
  while (nn >= 0) {
    int its = 0;
    int l;
    do {
      l = 0;
      for (int base = nn; base >= 1; base -= 32) {  // the largest l with a negligible A(l, l - 1)
        const int ll = base - lane;
        bool small = false;
        if (ll >= 1) {
          double s = fabs(A(ll - 1, ll - 1)) + fabs(A(ll, ll));
          if (s == 0.0) s = anorm;
          small = fabs(A(ll, ll - 1)) + s == s;
        }
        const unsigned b = __ballot_sync(0xffffffffu, small);
        if (b) {
          l = base - (__ffs((int)b) - 1);
          break;
        }
      }
      double x = A(nn, nn);
      double y = nn >= 1 ? A(nn - 1, nn - 1) : 0.0;
      double w = nn >= 1 ? A(nn, nn - 1) * A(nn - 1, nn) : 0.0;
      qr_sync();  // every warp has read
      if (l >= 1 && tid == 0) A(l, l - 1) = 0.0;
      if (l == nn) {  // one root
        if (tid == 0) { wr[nn] = x + t; wi[nn] = 0.0; }
        --nn;
        qr_sync();
      } else {
        if (l == nn - 1) {  // two roots
          const double p = 0.5 * (y - x);
          const double q = p * p + w;
          double z = sqrt(fabs(q));
          x += t;
          if (tid == 0) {
            if (q >= 0.0) {
              z = p + sgn_of(z, p);
              wr[nn - 1] = wr[nn] = x + z;
              if (z != 0.0) wr[nn] = x - w / z;
              wi[nn - 1] = wi[nn] = 0.0;
            } else {
              wr[nn - 1] = wr[nn] = x + p;  // the pair with the positive imaginary part first
              wi[nn - 1] = z;
              wi[nn] = -z;
            }
          }
          nn -= 2;
          qr_sync();
        } else {  // one double-shift step
          if (its == 60) return false;
          if (its == 10 || its == 20) {  // exceptional shift
            t += x;
            qr_sync();
            for (int i = tid; i <= nn; i += kQrThreads) A(i, i) -= x;
            qr_sync();
            const double s = fabs(A(nn, nn - 1)) + fabs(A(nn - 1, nn - 2));
            y = x = 0.75 * s;
            w = -0.4375 * s * s;
          }
          ++its;
          qr_sync();  // A(l, l - 1) is written
          int m = l;
          double p = 0.0, q = 0.0, r = 0.0, z;
          for (int base = nn - 2; base >= l; base -= 32) {  // the largest m that may start the bulge
            const int mm = base - lane;
            bool stop = false;
            if (mm >= l) {
              z = A(mm, mm);
              r = x - z;
              const double s0 = y - z;
              p = (r * s0 - w) / A(mm + 1, mm) + A(mm, mm + 1);
              q = A(mm + 1, mm + 1) - z - r - s0;
              r = A(mm + 2, mm + 1);
              if constexpr (FAST) {
                const int ex = max_exponent(p, q, r), sh = ex == 0 || ex == 0x7FF ? 0 : ex - 1023;
                p = scale_down(p, sh);
                q = scale_down(q, sh);
                r = scale_down(r, sh);
              } else {
                const double s = fabs(p) + fabs(q) + fabs(r);
                p /= s;
                q /= s;
                r /= s;
              }
              stop = mm == l;
              if (!stop) {
                const double u = fabs(A(mm, mm - 1)) * (fabs(q) + fabs(r));
                const double v = fabs(p) * (fabs(A(mm - 1, mm - 1)) + fabs(z) + fabs(A(mm + 1, mm + 1)));
                stop = u + v == v;
              }
            }
            const unsigned b = __ballot_sync(0xffffffffu, stop);
            if (b) {
              const int src = __ffs((int)b) - 1;
              m = base - src;
              p = __shfl_sync(0xffffffffu, p, src);
              q = __shfl_sync(0xffffffffu, q, src);
              r = __shfl_sync(0xffffffffu, r, src);
              break;
            }
          }
          qr_sync();
          for (int i = m + 2 + tid; i <= nn; i += kQrThreads) {
            A(i, i - 2) = 0.0;
            if (i != m + 2) A(i, i - 3) = 0.0;
          }
          qr_sync();
          if constexpr (FAST) {
            for (int k = m; k <= nn - 1; ++k) {
              if (k != m) {
                p = A(k, k - 1);
                q = A(k + 1, k - 1);
                r = k != nn - 1 ? A(k + 2, k - 1) : 0.0;
              }
              const int ex = max_exponent(p, q, r);
              if (ex == 0) continue;  // zero
              const int sh = ex == 0x7FF ? 0 : ex - 1023;  // the largest to [1, 2); infinities and NaN stay
              p = scale_down(p, sh);
              q = scale_down(q, sh);
              r = scale_down(r, sh);
              const double n2 = fma(p, p, fma(q, q, r * r));
              // the FP32 estimates of 1 / sqrt(n2) and of 1 / (|p| + s), the second while the first is refined
              const float n2f = to_float(n2);
              float fs, fp;
              asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(fs) : "f"(n2f));
              const double pa = with_sign(p, 1.0);
              const float pf = __double2hiint(pa) >= 0x3C000000 ? to_float(pa) : 0.f;
              asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(fp) : "f"(fmaf(n2f, fs, pf)));
              const double rs0 = fast_rsqrt(n2, fs);
              const double s = with_sign(n2 * rs0, p), rs = with_sign(rs0, p);
              p += s;
              const double rp = with_sign(fast_rcp(with_sign(p, 1.0), fp), p);
              {  // p / s, q / s, r / s, q / p, r / p in lanes 0 .. 4
                const double num = lane == 0 ? p : (lane == 1 || lane == 3) ? q : r;
                const double d = num * (lane < 3 ? rs : rp);
                x = __shfl_sync(0xffffffffu, d, 0);
                y = __shfl_sync(0xffffffffu, d, 1);
                z = __shfl_sync(0xffffffffu, d, 2);
                q = __shfl_sync(0xffffffffu, d, 3);
                r = __shfl_sync(0xffffffffu, d, 4);
              }
              const bool three = k != nn - 1;
              for (int j = k + tid; j <= nn; j += kQrThreads) {
                double *a = &A(k, j);
                const double a0 = a[0], a1 = a[1], a2 = three ? a[2] : 0.0;
                double pp = fma(q, a1, a0);
                if (three) {
                  pp = fma(r, a2, pp);
                  a[2] = fma(-pp, z, a2);
                }
                a[1] = fma(-pp, y, a1);
                a[0] = fma(-pp, x, a0);
              }
              qr_sync();
              if (tid == 0) {  // every warp has read A(k, k - 1)
                if (k != m) A(k, k - 1) = scale_up(-s, sh);
                else if (l != m) A(k, k - 1) = -A(k, k - 1);
              }
              const int mmin = nn < k + 3 ? nn : k + 3;
              for (int i = l + tid; i <= mmin; i += kQrThreads) {
                double *a = &A(i, k);
                const double a0 = a[0], a1 = a[ld], a2 = three ? a[2 * ld] : 0.0;
                double pp = fma(y, a1, x * a0);
                if (three) {
                  pp = fma(z, a2, pp);
                  a[2 * ld] = fma(-pp, r, a2);
                }
                a[ld] = fma(-pp, q, a1);
                a[0] = a0 - pp;
              }
              qr_sync();
            }
          } else for (int k = m; k <= nn - 1; ++k) {
            if (k != m) {
              p = A(k, k - 1);
              q = A(k + 1, k - 1);
              r = 0.0;
              if (k != nn - 1) r = A(k + 2, k - 1);
              x = fabs(p) + fabs(q) + fabs(r);
              if (x != 0.0) {  // p / x, q / x, r / x in lanes 0, 1, 2
                const double d = (lane == 0 ? p : lane == 1 ? q : r) / x;
                p = __shfl_sync(0xffffffffu, d, 0);
                q = __shfl_sync(0xffffffffu, d, 1);
                r = __shfl_sync(0xffffffffu, d, 2);
              }
            }
            const double s = sgn_of(sqrt(p * p + q * q + r * r), p);
            if (s != 0.0) {
              qr_sync();
              if (tid == 0) {
                if (k == m) {
                  if (l != m) A(k, k - 1) = -A(k, k - 1);
                } else {
                  A(k, k - 1) = -s * x;
                }
              }
              p += s;
              {  // p / s, q / s, r / s, q / p, r / p in lanes 0 .. 4
                const double num = lane == 0 ? p : (lane == 1 || lane == 3) ? q : r;
                const double d = num / (lane < 3 ? s : p);
                x = __shfl_sync(0xffffffffu, d, 0);
                y = __shfl_sync(0xffffffffu, d, 1);
                z = __shfl_sync(0xffffffffu, d, 2);
                q = __shfl_sync(0xffffffffu, d, 3);
                r = __shfl_sync(0xffffffffu, d, 4);
              }
              for (int j = k + tid; j <= nn; j += kQrThreads) {
                double pp = A(k, j) + q * A(k + 1, j);
                if (k != nn - 1) {
                  pp += r * A(k + 2, j);
                  A(k + 2, j) -= pp * z;
                }
                A(k + 1, j) -= pp * y;
                A(k, j) -= pp * x;
              }
              qr_sync();
              const int mmin = nn < k + 3 ? nn : k + 3;
              for (int i = l + tid; i <= mmin; i += kQrThreads) {
                double pp = x * A(i, k) + y * A(i, k + 1);
                if (k != nn - 1) {
                  pp += z * A(i, k + 2);
                  A(i, k + 2) -= pp * r;
                }
                A(i, k + 1) -= pp * q;
                A(i, k) -= pp;
              }
              qr_sync();
            }
          }
        }
      }
    } while (l < nn - 1);
  }
  return true;
}

// one thread: eigenvector of the Hessenberg H (n x n, ld) for the eigenvalue lam by inverse
// iteration (three steps) in complex arithmetic, with the cluster's earlier vectors projected
// out; z (complex, n) returned normalised.  M: 2 n^2 doubles of scratch, lv / pv: n.
__device__ void hess_inverse_iteration(const double *H, int64_t ld, int64_t n, cplx lam, double cn, cplx *M,
                                       cplx *lv, double *pv, const cplx *const *cluster, int ncl, cplx *z) {
  auto Mm = [&](int64_t r, int64_t c) -> cplx & { return M[r + n * c]; };
  for (int64_t c = 0; c < n; ++c)
    for (int64_t r = 0; r < n; ++r) {
      const double h = (r <= c + 1) ? H[r + ld * c] : 0.0;
      Mm(r, c) = (r == c) ? cplx{h - lam.re, -lam.im} : cplx{h, 0.0};
    }
  const double floor_piv = 1e-300 + 1e-14 * cn;
  for (int64_t k = 0; k + 1 < n; ++k) {
    if (cabs2(Mm(k + 1, k)) > cabs2(Mm(k, k))) {  // row interchange
      for (int64_t c = k; c < n; ++c) {
        const cplx tmp = Mm(k, c);
        Mm(k, c) = Mm(k + 1, c);
        Mm(k + 1, c) = tmp;
      }
      pv[k] = 1.0;
    } else {
      pv[k] = 0.0;
    }
    if (cabs2(Mm(k, k)) == 0.0) Mm(k, k) = cplx{floor_piv, 0.0};
    const cplx li = cdiv(Mm(k + 1, k), Mm(k, k));
    lv[k] = li;
    for (int64_t c = k + 1; c < n; ++c) Mm(k + 1, c) = csub(Mm(k + 1, c), cmul(li, Mm(k, c)));
  }
  if (cabs2(Mm(n - 1, n - 1)) == 0.0) Mm(n - 1, n - 1) = cplx{floor_piv, 0.0};
  for (int64_t i = 0; i < n; ++i) z[i] = cplx{1.0 + 0.1 * sin(1.7 * (double)i + 0.3), 0.0};
  auto project = [&]() {
    for (int q = 0; q < ncl; ++q) {  // z -= y (y^H z)
      const cplx *y = cluster[q];
      cplx d{0.0, 0.0};
      for (int64_t i = 0; i < n; ++i) {
        d.re += y[i].re * z[i].re + y[i].im * z[i].im;
        d.im += y[i].re * z[i].im - y[i].im * z[i].re;
      }
      for (int64_t i = 0; i < n; ++i) z[i] = csub(z[i], cmul(d, y[i]));
    }
  };
  auto normalise = [&]() {
    double s = 0.0;
    for (int64_t i = 0; i < n; ++i) s += cabs2(z[i]);
    s = sqrt(s);
    if (s > 0.0 && isfinite(s))
      for (int64_t i = 0; i < n; ++i) { z[i].re /= s; z[i].im /= s; }
    return s;
  };
  for (int it = 0; it < 3; ++it) {
    project();
    for (int64_t k = 0; k + 1 < n; ++k) {  // the row operations of the factorisation
      if (pv[k] != 0.0) {
        const cplx tmp = z[k];
        z[k] = z[k + 1];
        z[k + 1] = tmp;
      }
      z[k + 1] = csub(z[k + 1], cmul(lv[k], z[k]));
    }
    for (int64_t k = n - 1; k >= 0; --k) {  // upper triangular solve
      cplx s = z[k];
      for (int64_t c = k + 1; c < n; ++c) s = csub(s, cmul(Mm(k, c), z[c]));
      z[k] = cdiv(s, Mm(k, k));
    }
    const double s = normalise();
    if (!(s > 0.0) || !isfinite(s)) break;
  }
  project();
  normalise();
}

// Sum over the block as gsum gives it, when only the first nact warps hold a nonzero v; one thread
// adds the warp sums (the others would only queue for the FP64 pipe).
__device__ double gsum_few(double v, double *red, int nact, bool root) {
  const int warp = threadIdx.x >> 5;
  __syncthreads();
  if (warp < nact) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[warp] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < nact; ++w) t += red[w];
    red[31] = root ? sqrt(t) : t;
    red[30] = t;
  }
  __syncthreads();
  return red[31];
}

// Shared-memory doubles of one job, in the kernel's order while they fit: the small arrays, C, the
// LU factors (then the QR copy), the reflectors, the factors of the inverse iterations.
constexpr int kInvMaxM = 128;  // largest m of the parallel inverse iteration (row in registers)
__host__ __device__ inline int64_t gen_small_doubles(int64_t m, int64_t nw) { return 4 * m + 4 * m * nw + 6 * nw + 8; }
inline int64_t gen_smem_doubles(int64_t m, int64_t nw, int64_t limit) {
  int64_t need = 0;
  if (need + gen_small_doubles(m, nw) <= limit) need += gen_small_doubles(m, nw);
  for (int i = 0; i < 3; ++i) {
    const int64_t n = i == 1 ? (m | 1) * m : m * m;
    if (need + n <= limit) need += n;
  }
  if (need + nw * m * m <= limit) need += nw * m * m;
  return need;
}

// The vectors of ns selected eigenvalues that are real and apart from the others, listed in
// idx[0 .. L): inverse iteration on H = C (Hessenberg), x = Q z, normalisation, lambda.  The
// operations and their order are those of hess_inverse_iteration with zero imaginary parts.
// z, pr, lv: m x L (element (i, j) at i * L + j); pv likewise; U: row-major m x m per vector.
__device__ void real_vectors(const GenEigJob &q, const double *C, const double *Vh, const double *wr, const int *selv,
                             const int *idx, int L, double cn, double *z, double *pr, double *lv, double *pv,
                             double *scal, double *Uf) {
  const int m = (int)q.m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double floor_piv = 1e-300 + 1e-14 * cn;
  // ---- factorisations: a warp per vector, the current row in registers ----
  constexpr int R = kInvMaxM / 32;
  for (int j = warp; j < L; j += kGenWarps) {
    const double lam = wr[selv[idx[j]]] + 1e-10 * (cn + 1.0);
    double *U = Uf + (int64_t)j * m * m;
    double cur[R], nxt[R];
    auto load_row = [&](int r, double (&row)[R]) {
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int c = lane + 32 * u;
        double h = 0.0;
        if (c < m && r <= c + 1) h = C[r + m * c];
        row[u] = c == r ? __dsub_rn(h, lam) : h;
      }
    };
    auto at = [&](const double (&row)[R], int c) {
      double v = row[0];
#pragma unroll
      for (int u = 1; u < R; ++u)
        if (c >= 32 * u) v = row[u];
      return __shfl_sync(0xffffffffu, v, c & 31);
    };
    load_row(0, cur);
    for (int k = 0; k + 1 < m; ++k) {
      load_row(k + 1, nxt);
      double a = at(cur, k), b = at(nxt, k);
      const bool swap = __dmul_rn(b, b) > __dmul_rn(a, a);
      if (swap) {
#pragma unroll
        for (int u = 0; u < R; ++u) {
          const double t = cur[u];
          cur[u] = nxt[u];
          nxt[u] = t;
        }
        const double t = a;
        a = b;
        b = t;
      }
      if (__dmul_rn(a, a) == 0.0) a = floor_piv;
      const double li = b / a;
      if (lane == 0) {
        lv[k * L + j] = li;
        pv[k * L + j] = swap ? 1.0 : 0.0;
      }
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int c = lane + 32 * u;
        if (c >= k && c < m) U[k * m + c] = c == k ? a : cur[u];
        if (32 * u + 31 > k && 32 * u < m) nxt[u] = __dsub_rn(nxt[u], __dmul_rn(li, cur[u]));
        cur[u] = nxt[u];
      }
    }
    double a = at(cur, m - 1);
    if (__dmul_rn(a, a) == 0.0) a = floor_piv;
    if (lane == 0) U[(m - 1) * m + m - 1] = a;
  }
  for (int t = tid; t < m * L; t += kGenThreads) {
    const int i = t / L;
    z[t] = 1.0 + 0.1 * sin(1.7 * (double)i + 0.3);
  }
  int *alive = reinterpret_cast<int *>(scal + L);
  for (int j = tid; j < L; j += kGenThreads) alive[j] = 1;
  __syncthreads();
  // z /= |z| over the live vectors (all of them when final)
  auto normalise = [&](bool final) {
    for (int j = tid; j < L; j += kGenThreads) {
      double s = 0.0;
      for (int i = 0; i < m; ++i) s = __dadd_rn(s, __dmul_rn(z[i * L + j], z[i * L + j]));
      s = sqrt(s);
      const bool ok = s > 0.0 && isfinite(s);
      const bool act = final || alive[j];
      scal[j] = ok && act ? s : 0.0;  // 0: leave the vector
      if (!final && act && !ok) alive[j] = 0;
    }
    __syncthreads();
    for (int t = tid; t < m * L; t += kGenThreads) {
      const double s = scal[t % L];
      if (s != 0.0) z[t] /= s;
    }
    __syncthreads();
  };
  for (int it = 0; it < 3; ++it) {
    for (int j = tid; j < L; j += kGenThreads)
      if (alive[j])
        for (int k = 0; k + 1 < m; ++k) {  // the row operations of the factorisation
          double a = z[k * L + j], b = z[(k + 1) * L + j];
          if (pv[k * L + j] != 0.0) {
            const double t = a;
            a = b;
            b = t;
            z[k * L + j] = a;
          }
          z[(k + 1) * L + j] = __dsub_rn(b, __dmul_rn(lv[k * L + j], a));
        }
    __syncthreads();
    for (int k = m - 1; k >= 0; --k) {  // upper triangular solve: products, then the chain
      const int nc = m - 1 - k;
      for (int t = tid; t < nc * L; t += kGenThreads) {
        const int j = t / nc, c = k + 1 + t % nc;  // lanes along a row of U
        pr[c * L + j] = __dmul_rn(Uf[(int64_t)j * m * m + k * m + c], z[c * L + j]);
      }
      __syncthreads();
      for (int j = tid; j < L; j += kGenThreads)
        if (alive[j]) {
          double s = z[k * L + j];
          for (int c = k + 1; c < m; ++c) s = __dsub_rn(s, pr[c * L + j]);
          z[k * L + j] = s / Uf[(int64_t)j * m * m + k * m + k];
        }
      __syncthreads();
    }
    normalise(false);
  }
  normalise(true);
  // ---- x = Q z: reflectors in reverse order ----
  for (int k = m - 3; k >= 0; --k) {
    const double *v = Vh + m * k;
    for (int j = tid; j < L; j += kGenThreads) {
      double d = 0.0;
      for (int i = k + 1; i < m; ++i) d = fma(v[i], z[i * L + j], d);
      scal[j] = 2.0 * d;
    }
    __syncthreads();
    for (int t = tid; t < (m - 1 - k) * L; t += kGenThreads) {
      const int i = k + 1 + t / L, j = t % L;
      z[i * L + j] = fma(-scal[j], v[i], z[i * L + j]);
    }
    __syncthreads();
  }
  // normalise; sign: the largest component positive
  for (int j = tid; j < L; j += kGenThreads) {
    double nx = 0.0, best = __dmul_rn(z[j], z[j]), xm = z[j];
    for (int i = 0; i < m; ++i) {
      const double x = z[i * L + j], x2 = __dmul_rn(x, x);
      nx = __dadd_rn(nx, x2);
      if (x2 > best) {
        best = x2;
        xm = x;
      }
    }
    scal[j] = sqrt(nx);
    const double ax = sqrt(best);
    pr[j] = ax > 0.0 ? xm / ax : 1.0;
  }
  __syncthreads();
  for (int t = tid; t < m * L; t += kGenThreads) {
    const int j = t % L;
    z[t] = scal[j] > 0.0 ? __dmul_rn(z[t], pr[j]) / scal[j] : 0.0;
  }
  __syncthreads();
  for (int j = tid; j < L; j += kGenThreads) {
    double nu = 0.0;
    for (int i = 0; i < m; ++i) nu = fma(z[i * L + j], z[i * L + j], nu);
    scal[j] = sqrt(nu);
  }
  __syncthreads();
  for (int t = tid; t < m * L; t += kGenThreads) {
    const int i = t / L, j = t % L;
    if (scal[j] > 0.0) z[t] /= scal[j];
    q.U[i + q.ldu * idx[j]] = z[t];
  }
  __syncthreads();
  for (int t = tid; t < m * L; t += kGenThreads) {  // lambda = u^T T u
    const int a = t % m, j = t / m;
    double tu = 0.0;
    for (int b = 0; b < m; ++b) tu = fma(q.T[a + q.ldt * b], z[b * L + j], tu);
    pr[a * L + j] = tu;
  }
  __syncthreads();
  for (int j = tid; j < L; j += kGenThreads) {
    double lam = 0.0;
    for (int a = 0; a < m; ++a) lam = fma(z[a * L + j], pr[a * L + j], lam);
    q.lam[idx[j]] = lam;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kGenThreads) gen_eig_kernel(const __grid_constant__ GenEigGroup g) {
  pdl_wait();
  const GenEigJob q = g.j[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ double red[32];
  __shared__ int flag, bestidx, nsel, ncand, nreal;
  __shared__ double pivinv, cnorm;
  if (q.m < 1 || q.nw < 1 || q.nw > q.m || q.m > kGenEigMaxM) {
    if (tid == 0 && q.info) { q.info[0] = 1; q.info[1] = 0; }
    return;
  }
  const int m = (int)q.m, nw = (int)q.nw;
  const int64_t mm = (int64_t)m * m;
  const int hl = m | 1;  // odd: a row of the QR copy touches every bank
  extern __shared__ double sm[];
  // global scratch: LU, C, Vh, 5 m small, then per selected vector 2 m^2 + 5 m, then m (m + 1)
  double *gLU = q.work, *gC = gLU + mm, *gVh = gC + mm, *gsmall = gVh + mm, *vec = gsmall + 5 * (int64_t)m;
  int64_t off = 0;
  auto place = [&](int64_t n, double *glob) {
    if (off + n > g.smem_doubles) return glob;
    double *p = sm + off;
    off += n;
    return p;
  };
  double *small = place(gen_small_doubles(m, nw), (double *)nullptr);
  double *C = place(mm, gC);
  double *LU = place((int64_t)hl * m, gLU);  // then the QR copy
  double *Vh = place(mm, gVh);
  double *Uf = place((int64_t)nw * mm, vec);
  double *Hq = LU == gLU ? vec + nw * (2 * mm + 5 * (int64_t)m) : LU;
  double *piv = small ? small : gsmall, *wr = piv + m, *wi = wr + m, *colv = wi + m;
  int *selv = reinterpret_cast<int *>(small ? small + 4 * m + 4 * (int64_t)m * nw
                                            : vec + nw * (2 * mm + 5 * (int64_t)m) + (int64_t)hl * m);
  if (tid == 0) flag = 0;
  // ---- load ----
  double bm = 0.0;
  for (int t = tid; t < mm; t += kGenThreads) {
    const int r = t % m, c = t / m;
    const double v = q.B[r + q.ldt * c];
    LU[t] = v;
    C[t] = q.T[r + q.ldt * c];
    bm = fmax(bm, fabs(v));
  }
  const double tiny = gmax(bm, red) * 1e-300 + 1e-300;
  __syncthreads();
  // ---- 1. B = P L U ----
  for (int k = 0; k < m; ++k) {
    if (warp == 0) {  // pivot: the first largest |LU(i, k)|, i >= k
      unsigned long long best = 0;
      int p = k;
      for (int i = k + lane; i < m; i += 32) {
        const unsigned long long v = (unsigned long long)__double_as_longlong(LU[i + m * k]) & ~(1ull << 63);
        if (v > best || i == k + lane) { best = v; p = i; }
      }
      if (k + lane >= m) p = m;
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, best, o);
        const int pi = __shfl_xor_sync(0xffffffffu, p, o);
        if (v > best || (v == best && pi < p)) { best = v; p = pi; }
      }
      if (lane == 0) {
        bestidx = p;
        piv[k] = (double)p;
        if (__longlong_as_double((long long)best) <= tiny) flag = 2;
        pivinv = 1.0 / LU[p + m * k];
      }
    }
    __syncthreads();
    if (flag) break;
    const int p = bestidx;
    if (p != k)
      for (int c = tid; c < m; c += kGenThreads) {
        const double t = LU[k + m * c];
        LU[k + m * c] = LU[p + m * c];
        LU[p + m * c] = t;
      }
    __syncthreads();
    const double inv = pivinv;
    for (int i = k + 1 + tid; i < m; i += kGenThreads) LU[i + m * k] *= inv;
    __syncthreads();
    const int nr = m - k - 1;
    for (int t = tid; t < nr * nr; t += kGenThreads) {
      const int i = k + 1 + t % nr, c = k + 1 + t / nr;
      LU[i + m * c] -= LU[i + m * k] * LU[k + m * c];
    }
    __syncthreads();
  }
  if (flag) {
    if (tid == 0 && q.info) { q.info[0] = 2; q.info[1] = 0; }
    return;
  }
  // ---- C = B^-1 T: every column's operations in order, all columns at once ----
  for (int c = tid; c < m; c += kGenThreads) {
    double *x = C + (int64_t)m * c;
    for (int k = 0; k < m; ++k) {
      const int p = (int)piv[k];
      const double t = x[k];
      x[k] = x[p];
      x[p] = t;
    }
  }
  __syncthreads();
  for (int k = 0; k + 1 < m; ++k) {
    const int nr = m - k - 1;
    for (int t = tid; t < nr * m; t += kGenThreads) {
      const int i = k + 1 + t % nr, c = t / nr;
      C[i + m * c] -= LU[i + m * k] * C[k + m * c];
    }
    __syncthreads();
  }
  for (int k = m - 1; k >= 0; --k) {
    for (int c = tid; c < m; c += kGenThreads) C[k + m * c] /= LU[k + m * k];
    __syncthreads();
    for (int t = tid; t < k * m; t += kGenThreads) {
      const int i = t % k, c = t / k;
      C[i + m * c] -= LU[i + m * k] * C[k + m * c];
    }
    __syncthreads();
  }
  for (int t = tid; t < mm; t += kGenThreads)
    if (!isfinite(C[t])) flag = 2;
  __syncthreads();
  if (flag) {
    if (tid == 0 && q.info) { q.info[0] = 2; q.info[1] = 0; }
    return;
  }
  double cm = 0.0;
  for (int t = tid; t < mm; t += kGenThreads) cm = fmax(cm, fabs(C[t]));
  cm = gmax(cm, red);
  if (tid == 0) cnorm = cm;
  // ---- 2. Hessenberg reduction, reflectors kept in Vh (column k: rows k+1..m-1) ----
  for (int t = tid; t < mm; t += kGenThreads) Vh[t] = 0.0;
  __syncthreads();
  for (int k = 0; k + 2 < m; ++k) {
    const int nact = min(kGenWarps, (m - k - 1 + 31) / 32);  // warps with a row
    double sp = 0.0;
    for (int i = k + 1 + tid; i < m; i += kGenThreads) sp += fabs(C[i + m * k]);
    const double scale = gsum_few(sp, red, nact, false);
    if (scale == 0.0) continue;
    double sg = 0.0;
    for (int i = k + 1 + tid; i < m; i += kGenThreads) {
      const double v = C[i + m * k] / scale;
      Vh[i + m * k] = v;
      sg += v * v;
    }
    const double root = gsum_few(sg, red, nact, true);
    if (tid == 0) Vh[(k + 1) + m * k] -= -sgn_of(root, Vh[(k + 1) + m * k]);
    __syncthreads();
    double sv = 0.0;
    for (int i = k + 1 + tid; i < m; i += kGenThreads) sv += Vh[i + m * k] * Vh[i + m * k];
    const double vn = gsum_few(sv, red, nact, true);
    if (red[30] == 0.0) {
      for (int i = k + 1 + tid; i < m; i += kGenThreads) Vh[i + m * k] = 0.0;
      __syncthreads();
      continue;
    }
    for (int i = k + 1 + tid; i < m; i += kGenThreads) Vh[i + m * k] /= vn;
    __syncthreads();
    const double *v = Vh + m * k;
    const int nr = m - k - 1;
    for (int c = tid; c < m; c += kGenThreads) {  // C <- H C (columns)
      double s = 0.0;
      for (int i = k + 1; i < m; ++i) s += v[i] * C[i + m * c];
      s *= 2.0;
      colv[c] = s;
    }
    __syncthreads();
    for (int t = tid; t < nr * m; t += kGenThreads) {
      const int i = k + 1 + t % nr, c = t / nr;
      C[i + m * c] -= colv[c] * v[i];
    }
    __syncthreads();
    for (int r = tid; r < m; r += kGenThreads) {  // C <- C H (rows)
      double s = 0.0;
      for (int i = k + 1; i < m; ++i) s += C[r + m * i] * v[i];
      s *= 2.0;
      colv[r] = s;
    }
    __syncthreads();
    for (int t = tid; t < nr * m; t += kGenThreads) {
      const int r = t % m, i = k + 1 + t / m;
      C[r + m * i] -= colv[r] * v[i];
    }
    __syncthreads();
    for (int i = k + 2 + tid; i < m; i += kGenThreads) C[i + m * k] = 0.0;
    __syncthreads();
  }
  // ---- 3. eigenvalues: QR iteration on a copy of H, by the first four warps ----
  for (int t = tid; t < mm; t += kGenThreads) {
    const int c = t / m;
    Hq[t - c * m + hl * c] = C[t];
  }
  __syncthreads();
  if (tid < kQrThreads) {
    bool ok;
    if (q.fast && Hq == LU) ok = hqr_block<true>(sm + (Hq - sm), hl, m, wr, wi);  // shared loads, not generic ones
    else if (q.fast) ok = hqr_block<true>(Hq, hl, m, wr, wi);
    else ok = hqr_block<false>(Hq, hl, m, wr, wi);
    if (!ok && tid == 0) flag = 3;
  }
  __syncthreads();
  if (flag) {
    if (tid == 0 && q.info) { q.info[0] = 3; q.info[1] = 0; }
    return;
  }
  // ---- 4. the reference's selection (davidsonsolver.cc:261-320) ----
  int *pf = reinterpret_cast<int *>(Hq);  // first, second, per open pair (Hq is free now)
  int *cand = pf + 2 * m;
  if (tid == 0) {
    // complex partners: the second member of each pair is dropped
    int np = 0;
    for (int i = 0; i < m; ++i) {
      if (wi[i] == 0.0) continue;
      bool found = false;
      for (int p = 0; p < np; ++p) {
        if (pf[2 * p + 1] > -1) continue;
        const int f = pf[2 * p];
        if (fabs(wr[f] - wr[i]) < 1e-9 && fabs(wi[f] + wi[i]) < 1e-9) {
          pf[2 * p + 1] = i;
          found = true;
        }
      }
      if (!found) { pf[2 * np] = i; pf[2 * np + 1] = -1; ++np; }
    }
    for (int p = 0; p < np; ++p)
      if (pf[2 * p + 1] < 0) { flag = 4; q.info[1] = pf[2 * p]; }
    if (!flag) {
      int nc = 0;
      for (int i = 0; i < m; ++i) {
        bool second = false;
        for (int p = 0; p < np; ++p) second = second || pf[2 * p + 1] == i;
        if (!second) cand[nc++] = i;
      }
      ncand = nc;
      nsel = min(nc, nw);
      nreal = 0;
    }
  }
  __syncthreads();
  if (flag) {
    if (tid == 0 && q.info) q.info[0] = 4;
    return;
  }
  // stable ascending order of the candidates by real part, then reversed: each one's rank
  for (int a = tid; a < ncand; a += kGenThreads) {
    const double x = wr[cand[a]];
    int rank = 0;
    for (int b = 0; b < ncand; ++b) {
      const double y = wr[cand[b]];
      rank += (y < x || (y == x && b < a)) ? 1 : 0;
    }
    const int pos = ncand - 1 - rank;
    if (pos < nw) selv[pos] = cand[a];
  }
  __syncthreads();
  // ---- 5. eigenvectors of the selected eigenvalues ----
  const double cn = cnorm;
  const int ns = nsel;
  // clusters: runs of the selection (ordered by real part) whose neighbours are closer than
  // 1e-8 (|C| + 1); each run is handled by one thread, its vectors one after another
  auto close_to_prev = [&](int c) {
    if (c == 0) return false;
    const int a = selv[c], b = selv[c - 1];
    return hypot(wr[a] - wr[b], wi[a] - wi[b]) <= 1e-8 * (cn + 1.0);
  };
  // real eigenvalues that are clusters of one: all at once
  int *fast = selv + nw;  // 1 when handled there, then their list
  int *list = fast + nw;
  const bool can = small != nullptr && m <= kInvMaxM;
  for (int c = tid; c < nw; c += kGenThreads)
    fast[c] = can && c < ns && wi[selv[c]] == 0.0 && !close_to_prev(c) && !(c + 1 < ns && close_to_prev(c + 1));
  __syncthreads();
  if (tid == 0) {
    int n = 0;
    for (int c = 0; c < ns; ++c)
      if (fast[c]) list[n++] = c;
    nreal = n;
  }
  __syncthreads();
  if (nreal > 0) {
    double *z = small + 4 * m, *pr = z + (int64_t)m * nw, *lv = pr + (int64_t)m * nw, *pv = lv + (int64_t)m * nw;
    double *scal = small + 4 * m + 4 * (int64_t)m * nw + 2 * nw;  // behind selv, fast and list
    real_vectors(q, C, Vh, wr, selv, list, nreal, cn, z, pr, lv, pv, scal, Uf);
  }
  for (int c0 = tid; c0 < ns; c0 += kGenThreads) {
    if (fast[c0] || close_to_prev(c0)) continue;  // done, or not the first of its run
    const cplx *members[64];
    int nmem = 0;
    for (int c = c0; c < ns && (c == c0 || close_to_prev(c)); ++c) {
      const int64_t ic = selv[c];
      double *w = vec + (int64_t)c * (2 * mm + 5 * (int64_t)m);
      cplx *M = reinterpret_cast<cplx *>(w);
      cplx *lv = reinterpret_cast<cplx *>(w + 2 * mm);
      double *pv = w + 2 * mm + 2 * m;
      cplx *z = reinterpret_cast<cplx *>(w + 2 * mm + 3 * m);  // 2 m doubles
      hess_inverse_iteration(C, m, m, cplx{wr[ic] + 1e-10 * (cn + 1.0), wi[ic]}, cn, M, lv, pv, members,
                             nmem < 64 ? nmem : 64, z);
      if (nmem < 64) members[nmem++] = z;
      // x = Q z (reflectors in reverse order): stored over M, which is free now
      cplx *x = M;
      for (int64_t i = 0; i < m; ++i) x[i] = z[i];
      for (int64_t k = m - 3; k >= 0; --k) {
        const double *v = Vh + m * k;
        cplx d{0.0, 0.0};
        for (int64_t i = k + 1; i < m; ++i) { d.re += v[i] * x[i].re; d.im += v[i] * x[i].im; }
        for (int64_t i = k + 1; i < m; ++i) { x[i].re -= 2.0 * d.re * v[i]; x[i].im -= 2.0 * d.im * v[i]; }
      }
      // normalise, phase: the largest component real and positive; keep the real part
      double nx = 0.0;
      int64_t im = 0;
      for (int64_t i = 0; i < m; ++i) {
        nx += cabs2(x[i]);
        if (cabs2(x[i]) > cabs2(x[im])) im = i;
      }
      nx = sqrt(nx);
      const double ax = sqrt(cabs2(x[im]));
      const cplx ph = ax > 0.0 ? cplx{x[im].re / ax, -x[im].im / ax} : cplx{1.0, 0.0};
      double *u = q.U + q.ldu * c;
      double nu = 0.0;
      for (int64_t i = 0; i < m; ++i) {
        const double re = (nx > 0.0) ? (x[i].re * ph.re - x[i].im * ph.im) / nx : 0.0;
        u[i] = re;
        nu += re * re;
      }
      nu = sqrt(nu);
      if (nu > 0.0)
        for (int64_t i = 0; i < m; ++i) u[i] /= nu;
      // lambda = u^T T u
      double lam = 0.0;
      for (int64_t a = 0; a < m; ++a) {
        double tu = 0.0;
        for (int64_t b = 0; b < m; ++b) tu += q.T[a + q.ldt * b] * u[b];
        lam += u[a] * tu;
      }
      q.lam[c] = lam;
    }
  }
  __syncthreads();
  for (int64_t c = ns + warp; c < nw; c += kGenWarps)  // fewer candidates than wanted: zero columns
    for (int64_t i = lane; i < m; i += 32) {
      q.U[i + q.ldu * c] = 0.0;
      if (i == 0) q.lam[c] = 0.0;
    }
  if (tid == 0 && q.info) { q.info[0] = 0; q.info[1] = ns; }
}

// O = an orthonormal basis of the columns of U (m x r): modified Gram-Schmidt twice, one CTA.
__global__ void __launch_bounds__(kGenThreads) orthonormalise_kernel(const double *U, int64_t ldu, int64_t m,
                                                                    int64_t r, double *O, int64_t ldo) {
  pdl_wait();
  __shared__ double red[32];
  for (int64_t t = threadIdx.x; t < m * r; t += kGenThreads) O[(t % m) + ldo * (t / m)] = U[(t % m) + ldu * (t / m)];
  __syncthreads();
  for (int pass = 0; pass < 2; ++pass)
    for (int64_t j = 0; j < r; ++j) {
      double *oj = O + ldo * j;
      for (int64_t i = 0; i < j; ++i) {
        const double *oi = O + ldo * i;
        double s = 0.0;
        for (int64_t t = threadIdx.x; t < m; t += kGenThreads) s += oi[t] * oj[t];
        const double h = gsum(s, red);
        for (int64_t t = threadIdx.x; t < m; t += kGenThreads) oj[t] -= h * oi[t];
        __syncthreads();
      }
      double s = 0.0;
      for (int64_t t = threadIdx.x; t < m; t += kGenThreads) s += oj[t] * oj[t];
      const double nrm = sqrt(gsum(s, red));
      if (nrm > 0.0)
        for (int64_t t = threadIdx.x; t < m; t += kGenThreads) oj[t] /= nrm;
      __syncthreads();
    }
}

// The symmetric-definite pencil (S, J) of the HAM polish reduced to a standard problem:
// S = L L^T (Cholesky, lower), Mneg = -L^-1 J L^-T.  S: lower triangle read, J: full; both
// m x m with leading dimension ld.  W: 3 m^2 doubles (L, then Y = L^-1 J, then Mneg, each ld m);
// status = 1 when S is not positive definite, else 0.
__global__ void __launch_bounds__(kGenThreads) pencil_reduce_kernel(const double *S, const double *J, int64_t ld,
                                                                   int64_t m, double *W, int *status) {
  pdl_wait();
  __shared__ int bad;
  double *L = W, *Y = W + m * m, *Mn = W + 2 * m * m;
  if (threadIdx.x == 0) bad = 0;
  for (int64_t t = threadIdx.x; t < m * m; t += kGenThreads) {
    const int64_t r = t % m, c = t / m;
    L[t] = r >= c ? S[r + ld * c] : 0.0;
  }
  __syncthreads();
  for (int64_t k = 0; k < m; ++k) {  // right-looking Cholesky
    if (threadIdx.x == 0) {
      const double d = L[k + m * k];
      if (!(d > 0.0)) bad = 1;
      else L[k + m * k] = sqrt(d);
    }
    __syncthreads();
    if (bad) break;
    const double inv = 1.0 / L[k + m * k];
    for (int64_t i = k + 1 + threadIdx.x; i < m; i += kGenThreads) L[i + m * k] *= inv;
    __syncthreads();
    const int64_t nr = m - k - 1;
    for (int64_t t = threadIdx.x; t < nr * nr; t += kGenThreads) {
      const int64_t i = k + 1 + t % nr, c = k + 1 + t / nr;
      if (i >= c) L[i + m * c] -= L[i + m * k] * L[c + m * k];
    }
    __syncthreads();
  }
  if (bad) {
    if (threadIdx.x == 0) *status = 1;
    return;
  }
  for (int64_t c = threadIdx.x; c < m; c += kGenThreads) {  // Y = L^-1 J, one column per thread
    double *y = Y + m * c;
    for (int64_t r = 0; r < m; ++r) {
      double t = J[r + ld * c];
      for (int64_t k = 0; k < r; ++k) t -= L[r + m * k] * y[k];
      y[r] = t / L[r + m * r];
    }
  }
  __syncthreads();
  // M = L^-1 Y^T (M = Y L^-T is symmetric): column r of M from row r of Y; stored negated
  for (int64_t r = threadIdx.x; r < m; r += kGenThreads) {
    double *z = Mn + m * r;
    for (int64_t i = 0; i < m; ++i) {
      double t = Y[r + m * i];
      for (int64_t k = 0; k < i; ++k) t += L[i + m * k] * z[k];  // z holds -M: subtracting becomes adding
      z[i] = -t / L[i + m * i];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) *status = 0;
}

// After the eigenproblem of Mneg (ascending eigenvalues nu = -mu, eigenvectors Z, ld m): the np
// lowest positive roots omega = 1 / mu = -1 / nu and u = L^-T z.  status = 2 when fewer than np of
// the mu are positive.
__global__ void pencil_finish_kernel(const double *W, int64_t m, const double *nu, const double *Z, int64_t np,
                                     double *U, double *lam, int *status) {
  pdl_wait();
  const double *L = W;
  for (int64_t j = threadIdx.x; j < np; j += blockDim.x) {
    if (!(nu[j] < 0.0)) *status = 2;
    lam[j] = -1.0 / nu[j];
    double *u = U + m * j;
    const double *z = Z + m * j;
    for (int64_t r = m - 1; r >= 0; --r) {  // L^T u = z
      double t = z[r];
      for (int64_t k = r + 1; k < m; ++k) t -= L[k + m * r] * u[k];
      u[r] = t / L[r + m * r];
    }
  }
}

}  // namespace

void pencil_reduce_device(const double *S, const double *J, int64_t ld, int64_t m, double *W, int *status,
                          cudaStream_t s) {
  VGB_REQUIRE(m >= 1 && ld >= m, "pencil_reduce: invalid sizes");
  launch_pdl(pencil_reduce_kernel, 1, kGenThreads, 0, s, S, J, ld, m, W, status);
  VGB_LAUNCH_CHECK();
}

void pencil_finish_device(const double *W, int64_t m, const double *nu, const double *Z, int64_t np, double *U,
                          double *lam, int *status, cudaStream_t s) {
  launch_pdl(pencil_finish_kernel, 1, 128, 0, s, W, m, nu, Z, np, U, lam, status);
  VGB_LAUNCH_CHECK();
}

int64_t gen_eig_work_doubles(int64_t m, int64_t nw) {
  return 3 * m * m + 5 * m + nw * (2 * m * m + 5 * m) + m * (m + 1) + 2 * nw + 64;
}

void gen_eig_device(const GenEigJob *jobs, int64_t njobs, cudaStream_t s) {
  if (njobs <= 0) return;
  int dev = 0;
  VGB_CUDA(cudaGetDevice(&dev));
  int optin = 0;
  VGB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes fa;
  VGB_CUDA(cudaFuncGetAttributes(&fa, gen_eig_kernel));
  const int dyn_max = optin - (int)fa.sharedSizeBytes;
  static std::mutex mu;
  static int configured[64] = {0};
  {
    std::lock_guard<std::mutex> lk(mu);
    if (dev < 64 && !configured[dev]) {
      VGB_CUDA(cudaFuncSetAttribute(gen_eig_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn_max));
      configured[dev] = 1;
    }
  }
  const int64_t limit = dyn_max / (int64_t)sizeof(double);
  std::unique_ptr<GenEigGroup> g(new GenEigGroup());
  for (int64_t b = 0; b < njobs; b += kGenJobs) {
    g->n = (int)std::min<int64_t>(kGenJobs, njobs - b);
    int64_t need = 0;
    for (int i = 0; i < g->n; ++i) {
      const GenEigJob &jb = jobs[b + i];
      VGB_REQUIRE(jb.m >= 1 && jb.m <= kGenEigMaxM && jb.nw >= 1 && jb.nw <= jb.m && jb.ldu >= jb.m &&
                      jb.ldt >= jb.m && jb.work != nullptr && jb.info != nullptr,
                  "small generalized eigenproblem: invalid job");
      g->j[i] = jb;
      need = std::max(need, gen_smem_doubles(jb.m, jb.nw, limit));
    }
    g->smem_doubles = need;
    launch_pdl(gen_eig_kernel, g->n, kGenThreads, need * sizeof(double), s, *g);
    VGB_LAUNCH_CHECK();
  }
}

void orthonormalise_device(const double *U, int64_t ldu, int64_t m, int64_t r, double *O, int64_t ldo,
                           cudaStream_t s) {
  VGB_REQUIRE(m >= 1 && r >= 1 && r <= m && ldu >= m && ldo >= m, "orthonormalise: invalid sizes");
  launch_pdl(orthonormalise_kernel, 1, kGenThreads, 0, s, U, ldu, m, r, O, ldo);
  VGB_LAUNCH_CHECK();
}

}  // namespace vgb
