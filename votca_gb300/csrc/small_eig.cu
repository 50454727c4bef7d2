// Small dense symmetric eigenproblems on the device; the method is described in small_eig.cuh.
#include "small_eig.cuh"

#include "fast_fp64.cuh"

#include <algorithm>
#include <memory>
#include <mutex>

namespace vgb {

namespace {

constexpr int kEigThreads = 256;
constexpr int kEigWarps = kEigThreads / 32;
constexpr int kEigJobs = 256;  // jobs per launch (kernel-parameter space)

struct SymEigGroup {
  SymEigJob j[kEigJobs];
  int n;
  int64_t smem_doubles;  // dynamic shared memory of the launch
};

__host__ __device__ inline int64_t eig_ld(int64_t m) { return (m % 2 == 0) ? m + 1 : m; }
// doubles of the vector part of the shared layout: d, e, tau, v, p (5m), 32 reduction slots,
// then 3m + 2 four-byte words (FP32 diagonal, FP32 squared off-diagonal, FP32 eigenvalues)
// and m + 1 cluster starts
__host__ __device__ inline int64_t eig_vec_doubles(int64_t m) { return 5 * m + 32 + (4 * m + 4) / 2 + 2; }

// The sum over the block of v, of which only the first nact warps hold nonzeros, in two steps: a
// butterfly in those warps, then (after the caller's barrier) the warp sums in pairs, in a fixed
// order.  Idle warps stay off the FP64 pipe: an instruction holds its SM quarter for 64 clocks
// whatever its active lanes, so eight warps repeating a scalar queue two deep in every quarter.
__device__ __forceinline__ void sum_warps(double v, double *red, int nact, int64_t n) {
  const int warp = threadIdx.x >> 5;
  if (warp < nact) {
    // the first n lanes hold the values when one warp does: levels that add only zeros are left out
    for (int o = n > 16 ? 16 : n > 8 ? 8 : n > 4 ? 4 : n > 2 ? 2 : 1; o > 0; o >>= 1)
      v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[warp] = v;
  }
}
__device__ __forceinline__ double sum_combine(const double *red, int nact) {
  double a = red[0];
  if (nact > 1) a += red[1];
  if (nact > 2) {
    double b = red[2];
    if (nact > 3) b += red[3];
    a += b;
  }
  if (nact > 4) {
    double c = red[4];
    if (nact > 5) c += red[5];
    if (nact > 6) {
      double d = red[6];
      if (nact > 7) d += red[7];
      c += d;
    }
    a += c;
  }
  return a;
}
__device__ __forceinline__ int warps_for(int64_t n) { return (int)min((int64_t)kEigWarps, (n + 31) / 32); }
// integer forms of FP64 tests (no NaN): they do not use the FP64 pipe
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & ~(1ull << 63);
}
__device__ __forceinline__ bool negative(double x) { return __double_as_longlong(x) < 0 && abs_bits(x) != 0; }

__device__ double block_max(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = red[0];
  for (int w = 1; w < kEigWarps; ++w) t = fmax(t, red[w]);
  return t;
}

// number of eigenvalues of the FP32 tridiagonal (d, e2 = e^2) below x
__device__ int sturm_count(const float *d, const float *e2, int64_t m, float x, float pivmin) {
  float q = d[0] - x;
  if (fabsf(q) < pivmin) q = -pivmin;
  int c = q < 0.f;
  for (int64_t i = 1; i < m; ++i) {
    q = d[i] - x - __fdividef(e2[i - 1], q);
    if (fabsf(q) < pivmin) q = -pivmin;
    c += q < 0.f;
  }
  return c;
}

// LU with partial pivoting of the tridiagonal (d - sigma, e): rows i and i+1 swap when the
// subdiagonal entry is larger than the pivot; U has two superdiagonals.  r0 holds 1/U_ii.  Both
// cases share one division and one update (lanes of a warp take different cases).  ds: the
// shifted diagonal d - sigma; may be r0 itself (an entry is read before it is written).
template <bool FAST>
__device__ void tri_lu(const double *ds, const double *e, int m, double tiny,
                       double *r0, double *__restrict__ u1, double *__restrict__ u2, double *__restrict__ l,
                       double *__restrict__ pv) {
  double da = ds[0], db = m > 1 ? e[0] : 0.0;
  const unsigned long long tb = abs_bits(tiny);
  double c = db, an = m > 1 ? ds[1] : 0.0;  // row i + 1's entries are loaded a row ahead
  for (int i = 0; i + 1 < m; ++i) {
    const double bn = (i + 2 < m) ? e[i + 1] : 0.0, an1 = (i + 2 < m) ? ds[i + 2] : 0.0;
    const bool keep = abs_bits(da) >= abs_bits(c);
    if (keep && abs_bits(da) < tb) da = negative(da) ? -tiny : tiny;
    const double r = FAST ? rcp64(keep ? da : c) : 1.0 / (keep ? da : c);  // one division per row
    const double li = (keep ? c : da) * r;
    r0[i] = r; l[i] = li;
    u1[i] = keep ? db : an;
    u2[i] = keep ? 0.0 : bn;
    pv[i] = keep ? 0.0 : 1.0;
    const double x = keep ? an : db, y = keep ? db : an;
    da = x - li * y;
    db = keep ? bn : -li * bn;
    c = bn;
    an = an1;
  }
  if (abs_bits(da) < tb) da = negative(da) ? -tiny : tiny;
  r0[m - 1] = 1.0 / da;
}

// z <- (T - sigma)^-1 z with the factors of tri_lu
__device__ void tri_solve(int m, const double *r0, const double *u1,
                          const double *u2, const double *l,
                          const double *pv, double *__restrict__ z) {
  double a = z[0];
#pragma unroll 4
  for (int i = 0; i + 1 < m; ++i) {
    const double b = z[i + 1];
    const bool sw = abs_bits(pv[i]) != 0;
    const double x = sw ? b : a, y = sw ? a : b;
    z[i] = x;
    a = y - l[i] * x;
  }
  z[m - 1] = a;
  double z1 = a * r0[m - 1], z2 = 0.0;  // rows m - 1 and m - 2 have fewer superdiagonals
  z[m - 1] = z1;
  if (m > 1) {
    double s = z[m - 2];
    s -= u1[m - 2] * z1;
    z2 = z1;
    z1 = s * r0[m - 2];
    z[m - 2] = z1;
  }
#pragma unroll 4
  for (int i = m - 3; i >= 0; --i) {
    double s = z[i];
    s -= u1[i] * z1;
    s -= u2[i] * z2;
    s *= r0[i];
    z[i] = s;
    z2 = z1;
    z1 = s;
  }
}

__device__ double vdot(const double *z, int64_t m) {
  double s = 0.0;
#pragma unroll 4
  for (int i = 0; i < m; ++i) s = fma(z[i], z[i], s);
  return s;
}
__device__ double vnorm(const double *z, int64_t m) { return sqrt(vdot(z, m)); }
__device__ void vscale(double *z, int64_t m, double f) {
  for (int64_t i = 0; i < m; ++i) z[i] *= f;
}
// a fixed, well-spread positive start vector (an integer hash of (i, j) mapped to [0.5, 1.5))
__device__ double start_value(int64_t i, int64_t j) {
  uint32_t h = (uint32_t)i * 2654435761u ^ ((uint32_t)j * 40503u + 12345u);
  h ^= h >> 15;
  h *= 2246822519u;
  h ^= h >> 13;
  return 0.5 + (double)(h >> 8) * (1.0 / 16777216.0);
}
__device__ void start_vector(double *z, int64_t m, int64_t j) {
  for (int64_t i = 0; i < m; ++i) z[i] = start_value(i, j);
}

// z_c *= f[c - cb] for the vectors of the single clusters c = cb .. of a batch, over the block
__device__ void scale_singles(double *Z, int64_t ldz, int64_t m, const int *cl, int64_t cb, int64_t ncl,
                              const double *f) {
  const int64_t n = min((int64_t)kEigThreads, ncl - cb);
  for (int64_t t = threadIdx.x; t < m * n; t += kEigThreads) {
    const QuotRem x = quot_rem(t, m);
    const int64_t c = cb + x.q;
    if (cl[c + 1] - cl[c] == 1) Z[x.r + ldz * cl[c]] *= f[c - cb];
  }
}
// d - sigma into the first m of each one's 5 m scratch doubles
__device__ void shift_singles(const double *d, int64_t m, const int *cl, int64_t cb, int64_t ncl,
                              const double *sigma, double *scratch) {
  const int64_t n = min((int64_t)kEigThreads, ncl - cb);
  for (int64_t t = threadIdx.x; t < m * n; t += kEigThreads) {
    const QuotRem x = quot_rem(t, m);
    const int64_t c = cb + x.q, i = x.r;
    if (cl[c + 1] - cl[c] == 1) scratch[5 * m * cl[c] + i] = d[i] - sigma[c - cb];
  }
}
// y = T z of the same vectors into the last m of each one's 5 m scratch doubles
__device__ void tri_apply_singles(const double *d, const double *e, const double *Z, int64_t ldz, int64_t m,
                                  const int *cl, int64_t cb, int64_t ncl, double *scratch) {
  const int64_t n = min((int64_t)kEigThreads, ncl - cb);
  for (int64_t t = threadIdx.x; t < m * n; t += kEigThreads) {
    const QuotRem x = quot_rem(t, m);
    const int64_t c = cb + x.q, i = x.r;
    if (cl[c + 1] - cl[c] != 1) continue;
    const double *z = Z + ldz * cl[c];
    double y = d[i] * z[i];
    if (i > 0) y = fma(e[i - 1], z[i - 1], y);
    if (i + 1 < m) y = fma(e[i], z[i + 1], y);
    scratch[5 * m * cl[c] + 4 * m + i] = y;
  }
}

__global__ void __launch_bounds__(kEigThreads, 2) sym_eig_kernel(const __grid_constant__ SymEigGroup g) {
  pdl_wait();
  const SymEigJob q = g.j[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t m = q.m, nw = q.nw;
  if (m < 1 || nw < 1 || nw > m || m > kSymEigMaxM) {
    if (tid == 0 && q.info) *q.info = 1;
    return;
  }
  extern __shared__ double sm[];
  const int64_t ld = eig_ld(m);
  const int64_t nvec = eig_vec_doubles(m);
  double *d = sm, *e = d + m, *tau = e + m, *vv = tau + m, *pp = vv + m, *red = pp + m;
  float *d32 = reinterpret_cast<float *>(red + 32), *e2 = d32 + m, *lam32 = e2 + m;
  int *cl = reinterpret_cast<int *>(lam32 + m);
  // Shared memory behind the vectors, in this order while it lasts: the lower triangle A, the
  // eigenvectors of the tridiagonal (m per wanted eigenvalue), the LU factors of their inverse
  // iterations (5 m per wanted eigenvalue); the rest in global scratch.  The inverse iteration
  // and the back-transformation are serial chains over m, and each step through global memory
  // waits for an L2 round trip (the vectors are copied to U at the end).
  int64_t off = nvec;
  const bool a_sm = off + ld * m <= g.smem_doubles;
  double *A = a_sm ? sm + off : q.work;
  if (a_sm) off += ld * m;
  double *part4 = off + 4 * m <= g.smem_doubles ? sm + off : q.work + ld * m;  // step 1 only, before Z
  const bool z_sm = off + m * nw <= g.smem_doubles;
  double *Z = z_sm ? sm + off : q.U;
  const int64_t ldz = z_sm ? m : q.ldu;
  if (z_sm) off += m * nw;
  const bool lu_sm = z_sm && off + 5 * m * nw <= g.smem_doubles;
  double *scratch = lu_sm ? sm + off : q.work + ld * m;  // 5 m per wanted eigenvalue

  if (tid == 0 && q.clocks) q.clocks[0] = clock64();
  // ---- load the lower triangle ----
  for (int64_t t = tid; t < m * m; t += kEigThreads) {
    const QuotRem x = quot_rem(t, m);
    const int64_t j = x.q, i = x.r;
    if (i >= j) A[i + ld * j] = q.T[i + q.ldt * j];
  }
  __syncthreads();

  // ---- 1. Householder tridiagonalisation ----
  // fast (FP64 solves): square roots and divisions by rsqrt64 and rcp64, 781 to 753 us for the three
  // problems of a ten-root solve; split-precision solves keep the divisions and their bits.
  // Scalars are computed by warp 0 alone and broadcast; the two divisions of a reflector share an
  // instruction; the four interleaved chains of a row of A v run in four threads.
  __shared__ double sc[4], scl[kEigThreads];
  for (int64_t k = 0; k + 2 < m; ++k) {
    const int64_t k1 = k + 1;
    const int na = warps_for(m - k - 2), nr = warps_for(m - k1);
    double s = 0.0;
    for (int64_t i = k + 2 + tid; i < m; i += kEigThreads) s = fma(A[i + ld * k], A[i + ld * k], s);
    sum_warps(s, red, na, m - k - 2);
    if (na > 1) __syncthreads();
    else __syncwarp();
    if (warp == 0) {
      const double xn2 = sum_combine(red, na), alpha = A[k1 + ld * k];
      if (xn2 == 0.0) {
        if (lane == 0) { tau[k] = 0.0; e[k] = alpha; d[k] = A[k + ld * k]; sc[2] = 0.0; }
      } else {
        // beta = -|(alpha, x)| sign(alpha), tau = (beta - alpha) / beta, 1 / (alpha - beta)
        if (q.fast) {
          const double n2 = alpha * alpha + xn2, rs = rsqrt64(n2);
          const double beta = -with_sign(n2 * rs, alpha), diff = alpha - beta;
          const double t = diff * with_sign(rs, alpha), r = rcp64(diff);
          if (lane == 0) { sc[0] = t; sc[1] = r; tau[k] = t; e[k] = beta; d[k] = A[k + ld * k]; sc[2] = 1.0; }
        } else {
          const double beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
          const double diff = lane == 0 ? beta - alpha : alpha - beta;
          const double v = (lane == 0 ? diff : 1.0) / (lane == 0 ? beta : diff);
          if (lane < 2) sc[lane] = v;
          if (lane == 0) { tau[k] = v; e[k] = beta; d[k] = A[k + ld * k]; sc[2] = 1.0; }
        }
      }
    }
    __syncthreads();
    if (sc[2] == 0.0) {
      __syncthreads();
      continue;
    }
    const double tk = sc[0], scal = sc[1];
    for (int64_t i = k1 + tid; i < m; i += kEigThreads) {
      const double vi = (i == k1) ? 1.0 : A[i + ld * k] * scal;
      vv[i] = vi;
      if (i > k1) A[i + ld * k] = vi;
    }
    __syncthreads();
    // p = tau A22 v from the lower triangle, as four interleaved partial sums per row
    {
      const int u = tid >> 6;  // columns k1 + u, k1 + u + 4, ..
      for (int64_t i = k1 + (tid & 63); i < m; i += 64) {
        double acc = 0.0;
#pragma unroll 4
        for (int jj = (int)k1 + u; jj < (int)m; jj += 4) {
          const double a = A[jj <= i ? (int)i + (int)ld * jj : jj + (int)ld * (int)i];
          acc = fma(a, vv[jj], acc);
        }
        part4[u * m + i] = acc;
      }
    }
    __syncthreads();
    double pv_part = 0.0;
    for (int64_t i = k1 + tid; i < m; i += kEigThreads) {
      const double p = tk * ((part4[i] + part4[m + i]) + (part4[2 * m + i] + part4[3 * m + i]));
      pp[i] = p;
      pv_part = fma(p, vv[i], pv_part);
    }
    sum_warps(pv_part, red, nr, m - k1);
    if (nr > 1) __syncthreads();
    else __syncwarp();
    if (warp == 0) {
      const double K = -0.5 * tk * sum_combine(red, nr);
      if (lane == 0) sc[3] = K;
    }
    __syncthreads();
    const double K = sc[3];
    for (int64_t i = k1 + tid; i < m; i += kEigThreads) pp[i] = fma(K, vv[i], pp[i]);  // w
    __syncthreads();
    // A22 -= v w^T + w v^T, lower triangle: columns a and n - 1 - a make one run of n + 1
    // elements, so the warps' lanes are full
    {
      const int n = (int)(m - k1);
      const int total = (n + 1) / 2 * (n + 1);
      for (int t = tid; t < total; t += kEigThreads) {
        const int a = t / (n + 1), b = t % (n + 1);
        int j = a, i = a + b;
        if (b >= n - a) {
          j = n - 1 - a;
          i = j + b - (n - a);
          if (j == a) continue;  // the middle column is its own pair
        }
        const int64_t gi = k1 + i, gj = k1 + j;
        A[gi + ld * gj] -= fma(vv[gi], pp[gj], pp[gi] * vv[gj]);
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    if (m >= 2) {
      d[m - 2] = A[(m - 2) + ld * (m - 2)];
      d[m - 1] = A[(m - 1) + ld * (m - 1)];
      e[m - 2] = A[(m - 1) + ld * (m - 2)];
      tau[m - 2] = 0.0;
    } else {
      d[0] = A[0];
    }
    tau[m - 1] = 0.0;
  }
  __syncthreads();
  if (tid == 0 && q.clocks) q.clocks[1] = clock64();

  // ---- 2. wanted eigenvalues of the tridiagonal: FP32 bisection ----
  double lo = INFINITY, hi = -INFINITY, e2max = 0.0;
  for (int64_t i = tid; i < m; i += kEigThreads) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < m ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
    d32[i] = (float)d[i];
    if (i + 1 < m) {
      e2[i] = (float)(e[i] * e[i]);
      e2max = fmax(e2max, e[i] * e[i]);
    }
  }
  lo = -block_max(-lo, red);
  hi = block_max(hi, red);
  e2max = block_max(e2max, red);
  const double nrm = fmax(fmax(fabs(lo), fabs(hi)), 1e-300);
  const float pivmin = (float)(1e-30 * fmax(1.0, e2max));
  // Every eigenvalue's bisection runs on a group of 7, 3 or 1 threads: the counts at the mid
  // points that its next 3, 2 or 1 steps can reach are taken at once, then the steps are walked
  // (the same intervals as one step at a time).
  {
    const int lv = 7 * nw <= kEigThreads ? 3 : 3 * nw <= kEigThreads ? 2 : 1;
    const int G = (1 << lv) - 1;
    const int nslot = kEigThreads / G;
    int *cnt = reinterpret_cast<int *>(scl);  // one per thread
    for (int64_t j0 = 0; j0 < nw; j0 += nslot) {
      const int slot = tid / G, node = tid % G + 1;  // heap order: children of x are 2x, 2x + 1
      const int64_t j = j0 + slot;
      const bool act = slot < nslot && j < nw;
      float a = (float)(lo - 1e-6 * nrm) - 1e-30f, b = (float)(hi + 1e-6 * nrm) + 1e-30f;
      int it = 0;
      bool done = !act;
      while (__syncthreads_or(!done)) {
        if (!done) {
          float na = a, nb = b, mid = 0.5f * (a + b);
          int depth = 31 - __clz(node);
          for (int x = depth - 1; x >= 0; --x) {
            if ((node >> x) & 1) na = mid; else nb = mid;
            mid = 0.5f * (na + nb);
          }
          cnt[tid] = sturm_count(d32, e2, m, mid, pivmin);
        }
        __syncthreads();
        if (!done) {
          int x = 1;
          for (int st = 0; st < lv; ++st) {
            if (it >= 80 || b - a <= 2.4e-7f * fmaxf(fabsf(a), fabsf(b)) + 4.f * pivmin) { done = true; break; }
            const float mid = 0.5f * (a + b);
            if (cnt[slot * G + x - 1] > (int)j) { b = mid; x = 2 * x; } else { a = mid; x = 2 * x + 1; }
            ++it;
          }
        }
      }
      if (act && node == 1) lam32[j] = 0.5f * (a + b);
    }
  }
  __syncthreads();
  // clusters of eigenvalues closer than 1e-5 of the spectral radius (cl: starts, then nw): the
  // FP32 shifts are good to a few 1e-7 of it, so eigenvalues further apart converge separately
  __shared__ int ncl;
  if (tid == 0 && q.clocks) q.clocks[2] = clock64();
  if (tid == 0) {
    int c = 0;
    cl[c++] = 0;
    for (int64_t j = 1; j < nw; ++j)
      if ((double)lam32[j] - (double)lam32[j - 1] > 1e-5 * nrm) cl[c++] = (int)j;
    cl[c] = (int)nw;
    ncl = c;
  }
  __syncthreads();

  // ---- 3. eigenvectors of the tridiagonal by inverse iteration (FP64) ----
  // One thread per cluster runs the serial chains; the elementwise work of the single
  // eigenvalues (start vectors, scalings, T z) is spread over the block between barriers.
  const double tiny = 2.3e-16 * nrm;
  {
    for (int64_t cb = 0; cb < ncl; cb += kEigThreads) {
      const int64_t c = cb + tid;
      const bool single = c < ncl && cl[c + 1] - cl[c] == 1;
      const int64_t j = single ? cl[c] : 0;
      double *w = scratch + 5 * m * j, *z = Z + ldz * j;
      double *r0 = w, *u1 = w + m, *u2 = w + 2 * m, *l = w + 3 * m, *pv = w + 4 * m;
      const int64_t jb0 = cl[cb], jb1 = cl[min((int64_t)ncl, cb + kEigThreads)];  // vectors of this batch
      const int64_t nel = m * (jb1 - jb0);
      for (int64_t t = tid; t < nel; t += kEigThreads) {
        const QuotRem x = quot_rem(t, m);
        Z[x.r + ldz * (jb0 + x.q)] = start_value(x.r, jb0 + x.q);
      }
      __syncthreads();
      double sigma = single ? (double)lam32[j] : 0.0;
      for (int half = 0; half < 2; ++half) {
        scl[tid] = sigma;
        __syncthreads();
        shift_singles(d, m, cl, cb, ncl, scl, scratch);
        __syncthreads();
        if (single) {
          if (q.fast) tri_lu<true>(r0, e, (int)m, tiny, r0, u1, u2, l, pv);
          else tri_lu<false>(r0, e, (int)m, tiny, r0, u1, u2, l, pv);
        }
        for (int st = 0; st < 2; ++st) {
          if (single) {
            tri_solve((int)m, r0, u1, u2, l, pv, z);
            const double zz = vdot(z, m);
            scl[tid] = q.fast ? rsqrt64(zz) : 1.0 / sqrt(zz);
          } else {
            scl[tid] = 1.0;
          }
          __syncthreads();
          scale_singles(Z, ldz, m, cl, cb, ncl, scl);
          __syncthreads();
        }
        // T z beside the factors (pv is free), then the Rayleigh quotient
        tri_apply_singles(d, e, Z, ldz, m, cl, cb, ncl, scratch);
        __syncthreads();
        if (single) {
          double s = 0.0;
#pragma unroll 4
          for (int i = 0; i < m; ++i) s = fma(z[i], pv[i], s);
          sigma = s;
        }
      }
      if (single) q.lam[j] = sigma;
      __syncthreads();
    }
  }
  for (int c = tid; c < ncl; c += kEigThreads) {
    const int64_t j0 = cl[c], j1 = cl[c + 1], s = j1 - j0;
    if (s == 1) continue;
    double *w = scratch + 5 * m * j0;  // 5 m per member, contiguous over the cluster
    double *r0 = w, *u1 = w + m, *u2 = w + 2 * m, *l = w + 3 * m, *pv = w + 4 * m;
    for (int64_t jj = j0; jj < j1; ++jj) {
      double *z = Z + ldz * jj;
      start_vector(z, m, jj);
      for (int64_t i = 0; i < m; ++i) r0[i] = d[i] - (double)lam32[jj];
      tri_lu<false>(r0, e, (int)m, tiny, r0, u1, u2, l, pv);
      for (int st = 0; st < 5; ++st) {
        tri_solve((int)m, r0, u1, u2, l, pv, z);
        for (int64_t kk = j0; kk < jj; ++kk) {  // earlier members of the cluster
          const double *y = Z + ldz * kk;
          double dot = 0.0;
          for (int64_t i = 0; i < m; ++i) dot = fma(y[i], z[i], dot);
          for (int64_t i = 0; i < m; ++i) z[i] = fma(-dot, y[i], z[i]);
        }
        vscale(z, m, 1.0 / vnorm(z, m));
      }
    }
    {  // Rayleigh-Ritz on the cluster: cyclic Jacobi on C = Z_c^T T Z_c
      double *C = w, *W = w + s * s, *y = w + 2 * s * s;
      for (int64_t b = 0; b < s; ++b) {
        const double *zb = Z + ldz * (j0 + b);
        for (int64_t i = 0; i < m; ++i) {
          double t = d[i] * zb[i];
          if (i > 0) t = fma(e[i - 1], zb[i - 1], t);
          if (i + 1 < m) t = fma(e[i], zb[i + 1], t);
          y[i] = t;
        }
        for (int64_t a = 0; a < s; ++a) {
          const double *za = Z + ldz * (j0 + a);
          double t = 0.0;
          for (int64_t i = 0; i < m; ++i) t = fma(za[i], y[i], t);
          C[a + s * b] = t;
        }
      }
      for (int64_t b = 0; b < s; ++b)
        for (int64_t a = 0; a < s; ++a) {
          W[a + s * b] = a == b ? 1.0 : 0.0;
          if (a < b) C[a + s * b] = C[b + s * a] = 0.5 * (C[a + s * b] + C[b + s * a]);
        }
      for (int sweep = 0; sweep < 40; ++sweep) {
        double off = 0.0, dg = 0.0;
        for (int64_t b = 0; b < s; ++b)
          for (int64_t a = 0; a < s; ++a) {
            const double v = C[a + s * b] * C[a + s * b];
            if (a == b) dg += v; else off += v;
          }
        if (off <= 1e-34 * dg || off == 0.0) break;
        for (int64_t p = 0; p < s; ++p)
          for (int64_t r = p + 1; r < s; ++r) {
            const double apq = C[p + s * r];
            if (apq == 0.0) continue;
            const double th = (C[r + s * r] - C[p + s * p]) / (2.0 * apq);
            const double t = fabs(th) > 1e150 ? 0.5 / th : copysign(1.0, th) / (fabs(th) + sqrt(th * th + 1.0));
            const double cs = 1.0 / sqrt(t * t + 1.0), sn = t * cs;
            for (int64_t x = 0; x < s; ++x) {  // C J
              const double cp = C[x + s * p], cq = C[x + s * r];
              C[x + s * p] = cs * cp - sn * cq;
              C[x + s * r] = sn * cp + cs * cq;
            }
            for (int64_t x = 0; x < s; ++x) {  // J^T (C J)
              const double cp = C[p + s * x], cq = C[r + s * x];
              C[p + s * x] = cs * cp - sn * cq;
              C[r + s * x] = sn * cp + cs * cq;
            }
            for (int64_t x = 0; x < s; ++x) {
              const double wp = W[x + s * p], wq = W[x + s * r];
              W[x + s * p] = cs * wp - sn * wq;
              W[x + s * r] = sn * wp + cs * wq;
            }
          }
      }
      // ascending order of the Ritz values: selection sort of the columns of W
      for (int64_t a = 0; a < s; ++a) {
        int64_t best = a;
        for (int64_t b = a + 1; b < s; ++b)
          if (C[b + s * b] < C[best + s * best]) best = b;
        if (best != a) {
          const double t = C[a + s * a];
          C[a + s * a] = C[best + s * best];
          C[best + s * best] = t;
          for (int64_t x = 0; x < s; ++x) {
            const double u = W[x + s * a];
            W[x + s * a] = W[x + s * best];
            W[x + s * best] = u;
          }
        }
        q.lam[j0 + a] = C[a + s * a];
      }
      for (int64_t i = 0; i < m; ++i) {  // Z_c <- Z_c W, row by row
        for (int64_t a = 0; a < s; ++a) {
          double t = 0.0;
          for (int64_t b = 0; b < s; ++b) t = fma(Z[i + ldz * (j0 + b)], W[b + s * a], t);
          y[a] = t;
        }
        for (int64_t a = 0; a < s; ++a) Z[i + ldz * (j0 + a)] = y[a];
      }
    }
  }
  __syncthreads();
  if (tid == 0 && q.clocks) q.clocks[3] = clock64();

  // ---- 4. back-transformation U = H_0 H_1 ... H_{m-3} Z ----
  // Up to one vector per warp: each warp applies the reflectors to its vector (a warp reduction
  // per reflector).  More vectors: every reflector is applied to a batch of vectors at once, G
  // threads per vector (all threads busy), each summing every G-th row of the dot product; the
  // G partial sums of a vector are added in a fixed order by each of its threads (no FP64
  // shuffle tree: on GB300's narrow FP64 pipe the five butterfly levels of a warp reduction,
  // repeated for every vector of every warp, cost more than the dot products themselves).
  if (nw <= kEigWarps) {
    for (int64_t j = warp; j < nw; j += kEigWarps) {
      double *z = Z + ldz * j;
      for (int64_t k = m - 3; k >= 0; --k) {
        const double tk = tau[k];
        if (tk == 0.0) continue;
        double s = 0.0;
        for (int64_t i = k + 1 + lane; i < m; i += 32) s = fma(i == k + 1 ? 1.0 : A[i + ld * k], z[i], s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const double f = tk * s;
        for (int64_t i = k + 1 + lane; i < m; i += 32) z[i] = fma(-f, i == k + 1 ? 1.0 : A[i + ld * k], z[i]);
      }
    }
  } else {
    double *part = scl;
    double *fac = vv;  // one factor per vector of a batch (vv and pp are free)
    const int G = min(32, max(1, kEigThreads / (int)nw));
    const int per_batch = kEigThreads / G;
    const int slot = tid / G, sub = tid % G;
    for (int64_t j0 = 0; j0 < nw; j0 += per_batch) {
      const int64_t j = j0 + slot;
      const bool act = slot < per_batch && j < nw;
      double *z = act ? Z + ldz * j : nullptr;
      for (int64_t k = m - 3; k >= 0; --k) {
        const double tk = tau[k];
        if (tk == 0.0) continue;  // uniform over the block
        double s = 0.0;
        if (act)
          for (int64_t i = k + 1 + sub; i < m; i += G) s = fma(i == k + 1 ? 1.0 : A[i + ld * k], z[i], s);
        part[tid] = s;
        __syncthreads();
        if (tid < min((int64_t)per_batch, nw - j0)) {  // the partial sums of a vector by one thread: few warps add
          double t = 0.0;
          for (int p = 0; p < G; ++p) t += part[tid * G + p];
          fac[tid] = tk * t;
        }
        __syncthreads();
        if (act) {
          const double f = fac[slot];
          for (int64_t i = k + 1 + sub; i < m; i += G) z[i] = fma(-f, i == k + 1 ? 1.0 : A[i + ld * k], z[i]);
        }
        __syncthreads();  // part is written again for the next reflector
      }
    }
  }
  __syncthreads();
  if (z_sm)
    for (int64_t t = tid; t < m * nw; t += kEigThreads) {
      const QuotRem x = quot_rem(t, m);
      q.U[x.r + q.ldu * x.q] = Z[t];
    }
  if (tid == 0 && q.clocks) q.clocks[4] = clock64();
  if (tid == 0 && q.info) *q.info = 0;
}

}  // namespace

int64_t sym_eig_work_doubles(int64_t m, int64_t nw) { return eig_ld(m) * m + 5 * m * nw + 64; }

void sym_eig_device(const SymEigJob *jobs, int64_t njobs, cudaStream_t s) {
  if (njobs <= 0) return;
  int dev = 0;
  VGB_CUDA(cudaGetDevice(&dev));
  int optin = 0;
  VGB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes fa;
  VGB_CUDA(cudaFuncGetAttributes(&fa, sym_eig_kernel));
  const int dyn_max = optin - (int)fa.sharedSizeBytes;  // the static shared memory counts against the limit
  static std::mutex mu;
  static int configured[64] = {0};
  {
    std::lock_guard<std::mutex> lk(mu);
    if (dev < 64 && !configured[dev]) {
      VGB_CUDA(cudaFuncSetAttribute(sym_eig_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn_max));
      configured[dev] = 1;
    }
  }
  const int64_t limit = dyn_max / (int64_t)sizeof(double);
  std::unique_ptr<SymEigGroup> g(new SymEigGroup());
  for (int64_t b = 0; b < njobs; b += kEigJobs) {
    g->n = (int)std::min<int64_t>(kEigJobs, njobs - b);
    int64_t need = 0;
    for (int i = 0; i < g->n; ++i) {
      const SymEigJob &jb = jobs[b + i];
      VGB_REQUIRE(jb.m >= 1 && jb.m <= kSymEigMaxM && jb.nw >= 1 && jb.nw <= jb.m && jb.ldu >= jb.m &&
                      jb.ldt >= jb.m && jb.work != nullptr,
                  "small symmetric eigenproblem: invalid job");
      g->j[i] = jb;
      // the vectors, then A, the inverse-iteration vectors and their LU factors while they fit
      // (the kernel places them in the same order)
      int64_t job_need = eig_vec_doubles(jb.m);
      if (job_need + eig_ld(jb.m) * jb.m <= limit) job_need += eig_ld(jb.m) * jb.m;
      const int64_t with_part = job_need + 4 * jb.m;  // step 1's partial sums, before the vectors
      if (job_need + jb.m * jb.nw <= limit) {
        job_need += jb.m * jb.nw;
        if (job_need + 5 * jb.m * jb.nw <= limit) job_need += 5 * jb.m * jb.nw;
      }
      if (with_part <= limit) job_need = std::max(job_need, with_part);
      need = std::max(need, job_need);
    }
    g->smem_doubles = need;
    launch_pdl(sym_eig_kernel, g->n, kEigThreads, need * sizeof(double), s, *g);
    VGB_LAUNCH_CHECK();
  }
}

}  // namespace vgb
