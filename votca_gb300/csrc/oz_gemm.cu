// FP64 GEMM from exact bf16 digit products (see oz_gemm.cuh for the scheme and its accuracy).
#include "oz_gemm.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

#include "oz_plan.hpp"
#include "tc_ptx.cuh"

namespace vgb {

namespace {

constexpr int S = kOzDigits;
constexpr int LV = 8;         // levels a + b = 0 .. 7 kept (34 pairs)
constexpr int BM = kOzTileM;  // tile rows (A), one TMEM lane each
constexpr int BN = kOzTileN;  // tile columns (B): LV * BN = 512 TMEM columns
constexpr int BK = kOzStageK;  // K elements per pipeline stage (64-byte swizzle rows)
constexpr int RUN = kOzRun;    // K elements sharing one digit scale
constexpr int HB = kOzDrain;   // stages between drains of levels 0 .. 3: 4 pairs x 256 products of
                              // at most 2^14 sum exactly in FP32 (2^24)
constexpr int LB = 4;         // stages between drains of levels 4 .. 7: 7 pairs x 128 products
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
constexpr int STAGE_BYTES = S * (A_BYTES + B_BYTES);  // 86016
constexpr int STAGES = 2;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int kEpi = 16;                     // epilogue warps: four per TMEM lane quarter
constexpr int EC = BN / 4;                   // columns of an epilogue thread
constexpr int kGemmThreads = 64 + 32 * kEpi; // warp 0: TMA, warp 1: MMA, rest: epilogue
constexpr int BITS = 8 * S - 1;              // digit window: |x| < 2^e -> |m| <= 2^BITS
constexpr int BIAS = 50;                     // operand digits carry 2^(BIAS - row exponent)
constexpr int ZERO_RUN = -100000;            // exponent of a run of zeros
constexpr int E_MAX = 900;                   // larger or smaller exponents take the FMA path
static_assert(LV * BN <= 512 && SMEM_BYTES <= 232448, "tile exceeds the SM");

// One operand: rows [r0, r0 + rows) of the map, K columns ks apart, and its planes.
struct Operand {
  const double *p = nullptr;
  OzMap map;
  int64_t r0 = 0, rows = 0, K = 0, Kp = 0, ks = 1;
  uint16_t *planes = nullptr;  // [t][rows][Kp]
  int *erow = nullptr;         // exponent of the row's largest element (per row)
  int *erun = nullptr;         // per (row, run), only when there is more than one run
  int nruns = 1;
};

// ---------------- digits ----------------

// Digits of four consecutive K elements, packed per plane.  x = sum_t d_t 2^(e - 7 - 8 t), the
// value m = round(x 2^(BITS - e)) in 64-bit integers (the FP64 pipe is the slow one here) and its
// balanced bytes: adding 128 to every byte but the top one makes each byte d + 128.  The bf16
// value d 2^(rel + BIAS - 7 - 8 t) comes from one FFMA on 2^23 + byte.
__device__ __forceinline__ void digits4(const double (&x)[4], int e, const float (&sc)[S], uint2 (&out)[S]) {
  uint32_t lo[4], hi[4];
  int top[4];
  constexpr long long bias = 0x0000808080808080ll;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x[v]);
    const int ef = (int)((b >> 52) & 0x7FF);
    const int sh = e - (ef - 1022);  // 0 .. : |x| < 2^(ef - 1022) <= 2^e
    unsigned long long m = ((b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << (BITS - 53);
    m = (ef == 0 || sh > BITS + 1) ? 0ull : (sh > 0 ? (m + (1ull << (sh - 1))) >> sh : m);
    const long long u = ((b >> 63) ? -(long long)m : (long long)m) + bias;
    lo[v] = (uint32_t)u;
    hi[v] = (uint32_t)((unsigned long long)u >> 32);
    top[v] = (int)(u >> 48);  // -128 .. 128
  }
#pragma unroll
  for (int t = 0; t < S; ++t) {
    float f[4];
    const float c = -8388736.0f * sc[t];  // -(2^23 + 128) scale
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      uint32_t w;
      if (t == 0) w = 0x4B000000u + (uint32_t)(top[v] + 128);
      else if (t <= 2) w = __byte_perm(hi[v], 0x4B000000u, t == 1 ? 0x7651 : 0x7650);
      else w = __byte_perm(lo[v], 0x4B000000u, t == 3 ? 0x7653 : t == 4 ? 0x7652 : t == 5 ? 0x7651 : 0x7650);
      f[v] = fmaf(__uint_as_float(w), sc[t], c);
    }
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out[t].x) : "f"(f[1]), "f"(f[0]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out[t].y) : "f"(f[3]), "f"(f[2]));
  }
}

// One block per (32 rows, run).  phase 1: run and row exponents only (more than one run per row);
// phase 2: digits from stored exponents; phase 3: both (a row is one run: its elements are read
// twice, the second time through L2).  Reads are coalesced along K (ks == 1) or along the rows
// (through a shared-memory transpose); the planes are written along K.
// Bound: HBM (8 bytes read, 14 written per element) when large; about 40 integer and FP32
// instructions per element keep the issue slots under that.
constexpr int SROWS = 32, SK = 64, SLD = SK + 2;
__global__ void __launch_bounds__(256) oz_slice_kernel(const __grid_constant__ Operand oa,
                                                       const __grid_constant__ Operand ob, int64_t units_a,
                                                       int64_t units, int phase, int *flag) {
  __shared__ __align__(16) double tile[SROWS][SLD];
  __shared__ unsigned long long red[8][SROWS];
  __shared__ int s_e[SROWS], s_rel[SROWS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int64_t u0 = blockIdx.x; u0 < units; u0 += gridDim.x) {
    const bool is_a = u0 < units_a;
    const Operand &o = is_a ? oa : ob;
    const int64_t u = is_a ? u0 : u0 - units_a;
    const int64_t rb = u / o.nruns * SROWS, run = u % o.nruns;
    const int64_t k0 = run * RUN, k1 = min(o.K, k0 + RUN), kp1 = min(o.Kp, k0 + RUN);
    const bool kc = o.ks == 1;
    const int nrow = (int)min((int64_t)SROWS, o.rows - rb);
    __syncthreads();  // the previous unit's shared values are read
    if (phase & 1) {
      if (kc) {
        for (int q = 0; q < 4; ++q) {
          const int row = warp * 4 + q;
          unsigned long long mx = 0;
          if (row < nrow) {
            const double *src = o.p + o.map.at(o.r0 + rb + row);
#pragma unroll 4
            for (int64_t k = k0 + lane; k < k1; k += 32) {
              const unsigned long long a = (unsigned long long)__double_as_longlong(__ldg(src + k)) & ~(1ull << 63);
              mx = a > mx ? a : mx;
            }
          }
#pragma unroll
          for (int w = 16; w; w >>= 1) {
            const unsigned long long y = __shfl_xor_sync(0xffffffffu, mx, w);
            mx = y > mx ? y : mx;
          }
          if (lane == 0) red[0][row] = mx;
        }
        __syncthreads();
      } else {
        unsigned long long mx = 0;
        if (lane < nrow) {
          const double *src = o.p + o.map.at(o.r0 + rb + lane);
#pragma unroll 4
          for (int64_t k = k0 + warp; k < k1; k += 8) {
            const unsigned long long a =
                (unsigned long long)__double_as_longlong(__ldg(src + k * o.ks)) & ~(1ull << 63);
            mx = a > mx ? a : mx;
          }
        }
        red[warp][lane] = mx;
        __syncthreads();
        if (warp == 0) {
#pragma unroll
          for (int w = 1; w < 8; ++w) mx = red[w][lane] > mx ? red[w][lane] : mx;
          red[0][lane] = mx;
        }
        __syncthreads();
      }
      if (tid < SROWS) {
        const unsigned long long mx = red[0][tid];
        const int e = mx == 0 ? ZERO_RUN : (int)(mx >> 52) - 1022;  // mx < 2^e
        // infinities, NaNs and the ends of the exponent range: the whole product by FMA
        if (mx != 0 && (e > E_MAX || e < -E_MAX)) atomicMax(flag, 1);
        s_e[tid] = e;
        s_rel[tid] = 0;
        if (tid < nrow) {
          if (phase == 1) {
            o.erun[(rb + tid) * o.nruns + run] = e;
            atomicMax(o.erow + rb + tid, e);
          } else {
            o.erow[rb + tid] = e;
          }
        }
      }
      if (phase == 1) continue;
    } else {
      if (tid < nrow) {
        const int e = o.erun[(rb + tid) * o.nruns + run];
        s_e[tid] = e;
        s_rel[tid] = e - o.erow[rb + tid];
      }
    }
    __syncthreads();
    // digits: a thread takes four consecutive K elements of two rows of every 64-wide strip
    float sc[2][S];
    int ee[2];
    const double *src[2];
    const int kq = (tid & 15) * 4;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = (tid >> 4) + 16 * i;
      ee[i] = row < nrow ? s_e[row] : ZERO_RUN;
      const int rel = row < nrow && ee[i] != ZERO_RUN ? s_rel[row] : 0;
      src[i] = o.p + (row < nrow ? o.map.at(o.r0 + rb + row) : 0);
#pragma unroll
      for (int t = 0; t < S; ++t) {  // 2^(rel + BIAS - 7 - 8 t); below the FP32 range: 0
        const int pe = 127 + rel + BIAS - 7 - 8 * t;
        sc[i][t] = pe >= 1 ? __int_as_float(pe << 23) : 0.f;
      }
    }
    for (int64_t kt = k0; kt < kp1; kt += SK) {
      if (!kc) {
        __syncthreads();
        const double *sr = o.p + (lane < nrow ? o.map.at(o.r0 + rb + lane) : 0);
#pragma unroll
        for (int j = 0; j < SK / 8; ++j) {
          const int64_t k = kt + warp + 8 * j;
          tile[lane][warp + 8 * j] = (lane < nrow && k < k1) ? __ldg(sr + k * o.ks) : 0.0;
        }
        __syncthreads();
      }
      if (kt + kq >= kp1) continue;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int row = (tid >> 4) + 16 * i;
        if (row >= nrow) continue;
        double x[4];
        const int64_t k = kt + kq;
        if (kc) {
          const double *q = src[i] + k;
          if (k + 4 <= k1 && ((uintptr_t)q & 15) == 0) {
            const double2 a = __ldg(reinterpret_cast<const double2 *>(q));
            const double2 b = __ldg(reinterpret_cast<const double2 *>(q) + 1);
            x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
          } else {
#pragma unroll
            for (int v = 0; v < 4; ++v) x[v] = k + v < k1 ? __ldg(q + v) : 0.0;
          }
        } else {
          const double2 a = *reinterpret_cast<const double2 *>(&tile[row][kq]);
          const double2 b = *reinterpret_cast<const double2 *>(&tile[row][kq + 2]);
          x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        }
        uint2 d[S];
        digits4(x, ee[i], sc[i], d);
        uint16_t *out = o.planes + (rb + row) * o.Kp + k;
        const int64_t plane = o.rows * o.Kp;
#pragma unroll
        for (int t = 0; t < S; ++t) *reinterpret_cast<uint2 *>(out + t * plane) = d[t];
      }
    }
  }
}

// ---------------- product ----------------

struct GemmArgs {
  CUtensorMap map_a, map_b;
  int64_t M, N;              // per batch; operand rows of batch t start at t * M (A), t * N (B)
  int64_t K;
  int a_plane, b_plane;      // operand rows between planes
  int nkb, kb_per, splits;   // K stages, stages per split (a multiple of HB)
  int64_t m_first, b_first;  // first C row and batch of this launch (chunks)
  int64_t mt, nt, ntiles;
  const int *erow_a, *erow_b, *flag;
  Operand A, B;              // sources, for the FMA path
  OzMap crow, ccol, cbatch;  // C offsets of tile rows, columns and batches
  int64_t c_split;           // C offset between K splits (partials)
  double *C;
  double alpha, beta;
  int alpha_exp, alpha_pow2; // alpha = +-2^alpha_exp
  int *err;
};

struct Tile {
  int64_t m, n, b;
  int s;
};
// M tiles in panels of 16, so that the tiles in flight share their A and B planes in L2
__device__ __forceinline__ Tile tile_of(const GemmArgs &p, int64_t t) {
  Tile c;
  const int64_t per = p.mt * p.nt * p.splits;
  c.b = t / per;
  t -= c.b * per;
  const int64_t pw = 16 * p.nt * p.splits, pan = t / pw;
  t -= pan * pw;
  const int64_t g = min((int64_t)16, p.mt - pan * 16);
  c.m = pan * 16 + t % g;
  t /= g;
  c.n = t % p.nt;
  c.s = (int)(t / p.nt);
  return c;
}

__device__ __forceinline__ void two_sum(float &h, float &l, float x) {
  const float s = h + x, bb = s - h;
  l += (h - (s - bb)) + (x - bb);
  h = s;
}

__device__ __forceinline__ void add_level(float (&h)[EC], float (&l)[EC], const uint32_t (&r)[EC]) {
#pragma unroll
  for (int j = 0; j < EC; ++j) two_sum(h[j], l[j], __uint_as_float(r[j]));
}
__device__ __forceinline__ void add_low(float (&l)[EC], const uint32_t (&r)[EC]) {
#pragma unroll
  for (int j = 0; j < EC; ++j) l[j] += __uint_as_float(r[j]);
}

__device__ __forceinline__ long long mant24(float f) {
  const uint32_t b = __float_as_uint(f);
  const int m = (b & 0x7F800000u) ? (int)((b & 0x7FFFFFu) | 0x800000u) : 0;
  return (b >> 31) ? -m : m;
}

// (h1 + l1 + h2 + l2) 2^e rounded to FP64, in integers (an FP64 instruction costs 16 clocks of a
// warp here): the sum as three non-overlapping floats, a 61-bit fixed point, a rounded mantissa.
__device__ __forceinline__ double assemble(float h1, float l1, float h2, float l2, int e, bool neg) {
  float z = 0.f, c = l1, x = h1, y = 0.f, w = 0.f;
  two_sum(c, z, h2);
  z += l2;
  two_sum(x, y, c);   // x + y = h1 + c
  two_sum(y, w, z);   // y + w = y + z
  float t = 0.f;
  two_sum(x, t, y);   // renormalise: x leads, t + w trail
  float t2 = 0.f;
  two_sum(t, t2, w);
  const uint32_t bx = __float_as_uint(x);
  const int ex = (int)((bx >> 23) & 0xFF);
  if (ex == 0) return neg ? -0.0 : 0.0;
  long long T = mant24(x) << 36;  // unit 2^(ex - 186)
  const int s1 = 36 - (ex - (int)((__float_as_uint(t) >> 23) & 0xFF));
  const long long m1 = mant24(t);
  T += s1 >= 0 ? m1 << s1 : (s1 > -32 ? m1 >> -s1 : 0);
  const int s2 = 36 - (ex - (int)((__float_as_uint(t2) >> 23) & 0xFF));
  const long long m2 = mant24(t2);
  T += s2 >= 0 ? m2 << s2 : (s2 > -32 ? m2 >> -s2 : 0);
  unsigned long long u = (unsigned long long)(T < 0 ? -T : T);
  const int lz = __clzll((long long)u);
  u <<= lz;
  const unsigned long long v = u + 0x3FFull + ((u >> 11) & 1ull);  // round to nearest even
  const int be = ex - 123 - lz + e + 1023 + (v < u ? 1 : 0);
  const bool sg = (T < 0) != neg;
  if (be >= 1 && be <= 2046) {
    const unsigned long long bits = ((unsigned long long)sg << 63) | ((unsigned long long)be << 52) |
                                    ((v >> 11) & 0xFFFFFFFFFFFFFull);
    return __longlong_as_double((long long)bits);
  }
  const double r = scalbn((double)(u >> 11), ex - 186 - lz + 11 + e);  // over- or underflow
  return sg ? -r : r;
}

__device__ __forceinline__ void store_c(const GemmArgs &p, double *c, double v) {
  *c = p.beta == 0.0 ? v : fma(p.beta, *c, v);
}

// The tile by FP64 FMA, for operands with infinities, NaNs or exponents at the ends of the range:
// the 64 x 64 register tiles of dgemm.cu on the CTA's first 256 threads.
__device__ __noinline__ void fma_tile(const GemmArgs &p, const Tile &tc, double *smem) {
  constexpr int TK = 16, LD = 65;
  double *As = smem, *Bs = As + TK * LD;
  int64_t *ra = reinterpret_cast<int64_t *>(Bs + TK * LD), *rb = ra + 64;
  const int tid = threadIdx.x, tx = tid & 15, ty = (tid >> 4) & 15;
  const int64_t kbeg = (int64_t)tc.s * p.kb_per * BK;
  const int64_t kend = min(p.K, kbeg + (int64_t)p.kb_per * BK);
  const int64_t cb = p.cbatch.at(p.b_first + tc.b) + tc.s * p.c_split;
  const bool ak = p.A.ks == 1, bk = p.B.ks == 1;
  for (int h = 0; h < 2; ++h) {
    const int64_t m0 = tc.m * BM + 64 * h, n0 = tc.n * BN;
    if (m0 >= p.M) break;
    __syncthreads();
    if (tid < 64) {
      ra[tid] = m0 + tid < p.M ? p.A.map.at(p.A.r0 + tc.b * p.M + m0 + tid) : -1;
      rb[tid] = n0 + tid < p.N ? p.B.map.at(p.B.r0 + tc.b * p.N + n0 + tid) : -1;
    }
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    for (int64_t k0 = kbeg; k0 < kend; k0 += TK) {
      __syncthreads();
      for (int e = tid; e < 64 * TK; e += kGemmThreads) {
        const int ia = ak ? e / TK : e % 64, la = ak ? e % TK : e / 64;
        As[la * LD + ia] = (ra[ia] >= 0 && k0 + la < kend) ? p.A.p[ra[ia] + (k0 + la) * p.A.ks] : 0.0;
        const int ib = bk ? e / TK : e % 64, lb = bk ? e % TK : e / 64;
        Bs[lb * LD + ib] = (rb[ib] >= 0 && k0 + lb < kend) ? p.B.p[rb[ib] + (k0 + lb) * p.B.ks] : 0.0;
      }
      __syncthreads();
      for (int l = 0; l < TK; ++l)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            acc[i][j] = fma(As[l * LD + ty + 16 * i], Bs[l * LD + tx + 16 * j], acc[i][j]);
    }
    if (tid < 256) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t gi = m0 + ty + 16 * i;
        if (gi >= p.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t gn = n0 + tx + 16 * j;
          if (gn >= p.N) continue;
          store_c(p, p.C + cb + p.crow.at(p.m_first + gi) + p.ccol.at(gn), p.alpha * acc[i][j]);
        }
      }
    }
  }
  __syncthreads();
}

// Persistent kernel, one CTA per SM.  A stage holds the seven A planes (128 rows) and the seven B
// planes (64 rows) of 32 K elements: every plane is loaded once for its 34 pair products, 48
// bytes per clock and SM at the full MMA rate (a stage per pair group, as the slice mode of
// tc_gemm.cu, loads 96).  One MMA multiplies A plane a with up to four stacked B planes
// b .. b + 3 into the adjacent accumulators of levels a + b .. a + b + 3: the TMEM column of a
// product is its level, so the pairs of a level add up in the tensor core.  Levels 0..3 (H) are
// issued before levels 4..7 (L) in every stage, and the epilogue drains H while the MMAs of L
// run and L while those of the next stage's H run.
template <int N>
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
                             ((uint32_t)(BM >> 4) << 24);
  mma_bf16(d, a, b, idesc, acc);
}

__global__ void __launch_bounds__(kGemmThreads, 1) oz_gemm_kernel(const __grid_constant__ GemmArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  if (*p.flag > 0) {  // uniform over the grid: set by the slicer, an earlier launch
    for (int64_t R = blockIdx.x; R < p.ntiles; R += gridDim.x)
      fma_tile(p, tile_of(p, R), reinterpret_cast<double *>(smem));
    return;
  }
  uint64_t *full = (uint64_t *)(smem + STAGES * STAGE_BYTES);
  uint64_t *empty = full + STAGES;
  uint64_t *accf = empty + STAGES;  // [0]: H complete, [1]: L complete
  uint64_t *acce = accf + 2;        // drained
  uint32_t *tmem_slot = (uint32_t *)(acce + 2);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&accf[i], 1);
      mbar_init(&acce[i], kEpi);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int64_t R = blockIdx.x; R < p.ntiles; R += gridDim.x) {
        const Tile tc = tile_of(p, R);
        const int ya = (int)(tc.b * p.M + tc.m * BM), yb = (int)(tc.b * p.N + tc.n * BN);
        const int kb0 = tc.s * p.kb_per, kb1 = min(p.nkb, kb0 + p.kb_per);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.err, 11)) goto tma_done;
          const uint32_t st = smem_u32(smem + stage * STAGE_BYTES);
          mbar_expect_tx(&full[stage], (uint32_t)STAGE_BYTES);
          for (int t = 0; t < S; ++t) {
            tma_load_2d(st + t * A_BYTES, &p.map_a, &full[stage], kb * BK, ya + t * p.a_plane);
            tma_load_2d(st + S * A_BYTES + t * B_BYTES, &p.map_b, &full[stage], kb * BK, yb + t * p.b_plane);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      for (int i = 0; i < STAGES; ++i) {  // every stage consumed before the CTA leaves
        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.err, 15)) break;
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    tma_done:;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, eh = 0, el = 0;
      for (int64_t R = blockIdx.x; R < p.ntiles; R += gridDim.x) {
        const Tile tc = tile_of(p, R);
        const int kb0 = tc.s * p.kb_per, n = min(p.nkb, kb0 + p.kb_per) - kb0;
        for (int i = 0; i < n; ++i) {
          if (!mbar_wait(&full[stage], phase, abort_flag, p.err, 13)) goto mma_done;
          const bool h0 = i % HB == 0, l0 = i % LB == 0;
          if (h0) {
            if (!mbar_wait(&acce[0], eh ^ 1, abort_flag, p.err, 12)) goto mma_done;
            eh ^= 1;
          }
          fence_after();
          const uint32_t st = smem_u32(smem + stage * STAGE_BYTES);
          // descriptors are linear in the address (units of 16 bytes): + 2 per 16 K elements
          const uint64_t a0d = sdesc(st, 512, 4), b0d = sdesc(st + S * A_BYTES, 512, 4);
          auto da = [&](int t, int kk) { return a0d + (uint64_t)(t * (A_BYTES >> 4) + 2 * kk); };
          auto db = [&](int t, int kk) { return b0d + (uint64_t)(t * (B_BYTES >> 4) + 2 * kk); };
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {  // levels 0 .. 3
            const uint32_t a0 = h0 && kk == 0 ? 0u : 1u;
            mma_pair<256>(tmem, da(0, kk), db(0, kk), a0);
            mma_pair<192>(tmem + 64, da(1, kk), db(0, kk), 1u);
            mma_pair<128>(tmem + 128, da(2, kk), db(0, kk), 1u);
            mma_pair<64>(tmem + 192, da(3, kk), db(0, kk), 1u);
          }
          if ((i + 1) % HB == 0 || i + 1 == n) mma_commit(&accf[0]);
          if (l0) {
            if (!mbar_wait(&acce[1], el ^ 1, abort_flag, p.err, 16)) goto mma_done;
            el ^= 1;
            fence_after();
          }
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {  // levels 4 .. 7
            const uint32_t a0 = l0 && kk == 0 ? 0u : 1u;
            mma_pair<256>(tmem + 256, da(1, kk), db(3, kk), a0);
            mma_pair<192>(tmem + 256, da(0, kk), db(4, kk), 1u);
            mma_pair<256>(tmem + 256, da(2, kk), db(2, kk), 1u);
            mma_pair<256>(tmem + 256, da(3, kk), db(1, kk), 1u);
            mma_pair<256>(tmem + 256, da(4, kk), db(0, kk), 1u);
            mma_pair<192>(tmem + 320, da(5, kk), db(0, kk), 1u);
            mma_pair<128>(tmem + 384, da(6, kk), db(0, kk), 1u);
          }
          mma_commit(&empty[stage]);
          if ((i + 1) % LB == 0 || i + 1 == n) mma_commit(&accf[1]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    mma_done:;
    }
  } else {
    const int q = warp % 4, part = (warp - 2) / 4;
    const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * EC);
    uint32_t ph = 0, pl = 0;
    float h1[EC], l1[EC], h2[EC], l2[EC];  // levels 0..2 as one pair, 3..7 as the other
    for (int64_t R = blockIdx.x; R < p.ntiles; R += gridDim.x) {
      const Tile tc = tile_of(p, R);
      const int kb0 = tc.s * p.kb_per, n = min(p.nkb, kb0 + p.kb_per) - kb0;
#pragma unroll
      for (int j = 0; j < EC; ++j) h1[j] = l1[j] = h2[j] = l2[j] = 0.f;
      for (int i = 0; i < n; ++i) {
        uint32_t r[EC];
        if ((i + 1) % HB == 0 || i + 1 == n) {
          if (!mbar_wait(&accf[0], ph, abort_flag, p.err, 14)) goto epi_done;
          ph ^= 1;
          fence_after();
          tmem_ld16(tl, r);
          add_level(h1, l1, r);
          tmem_ld16(tl + 64, r);
          add_level(h1, l1, r);
          tmem_ld16(tl + 128, r);
          add_level(h1, l1, r);
          tmem_ld16(tl + 192, r);
          add_level(h2, l2, r);
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[0]);
        }
        if ((i + 1) % LB == 0 || i + 1 == n) {
          if (!mbar_wait(&accf[1], pl, abort_flag, p.err, 17)) goto epi_done;
          pl ^= 1;
          fence_after();
          tmem_ld16(tl + 448, r);
          add_low(l2, r);
          tmem_ld16(tl + 384, r);
          add_low(l2, r);
          tmem_ld16(tl + 320, r);
          add_low(l2, r);
          tmem_ld16(tl + 256, r);
          add_level(h2, l2, r);
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[1]);
        }
      }
      const int64_t row = tc.m * BM + q * 32 + lane;
      if (row < p.M) {
        const int64_t cb = p.cbatch.at(p.b_first + tc.b) + tc.s * p.c_split;
        double *crow = p.C + cb + p.crow.at(p.m_first + row);
        const int ea = max(p.erow_a[tc.b * p.M + row], -5000) - 2 * BIAS + p.alpha_exp;
        const bool neg = p.alpha_pow2 < 0;
        const int64_t n0 = tc.n * BN + part * EC;
        int64_t q0 = n0 % p.ccol.n0, q1 = (n0 / p.ccol.n0) % p.ccol.n1, q2 = n0 / p.ccol.n0 / p.ccol.n1;
#pragma unroll
        for (int j = 0; j < EC; ++j) {
          if (n0 + j < p.N) {
            const int e = ea + max(__ldg(p.erow_b + tc.b * p.N + n0 + j), -5000);
            double v = assemble(h1[j], l1[j], h2[j], l2[j], e, neg);
            if (p.alpha_pow2 == 0) v *= p.alpha;
            store_c(p, crow + q2 * p.ccol.s2 + q1 * p.ccol.s1 + q0 * p.ccol.s0, v);
          }
          if (++q0 == p.ccol.n0) {
            q0 = 0;
            if (++q1 == p.ccol.n1) { q1 = 0; ++q2; }
          }
        }
      }
    }
  epi_done:;
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// C (+)= alpha * sum over the K splits of the FP64 partials, in split order; M fastest.
__global__ void oz_reduce_kernel(const double *__restrict__ part, int64_t M, int64_t N, int64_t nbt, int splits,
                                 const OzMap crow, const OzMap ccol, const OzMap cbatch, double *__restrict__ C,
                                 double alpha, double beta) {
  const int64_t mn = M * N, total = mn * nbt;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / mn, e = t % mn;
    const double *q = part + b * splits * mn + e;
    double acc = 0.0;
#pragma unroll 4
    for (int s = 0; s < splits; ++s) acc += q[s * mn];
    double *c = C + cbatch.at(b) + crow.at(e % M) + ccol.at(e / M);
    const double v = alpha * acc;
    *c = beta == 0.0 ? v : fma(beta, *c, v);
  }
}

// ---------------- host ----------------

constexpr int64_t kPlaneBudget = 1LL << 30;  // bytes of digit planes per operand and launch

}  // namespace

bool oz_dgemm(const GemmDesc &d, cudaStream_t stream, GemmWorkspace *ws) {
  OzPlan q;
  if (!ws || !oz_plan(d, sm_count(), kPlaneBudget, q) || !q.faster) return false;
  const int nruns = (int)ceil_div(q.Kp, RUN);
  const int64_t rows_a = q.m_chunk * q.tb_chunk, rows_b = q.N * q.tb_chunk;
  const int64_t ni = 64 + rows_a + rows_b;  // [flag | row exponents of A | of B], then run exponents
  double *partial = nullptr;
  try {
    ws->oz_int.resize((size_t)(ni + (nruns > 1 ? (rows_a + rows_b) * nruns : 0)));
    ws->oz_a.resize((size_t)(rows_a * q.Kp * S));
    ws->oz_b.resize((size_t)(rows_b * q.Kp * S));
    if (q.splits > 1) {
      ws->partial.resize((size_t)(q.nbatch * q.splits * q.M * q.N));
      partial = ws->partial.get();
    }
  } catch (const Error &e) {
    if (e.code != BSE_ERR_OUT_OF_MEMORY) throw;
    cudaGetLastError();  // no room for the planes: the FMA kernel needs none
    return false;
  }
  static std::once_flag attr;
  std::call_once(attr, [] {
    VGB_CUDA(cudaFuncSetAttribute(oz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  });
  GemmArgs p;
  Operand A, B;
  A.p = q.A; A.ks = q.ka; A.map = q.amap;
  B.p = q.B; B.ks = q.kb; B.map = q.bmap;
  A.K = B.K = d.K;
  A.Kp = B.Kp = q.Kp;
  A.nruns = B.nruns = nruns;
  A.planes = ws->oz_a.get();
  B.planes = ws->oz_b.get();
  int *ip = ws->oz_int.get();
  A.erow = ip + 64;
  B.erow = A.erow + rows_a;
  A.erun = B.erow + rows_b;
  B.erun = A.erun + rows_a * nruns;
  p.K = d.K;
  p.nkb = q.nkb;
  p.kb_per = q.kb_per;
  p.splits = q.splits;
  p.flag = ip;
  p.err = ws->error_slot();
  p.c_split = 0;
  if (q.splits > 1) {  // FP64 partials [batch][split][column][row]
    p.C = partial;
    p.alpha = 1.0; p.beta = 0.0;
    p.c_split = q.M * q.N;
    p.cbatch = OzMap{kOzOne, 1, q.splits * q.M * q.N, 0, 0};
    p.crow = OzMap{kOzOne, 1, 1, 0, 0};
    p.ccol = OzMap{kOzOne, 1, q.M, 0, 0};
  } else {
    p.C = d.C;
    p.alpha = d.alpha; p.beta = d.beta;
    p.crow = q.crow; p.ccol = q.ccol; p.cbatch = q.cbatch;
  }
  int ae = 0;
  const double am = std::frexp(p.alpha, &ae);
  p.alpha_pow2 = am == 0.5 ? 1 : am == -0.5 ? -1 : 0;
  p.alpha_exp = p.alpha_pow2 ? ae - 1 : 0;
  // exponents start below any value (0x80808080), the flag at "not set"
  VGB_CUDA(cudaMemsetAsync(ip, 0x80, (size_t)ni * sizeof(int), stream));
  for (int64_t t0 = 0; t0 < q.nbatch; t0 += q.tb_chunk)
    for (int64_t m0 = 0; m0 < q.M; m0 += q.m_chunk) {
      const int64_t tn = std::min(q.tb_chunk, q.nbatch - t0), mn = std::min(q.m_chunk, q.M - m0);
      const bool new_b = m0 == 0;
      A.r0 = t0 * q.M + m0; A.rows = tn * mn;  // row chunks only without batches
      B.r0 = t0 * q.N; B.rows = tn * q.N;
      if (t0 + m0 > 0 && nruns > 1) {
        VGB_CUDA(cudaMemsetAsync(A.erow, 0x80, (size_t)A.rows * sizeof(int), stream));
        if (new_b) VGB_CUDA(cudaMemsetAsync(B.erow, 0x80, (size_t)B.rows * sizeof(int), stream));
      }
      const int64_t ua = ceil_div(A.rows, SROWS) * nruns, ub = new_b ? ceil_div(B.rows, SROWS) * nruns : 0;
      const unsigned sg = (unsigned)std::min<int64_t>(ua + ub, 64LL * sm_count());
      if (nruns > 1) {
        oz_slice_kernel<<<sg, 256, 0, stream>>>(A, B, ua, ua + ub, 1, ip);
        VGB_LAUNCH_CHECK();
      }
      oz_slice_kernel<<<sg, 256, 0, stream>>>(A, B, ua, ua + ub, nruns > 1 ? 2 : 3, ip);
      VGB_LAUNCH_CHECK();
      encode_kmajor(&p.map_a, A.planes, S * A.rows, q.Kp, q.Kp, BM, BK);
      encode_kmajor(&p.map_b, B.planes, S * B.rows, q.Kp, q.Kp, BN, BK);
      p.A = A;
      p.B = B;
      p.M = q.nbatch > 1 ? q.M : mn;
      p.N = q.N;
      p.a_plane = (int)A.rows;
      p.b_plane = (int)B.rows;
      p.erow_a = A.erow;
      p.erow_b = B.erow;
      p.mt = ceil_div(p.M, BM);
      p.nt = ceil_div(p.N, BN);
      p.ntiles = p.mt * p.nt * tn * q.splits;
      p.m_first = m0;
      p.b_first = t0;
      oz_gemm_kernel<<<(unsigned)std::min<int64_t>(p.ntiles, sm_count()), kGemmThreads, SMEM_BYTES, stream>>>(p);
      VGB_LAUNCH_CHECK();
    }
  if (q.splits > 1) {
    const int64_t total = q.nbatch * q.M * q.N;
    oz_reduce_kernel<<<(unsigned)std::min<int64_t>(ceil_div(total, 256), 8LL * sm_count()), 256, 0, stream>>>(
        partial, q.M, q.N, q.nbatch, q.splits, q.crow, q.ccol, q.cbatch, d.C, d.alpha, d.beta);
    VGB_LAUNCH_CHECK();
  }
  return true;
}

}  // namespace vgb
