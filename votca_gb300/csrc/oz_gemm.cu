// FP64 GEMM from exact bf16 digit products (see oz_gemm.cuh for the scheme and its accuracy).
#include "oz_gemm.cuh"

#include <algorithm>
#include <cmath>

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
// output offsets and scale exponents of a tile's rows and columns, two tiles deep
struct TileTab {
  int64_t row[BM], col[BN];  // row: -1 beyond the matrix
  int ea[BM], eb[BN];
};
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256 + 2 * (int)sizeof(TileTab);
constexpr int kEpi = 16;                     // epilogue warps: four per TMEM lane quarter
constexpr int EC = BN / 4;                   // columns of an epilogue thread
constexpr int kTab = 2;                       // warps that prepare a tile's output addresses
constexpr int kGemmThreads = 64 + 32 * (kEpi + kTab);  // warp 0: TMA, warp 1: MMA, epilogue, tables
constexpr int BITS = 8 * S - 1;              // digit window: |x| < 2^e -> |m| <= 2^BITS
constexpr int BIAS = 50;                     // operand digits carry 2^(BIAS - row exponent)
constexpr int ZERO_RUN = -100000;            // exponent of a run of zeros
constexpr int kOpposed = 12;                 // bits that opposed gradings along K may have
constexpr int TOP = 127 + BIAS - 1;          // exponent of a row's largest first digits (64 .. 127)
constexpr int E_MAX = 900;                   // larger or smaller exponents take the FMA path
static_assert(LV * BN <= 512 && SMEM_BYTES <= 232448, "tile exceeds the SM");

// One operand: rows [r0, r0 + rows) of the map, K columns ks apart, and its planes.
struct Operand {
  const double *p = nullptr;
  OzMap map;
  int64_t r0 = 0, rows = 0, K = 0, Kp = 0, ks = 1;
  uint16_t *planes = nullptr;  // [t][rows][Kp]
  int *erow = nullptr;         // exponent of the row's largest element (per row)
  int *erun = nullptr;         // per (row, run), only for rows of several segments
  int nruns = 1;
  int *prof = nullptr;         // per K element: the largest first digit of any row, as bf16 bits
};

// ---------------- digits ----------------

// Digits of two consecutive K elements, one packed word per plane.  x = +-sum_t d_t 2^(e - 7 - 8 t):
// the value m = round(|x| 2^(BITS - e)) in 64-bit integers and its balanced bytes (adding 128 to
// every byte but the top one makes each byte d + 128); the bf16 value d sc_t comes from one FFMA
// on 2^23 + byte, the sign from one XOR per pair.  Zeros, subnormals and runs of zeros
// (e = ZERO_RUN) shift out to 0.
__device__ __forceinline__ void digits2(unsigned long long x0, unsigned long long x1, int e, const float (&sc)[S],
                                        const float (&cc)[S], uint32_t (&out)[S]) {
  // (m << 1) + 1 + 2 bias before the last shift: rounding and bias in one addition
  constexpr unsigned long long rb = 2 * 0x0000808080808080ull + 1;
  auto fixed = [&](unsigned long long x) {
    const uint32_t h = (uint32_t)(x >> 32), l = (uint32_t)x;
    // mantissa 2^10 (63 bits) shifted right by (e - exponent) + 62 - BITS: 2 m with one guard bit
    const unsigned long long M = ((unsigned long long)((h & 0xFFFFFu) | 0x100000u) << 32 | l) << 10;
    const uint32_t sh = (uint32_t)(e + 1022 + 62 - BITS) - ((h >> 20) & 0x7FFu);
    unsigned long long t;
    asm("shr.u64 %0, %1, %2;" : "=l"(t) : "l"(M), "r"(sh));  // amounts beyond 63 give 0
    return (t + rb) >> 1;
  };
  const unsigned long long u0 = fixed(x0), u1 = fixed(x1);
  const uint32_t lo0 = (uint32_t)u0, hi0 = (uint32_t)(u0 >> 32), lo1 = (uint32_t)u1, hi1 = (uint32_t)(u1 >> 32);
  const uint32_t sg = __byte_perm((uint32_t)(x0 >> 32), (uint32_t)(x1 >> 32), 0x7632) & 0x80008000u;
#pragma unroll
  for (int t = 0; t < S; ++t) {
    uint32_t w0, w1;
    if (t == 0) {
      w0 = 0x4B000080u + (hi0 >> 16);  // the top digit is not biased: 0 .. 128
      w1 = 0x4B000080u + (hi1 >> 16);
    } else {
      const int sel = t == 1 || t == 5 ? 0x7651 : t == 2 || t == 6 ? 0x7650 : t == 3 ? 0x7653 : 0x7652;
      w0 = __byte_perm(t <= 2 ? hi0 : lo0, 0x4B000000u, sel);
      w1 = __byte_perm(t <= 2 ? hi1 : lo1, 0x4B000000u, sel);
    }
    const float f0 = fmaf(__uint_as_float(w0), sc[t], cc[t]), f1 = fmaf(__uint_as_float(w1), sc[t], cc[t]);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out[t]) : "f"(f1), "f"(f0));
    out[t] ^= sg;
  }
}

// Eight consecutive K elements into the planes (16 bytes each); top: the largest magnitudes of their first
// digits so far, two bf16 to a word.
__device__ __forceinline__ void store8(const unsigned long long *x, int e, const float (&sc)[S], const float (&cc)[S],
                                       uint16_t *out, int64_t plane, uint32_t (&top)[4]) {
  uint32_t d[4][S];
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    digits2(x[2 * v], x[2 * v + 1], e, sc, cc, d[v]);
    top[v] = __vmaxu2(top[v], d[v][0] & 0x7FFF7FFFu);
  }
#pragma unroll
  for (int t = 0; t < S; ++t, out += plane)
    *reinterpret_cast<uint4 *>(out) = make_uint4(d[0][t], d[1][t], d[2][t], d[3][t]);
}

// Scales of a row's digits, sc[t] = 2^(rel + BIAS - 7 - 8 t), and cc[t] = -(2^23 + 128) sc[t]; runs
// far below their row (rel < -169) vanish.
__device__ __forceinline__ void digit_scales(int rel, float (&sc)[S], float (&cc)[S]) {
  const int pe = 127 + rel + BIAS - 7;
  sc[0] = pe >= 1 ? __int_as_float(pe << 23) : 0.f;
#pragma unroll
  for (int t = 1; t < S; ++t) sc[t] = sc[t - 1] * 0.00390625f;
#pragma unroll
  for (int t = 0; t < S; ++t) cc[t] = -8388736.0f * sc[t];
}

// Rows of one block's unit (256 threads, segments of 256 K elements): 32, and more where the rows
// are shorter.
constexpr int SEG = 256;
__host__ __device__ __forceinline__ int slice_rows(int64_t Kp) {
  return Kp <= 32 ? 256 : Kp <= 64 ? 128 : Kp <= 128 ? 64 : 32;
}

// Digit planes of slice_rows rows and a segment of K per block.  phase 3 (rows of one segment): the
// row maxima, then the digits; longer rows: phase 1 takes the run and row exponents, phase 2 the
// digits and, for the check of opposed gradings, the largest first digit of every K element (3 % of the
// kernel's time).  Every element is loaded once per phase.  The digits are made by a warp (part) per row,
// eight elements per lane, so that the planes are written in whole lines; operands contiguous
// along K are read that way, others (contiguous along the rows) with a lane per row, 32 elements
// of it in flight, and turned in shared memory.  Bound: HBM (8 bytes read, 14 written per element)
// when large.  66000 x 220 contiguous along the rows: 125 us in strips of 64 elements with 130
// instructions per element, 143 us with a lane per row to the end (16-byte stores to 32 lines),
// 70 us.
constexpr int SLICE_SMEM = 256 * (32 + 2) * 8;  // the largest tile: rows x (elements + 2)
__global__ void __launch_bounds__(256, 2) oz_slice_kernel(const __grid_constant__ Operand oa,
                                                          const __grid_constant__ Operand ob, int units_a, int units,
                                                          int phase, int *flag) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned long long tile[];
  __shared__ unsigned long long red[256];
  __shared__ int s_e[256];
  __shared__ uint4 s_top[2][8][SEG / 8];  // first digits per warp, two units deep
  int pair = 0;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr unsigned long long kAbs = ~(1ull << 63);  // |x| as integers: of a double it is an FP64 instruction
  for (int u0 = blockIdx.x; u0 < units; u0 += gridDim.x) {  // 32-bit divisions: 64-bit ones use the FP64 pipe
    const bool is_a = u0 < units_a;
    const Operand &o = is_a ? oa : ob;
    const int u = is_a ? u0 : u0 - units_a;
    const int nseg = ((int)o.Kp + SEG - 1) / SEG, urows = slice_rows(o.Kp);
    const int64_t rb = (int64_t)(u / nseg) * urows;
    const int nrow = (int)min((int64_t)urows, o.rows - rb);
    const int seg = u % nseg, run = seg / (RUN / SEG);
    const int64_t k0 = (int64_t)seg * SEG;
    const int kn = (int)min((int64_t)SEG, o.K - k0), kp = (int)min((int64_t)SEG, o.Kp - k0);  // and with padding
    const int64_t plane = o.rows * o.Kp;
    const unsigned long long *base = reinterpret_cast<const unsigned long long *>(o.p);
    const int nwk = 256 / urows, ldt = 32 * nwk + 2;  // warps along K (32 elements each), row stride of the tile
    auto exponent = [&](unsigned long long mx) {  // mx < 2^e
      const int e = mx == 0 ? ZERO_RUN : (int)(mx >> 52) - 1022;
      // infinities, NaNs and the ends of the exponent range: the whole product by FMA
      if (mx != 0 && (e > E_MAX || e < -E_MAX)) atomicMax(flag, 1);
      return e;
    };
    auto record = [&](int64_t row, int e) {
      if (phase == 1) {
        atomicMax(o.erun + row * o.nruns + run, e);
        atomicMax(o.erow + row, e);
      } else {
        o.erow[row] = e;
      }
    };
    const bool turned = o.ks != 1;
    uint32_t top[4] = {0, 0, 0, 0};
    // read ahead: most units find nothing larger, and need no atomic on a line that all of them share
    const int known = phase != 1 && tid < kn ? __ldcg(o.prof + k0 + tid) : 0;
    if (turned) {  // lanes along the rows: loads, maxima, tile
      const int r = (warp / nwk) * 32 + lane, k = (warp % nwk) * 32;
      const bool in = r < nrow && k < kp;
      unsigned long long x[32];
      const unsigned long long *src = base + o.map.at(o.r0 + rb + (in ? r : 0)) + (k0 + k) * o.ks;
#pragma unroll
      for (int v = 0; v < 32; ++v, src += o.ks) x[v] = in && k + v < kn ? *src : 0ull;
      __syncthreads();  // the previous unit's shared values are read
      if (phase & 1) {
        unsigned long long mx = 0;
#pragma unroll
        for (int v = 0; v < 32; ++v) mx = (x[v] & kAbs) > mx ? (x[v] & kAbs) : mx;
        red[tid] = mx;
      }
      if (phase != 1) {
#pragma unroll
        for (int v = 0; v < 32; ++v) tile[r * ldt + k + v] = x[v];
      }
      __syncthreads();
      if ((phase & 1) && warp % nwk == 0 && r < nrow) {
        unsigned long long mx = red[tid];
        for (int w = 1; w < nwk; ++w) mx = red[tid + 32 * w] > mx ? red[tid + 32 * w] : mx;
        const int e = exponent(mx);
        s_e[r] = e;
        record(rb + r, e);
      }
      if (phase == 1) continue;
      if (phase == 3) __syncthreads();
    }
    // digits: lanes of one row, eight elements each
    const int lpr = kp <= 32 ? 4 : kp <= 64 ? 8 : kp <= 128 ? 16 : 32, rpw = 32 / lpr;
    const int k = 8 * (lane & (lpr - 1));
    for (int q = 0; q < urows / 8; q += rpw) {
      const int r = warp * (urows / 8) + q + lane / lpr;
      const int64_t row = rb + r;
      const bool in = r < nrow && k < kp;
      unsigned long long x[8];
      if (turned) {
        const unsigned long long *src = tile + (in ? r * ldt + k : 0);
#pragma unroll
        for (int v = 0; v < 8; v += 2) {
          const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(src + v);
          x[v] = a.x;
          x[v + 1] = a.y;
        }
      } else {
        const unsigned long long *src = base + (in ? o.map.at(o.r0 + row) + k0 + k : 0);
        if (in && ((uintptr_t)src & 15) == 0 && k + 8 <= kn) {
#pragma unroll
          for (int v = 0; v < 8; v += 2) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(src + v);
            x[v] = a.x;
            x[v + 1] = a.y;
          }
        } else {
#pragma unroll
          for (int v = 0; v < 8; ++v) x[v] = in && k + v < kn ? src[v] : 0ull;
        }
      }
      int e = 0, rel = 0;
      if (phase == 2) {
        if (in) {
          e = o.erun[row * o.nruns + run];
          rel = e == ZERO_RUN ? 0 : e - o.erow[row];
        }
      } else if (turned) {
        if (in) e = s_e[r];
      } else {
        unsigned long long mx = 0;
#pragma unroll
        for (int v = 0; v < 8; ++v) mx = (x[v] & kAbs) > mx ? (x[v] & kAbs) : mx;
        for (int w = lpr / 2; w; w >>= 1) {
          const unsigned long long y = __shfl_xor_sync(0xffffffffu, mx, w);
          mx = y > mx ? y : mx;
        }
        e = mx == 0 ? ZERO_RUN : (int)(mx >> 52) - 1022;
        if (k == 0 && in) record(row, exponent(mx));
        if (phase == 1) continue;
      }
      if (in) {
        float sc[S], cc[S];
        digit_scales(rel, sc, cc);
        store8(x, e, sc, cc, o.planes + row * o.Kp + k0 + k, plane, top);
      }
    }
    if (phase == 1) continue;
    for (int w = lpr; w < 32; w *= 2) {  // lanes of other rows
#pragma unroll
      for (int v = 0; v < 4; ++v) top[v] = __vmaxu2(top[v], __shfl_xor_sync(0xffffffffu, top[v], w));
    }
    if (lane < lpr) s_top[pair][warp][lane] = make_uint4(top[0], top[1], top[2], top[3]);
    __syncthreads();
    if (tid < kn) {
      unsigned t = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) t = max(t, (unsigned)reinterpret_cast<const uint16_t *>(s_top[pair][w])[tid]);
      if ((int)t > max(known, 0)) atomicMax(o.prof + k0 + tid, (int)t);
    }
    pair ^= 1;
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
  int mt, nt, ntiles;
  const int *erow_a, *erow_b, *flag;
  const int *prof_a, *prof_b;  // 4 nprof each
  int nprof;
  Operand A, B;              // sources, for the FMA path
  OzMap crow, ccol, cbatch;  // C offsets of tile rows, columns and batches
  int64_t c_split;           // C offset between K splits (partials)
  double *C;
  double alpha, beta;
  int alpha_exp, alpha_pow2; // alpha = +-2^alpha_exp
  int accumulate;            // beta != 0 (an FP64 comparison costs what an FMA does)
  int wait_us;               // limit of the waits
  int plain;                 // neither alpha (a power of two) nor beta costs FP64 work per element
  int *err;
};

struct Tile {
  int m, n, b, s;
};
// M tiles in panels of 16, so that the tiles in flight share their A and B planes in L2
__device__ __forceinline__ Tile tile_of(const GemmArgs &p, int tile) {
  Tile c;
  uint32_t t = (uint32_t)tile;
  const uint32_t per = (uint32_t)(p.mt * p.nt * p.splits);
  c.b = (int)(t / per);
  t -= c.b * per;
  const uint32_t pw = 16u * (uint32_t)(p.nt * p.splits), pan = t / pw;
  t -= pan * pw;
  const uint32_t g = min(16u, (uint32_t)p.mt - pan * 16u);
  c.m = (int)(pan * 16 + t % g);
  t /= g;
  c.n = (int)(t % (uint32_t)p.nt);
  c.s = (int)(t / (uint32_t)p.nt);
  return c;
}

__device__ __forceinline__ void two_sum(float &h, float &l, float x) {
  const float s = h + x, bb = s - h;
  l += (h - (s - bb)) + (x - bb);
  h = s;
}

// the 16 columns of a thread at TMEM address t, eight at a time, into the pair sums (h, l) or l
__device__ __forceinline__ void add_level(float (&h)[EC], float (&l)[EC], uint32_t t) {
#pragma unroll
  for (int j0 = 0; j0 < EC; j0 += 8) {
    uint32_t r[8];
    tmem_ld(t + j0, r);
#pragma unroll
    for (int j = 0; j < 8; ++j) two_sum(h[j0 + j], l[j0 + j], __uint_as_float(r[j]));
  }
}
__device__ __forceinline__ void add_low(float (&l)[EC], uint32_t t) {
#pragma unroll
  for (int j0 = 0; j0 < EC; j0 += 8) {
    uint32_t r[8];
    tmem_ld(t + j0, r);
#pragma unroll
    for (int j = 0; j < 8; ++j) l[j0 + j] += __uint_as_float(r[j]);
  }
}

// The float with bits b as a fixed point: mantissa 2^36 shifted down by top - its exponent (a zero
// has no exponent to speak of and shifts out)
__device__ __forceinline__ long long place(uint32_t b, int top) {
  const int sg = (int)b >> 31;
  const int m = ((int)((b & 0x7FFFFFu) | 0x800000u) ^ sg) - sg;
  long long r;
  // shifts beyond 63 give the sign
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"((long long)((unsigned long long)(uint32_t)(m << 4) << 32)),
      "r"((uint32_t)(top - (int)((b >> 23) & 0xFF))));
  return r;
}

// (h1 + l1 + h2 + l2) 2^e rounded to FP64: l1 + h2 + l2 as a float pair, the three floats in one
// 62-bit fixed point, one conversion, the exponent in integers.  Every FP64 instruction of an
// element (also one behind a false predicate) is 64 clocks of an SM quarter, 4096 a tile: with a
// comparison, a scaling and an update compiled in for all, the last step was a third of the
// kernel on 66000 x 450 x 220 (440 us, 345 without them).
__device__ __forceinline__ double assemble(float h1, float l1, float h2, float l2, int e, bool neg) {
  float c = l1, z = 0.f;
  two_sum(c, z, h2);
  z += l2;
  const uint32_t b0 = __float_as_uint(h1), b1 = __float_as_uint(c), b2 = __float_as_uint(z);
  const int top = max((int)((b0 >> 23) & 0xFF), max((int)((b1 >> 23) & 0xFF), (int)((b2 >> 23) & 0xFF)));
  const double v = __ll2double_rn(place(b0, top) + place(b1, top) + place(b2, top));
  const int hi = __double2hiint(v), lo = __double2loint(v);
  const int sg = neg ? (int)0x80000000 : 0;
  if (top == 0 || hi == 0) return __hiloint2double(sg, 0);  // zero
  const int k = e + top - 186;  // 2^36 and the float's 2^(top - 150)
  const int be = ((hi >> 20) & 0x7FF) + k;
  if (be >= 1 && be <= 2046) return __hiloint2double((hi + (k << 20)) ^ sg, lo);
  const double r = scalbn(v, k);  // over- or underflow
  return neg ? -r : r;
}

__device__ __forceinline__ void store_c(const GemmArgs &p, double *c, double v) {
  *c = p.accumulate ? fma(p.beta, *c, v) : v;
}

// The tile by FP64 FMA, for operands with infinities, NaNs or exponents at the ends of the range, and for
// operands graded in opposite directions: the 64 x 64 register tiles of dgemm.cu on the CTA's first 256 threads.
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
    const int64_t m0 = (int64_t)tc.m * BM + 64 * h, n0 = (int64_t)tc.n * BN;
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
// bytes per clock and SM at the full MMA rate (a stage per pair group would
// load 96).  One MMA multiplies A plane a with up to four stacked B planes
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
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  if (*p.flag > 0) {  // uniform over the grid: set by the slicer, an earlier launch
    for (int R = blockIdx.x; R < p.ntiles; R += gridDim.x)
      fma_tile(p, tile_of(p, R), reinterpret_cast<double *>(smem));
    return;
  }
  uint64_t *full = (uint64_t *)(smem + STAGES * STAGE_BYTES);
  uint64_t *empty = full + STAGES;
  uint64_t *accf = empty + STAGES;  // [0]: H complete, [1]: L complete
  uint64_t *acce = accf + 2;        // drained
  uint64_t *tabf = acce + 2;        // table of a tile ready / read, two deep
  uint64_t *tabe = tabf + 2;
  TcControl *ctl = (TcControl *)(tabe + 2);
  volatile int *abort_flag = &ctl->abort;
  TileTab *tabs = reinterpret_cast<TileTab *>(smem + STAGES * STAGE_BYTES + 256);
  __shared__ int s_meet[3];  // A has elements, B has, some meet
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&accf[i], 1);
      mbar_init(&acce[i], kEpi);
      mbar_init(&tabf[i], 32 * kTab);
      mbar_init(&tabe[i], kEpi);
    }
    ctl->init(p.wait_us);
    s_meet[0] = s_meet[1] = s_meet[2] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = ctl->tmem;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int R = blockIdx.x; R < p.ntiles; R += gridDim.x) {
        const Tile tc = tile_of(p, R);
        const int ya = (int)(tc.b * p.M) + tc.m * BM, yb = (int)(tc.b * p.N) + tc.n * BN;
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
      for (int j = 0; j < STAGES; ++j)  // every stage consumed before the CTA leaves
        if (!mbar_wait(&empty[j], j < stage ? phase : phase ^ 1, abort_flag, p.err, 15)) break;
    tma_done:
      drain_loads(full, STAGES, stage, phase);  // passes at once unless a wait gave up
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, eh = 0, el = 0;
      for (int R = blockIdx.x; R < p.ntiles; R += gridDim.x) {
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
    mma_done:
      drain_mmas(&ctl->mma_done);  // the epilogue may have given up before the last of them
    }
  } else if (warp >= 2 + kEpi) {
    // ---- output offsets and exponents of every tile, ahead of its epilogue ----
    const int i = threadIdx.x - 64 - 32 * kEpi;  // 0 .. 63
    static_assert(32 * kTab == BN && 2 * BN == BM, "two rows and one column per table thread");
    // Operands graded in opposite directions along K: with their rows scaled to one, no two first digits
    // meet in a product above 2^-kOpposed, and the digits, cut 2^-56 below the largest element of a
    // row, are too few for the whole result.  The same on every CTA.
    {
      int any_a = 0, any_b = 0;
      bool meet = false;  // as a rule among the first K elements; unit vectors may have theirs last
      const int4 *qa = reinterpret_cast<const int4 *>(p.prof_a), *qb = reinterpret_cast<const int4 *>(p.prof_b);
      auto one = [&](int a, int b) {
        a = max(a, 0) >> 7;
        b = max(b, 0) >> 7;
        any_a |= a;
        any_b |= b;
        meet |= a && b && a + b >= 2 * TOP - kOpposed;
      };
      for (int k0 = 0; k0 < p.nprof && !__any_sync(0xffffffffu, meet); k0 += 4 * 32 * kTab) {
        int4 a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = k0 + u * 32 * kTab + i;
          a[u] = k < p.nprof ? __ldcg(qa + k) : make_int4(0, 0, 0, 0);
          b[u] = k < p.nprof ? __ldcg(qb + k) : make_int4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          one(a[u].x, b[u].x);
          one(a[u].y, b[u].y);
          one(a[u].z, b[u].z);
          one(a[u].w, b[u].w);
        }
      }
      if (any_a) s_meet[0] = 1;
      if (any_b) s_meet[1] = 1;
      if (meet) s_meet[2] = 1;
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kTab) : "memory");
    }
    int it = 0;
    for (int R = blockIdx.x; R < p.ntiles; R += gridDim.x, ++it) {
      const Tile tc = tile_of(p, R);
      TileTab &tb = tabs[it & 1];
      if (!mbar_wait(&tabe[it & 1], ((it >> 1) & 1) ^ 1, abort_flag, p.err, 18)) break;
      const int64_t cb = p.cbatch.at(p.b_first + tc.b) + tc.s * p.c_split;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t row = (int64_t)tc.m * BM + i + 64 * h;
        const bool in = row < p.M;
        tb.row[i + 64 * h] = in ? cb + p.crow.at(p.m_first + row) : -1;
        tb.ea[i + 64 * h] = in ? max(p.erow_a[tc.b * p.M + row], -5000) - 2 * BIAS + p.alpha_exp : 0;
      }
      const int64_t col = (int64_t)tc.n * BN + i;
      const bool in = col < p.N;
      tb.col[i] = in ? p.ccol.at(col) : -1;
      tb.eb[i] = in ? max(p.erow_b[tc.b * p.N + col], -5000) : 0;
      mbar_arrive(&tabf[it & 1]);
    }
  } else {
    const int q = warp % 4, part = (warp - 2) / 4;
    const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * EC);
    const bool neg = p.alpha_pow2 < 0;
    int it = 0;
    uint32_t ph = 0, pl = 0;
    float h1[EC], l1[EC], h2[EC], l2[EC];  // levels 0..2 as one pair, 3..7 as the other
    for (int R = blockIdx.x; R < p.ntiles; R += gridDim.x, ++it) {
      const int kb0 = tile_of(p, R).s * p.kb_per, n = min(p.nkb, kb0 + p.kb_per) - kb0;
#pragma unroll
      for (int j = 0; j < EC; ++j) h1[j] = l1[j] = h2[j] = l2[j] = 0.f;
      for (int i = 0; i < n; ++i) {
        if ((i + 1) % HB == 0 || i + 1 == n) {
          if (!mbar_wait_warp(&accf[0], ph, abort_flag, p.err, 14)) goto epi_done;
          ph ^= 1;
          fence_after();
          add_level(h1, l1, tl);
          add_level(h1, l1, tl + 64);
          add_level(h1, l1, tl + 128);
          add_level(h2, l2, tl + 192);
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[0]);
        }
        if ((i + 1) % LB == 0 || i + 1 == n) {
          if (!mbar_wait_warp(&accf[1], pl, abort_flag, p.err, 17)) goto epi_done;
          pl ^= 1;
          fence_after();
          add_low(l2, tl + 448);
          add_low(l2, tl + 384);
          add_low(l2, tl + 320);
          add_level(h2, l2, tl + 256);
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[1]);
        }
      }
      if (!mbar_wait_warp(&tabf[it & 1], (it >> 1) & 1, abort_flag, p.err, 19)) goto epi_done;
      const TileTab &tb = tabs[it & 1];
      const int64_t ro = tb.row[q * 32 + lane];
      const bool opposed = s_meet[0] && s_meet[1] && !s_meet[2];  // written before the first table
      if (ro >= 0 && !opposed) {
        double *crow = p.C + ro;
        const int ea = tb.ea[q * 32 + lane];
        if (p.plain) {
#pragma unroll
          for (int j = 0; j < EC; ++j) {
            const int64_t co = tb.col[part * EC + j];
            if (co >= 0) crow[co] = assemble(h1[j], l1[j], h2[j], l2[j], ea + tb.eb[part * EC + j], neg);
          }
        } else {
#pragma unroll
          for (int j0 = 0; j0 < EC; j0 += 4) {  // four columns at a time: their loads overlap
            double old[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int64_t co = tb.col[part * EC + j0 + v];
              old[v] = co >= 0 && p.accumulate ? crow[co] : 0.0;
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int j = j0 + v;
              const int64_t co = tb.col[part * EC + j];
              if (co >= 0) {
                double x = assemble(h1[j], l1[j], h2[j], l2[j], ea + tb.eb[part * EC + j], neg);
                if (p.alpha_pow2 == 0) x *= p.alpha;
                crow[co] = p.accumulate ? fma(p.beta, old[v], x) : x;
              }
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&tabe[it & 1]);
    }
  epi_done:;
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
  if (s_meet[0] && s_meet[1] && !s_meet[2])
    for (int R = blockIdx.x; R < p.ntiles; R += gridDim.x)
      fma_tile(p, tile_of(p, R), reinterpret_cast<double *>(smem));
}

// C (+)= alpha * sum over the K splits of the FP64 partials, in split order; M fastest.
__global__ void oz_reduce_kernel(const double *part, int64_t M, int64_t N, int64_t nbt, int splits,
                                 const OzMap crow, const OzMap ccol, const OzMap cbatch, double *__restrict__ C,
                                 double alpha, double beta) {
  pdl_wait();
  const int64_t mn = M * N, total = mn * nbt;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const QuotRem tx = quot_rem(t, mn), ex = quot_rem(tx.r, M);
    const int64_t b = tx.q, e = tx.r;
    const double *q = part + b * splits * mn + e;
    double acc = 0.0;
#pragma unroll 4
    for (int s = 0; s < splits; ++s) acc += q[s * mn];
    double *c = C + cbatch.at(b) + crow.at(ex.r) + ccol.at(ex.q);
    const double v = alpha * acc;
    *c = beta == 0.0 ? v : fma(beta, *c, v);
  }
}

// ---------------- host ----------------

// Digit planes of one operand: the workspace's, or beyond what it keeps a block of the stream-ordered
// pool that goes back on the stream after the product.  They are 14 bytes an element, up to several
// GB, and a handle that kept them would take that from the next one's staging.
constexpr int64_t kPlaneKeep = 64LL << 20;
struct Planes {
  cudaStream_t s;
  DeviceBuffer<uint16_t> own;
  uint16_t *p = nullptr;
  explicit Planes(cudaStream_t stream) : s(stream ? stream : cudaStreamLegacy) {}
  void take(DeviceBuffer<uint16_t> &kept, int64_t elems) {
    if (elems * (int64_t)sizeof(uint16_t) <= kPlaneKeep) {
      kept.resize((size_t)elems);
      p = kept.get();
    } else {
      AllocStreamScope scope(s);
      own.resize((size_t)elems);
      p = own.get();
    }
  }
  ~Planes() {
    AllocStreamScope scope(s);
    own.release();
  }
};

}  // namespace

bool oz_dgemm(const GemmDesc &d, cudaStream_t stream, GemmWorkspace *ws) {
  OzPlan q;
  if (!ws || !oz_plan(d, sm_count(), ws->plane_budget, q) || !q.faster) return false;
  const int nruns = (int)ceil_div(q.Kp, RUN);
  const int64_t nseg = ceil_div(q.Kp, SEG);
  const bool two = nseg > 1;  // exponents before digits
  const int64_t rows_a = q.m_chunk * q.tb_chunk, rows_b = q.N * q.tb_chunk;
  // [flag | K profiles of A | of B (16-byte aligned) | row exponents of A | of B], then run exponents
  const int64_t ni = 64 + 2 * q.Kp + rows_a + rows_b;
  double *partial = nullptr;
  Planes pa(stream), pb(stream);
  try {
    ws->oz_int.resize((size_t)(ni + (two ? (rows_a + rows_b) * nruns : 0)));
    pa.take(ws->oz_a, rows_a * q.Kp * S);
    pb.take(ws->oz_b, rows_b * q.Kp * S);
    if (q.splits > 1) {
      ws->partial.resize((size_t)(q.nbatch * q.splits * q.M * q.N));
      partial = ws->partial.get();
    }
  } catch (const Error &e) {
    if (e.code != BSE_ERR_OUT_OF_MEMORY) throw;
    cudaGetLastError();  // no room for the planes: the FMA kernel needs none, and its caller the memory
    ws->oz_int.release();
    ws->oz_a.release();
    ws->oz_b.release();
    return false;
  }
  static PerDevice attr;
  attr.run(current_device(), [] {
    VGB_CUDA(cudaFuncSetAttribute(oz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    VGB_CUDA(cudaFuncSetAttribute(oz_slice_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SLICE_SMEM));
  });
  GemmArgs p;
  Operand A, B;
  A.p = q.A; A.ks = q.ka; A.map = q.amap;
  B.p = q.B; B.ks = q.kb; B.map = q.bmap;
  A.K = B.K = d.K;
  A.Kp = B.Kp = q.Kp;
  A.nruns = B.nruns = nruns;
  A.planes = pa.p;
  B.planes = pb.p;
  int *ip = ws->oz_int.get();
  A.prof = ip + 64;
  B.prof = A.prof + q.Kp;
  A.erow = B.prof + q.Kp;
  B.erow = A.erow + rows_a;
  A.erun = B.erow + rows_b;
  B.erun = A.erun + rows_a * nruns;
  p.K = d.K;
  p.nkb = q.nkb;
  p.kb_per = q.kb_per;
  p.splits = q.splits;
  p.flag = ip;
  p.err = ws->error_slot();
  p.wait_us = ws->wait_us;
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
  p.accumulate = p.beta != 0.0 ? 1 : 0;
  int ae = 0;
  const double am = std::frexp(p.alpha, &ae);
  p.alpha_pow2 = am == 0.5 ? 1 : am == -0.5 ? -1 : 0;
  p.alpha_exp = p.alpha_pow2 ? ae - 1 : 0;
  p.plain = p.alpha_pow2 && !p.accumulate ? 1 : 0;
  // exponents start below any value (0x80808080), the flag at "not set"
  const int64_t nrun_ints = two ? (rows_a + rows_b) * nruns : 0;
  VGB_CUDA(cudaMemsetAsync(ip, 0x80, (size_t)(ni + nrun_ints) * sizeof(int), stream));
  for (int64_t t0 = 0; t0 < q.nbatch; t0 += q.tb_chunk)
    for (int64_t m0 = 0; m0 < q.M; m0 += q.m_chunk) {
      const int64_t tn = std::min(q.tb_chunk, q.nbatch - t0), mn = std::min(q.m_chunk, q.M - m0);
      const bool new_b = m0 == 0;
      A.r0 = t0 * q.M + m0; A.rows = tn * mn;  // row chunks only without batches
      B.r0 = t0 * q.N; B.rows = tn * q.N;
      if (t0 + m0 > 0 && two) {
        VGB_CUDA(cudaMemsetAsync(A.erow, 0x80, (size_t)A.rows * sizeof(int), stream));
        VGB_CUDA(cudaMemsetAsync(A.erun, 0x80, (size_t)(A.rows * nruns) * sizeof(int), stream));
        if (new_b) {
          VGB_CUDA(cudaMemsetAsync(B.erow, 0x80, (size_t)B.rows * sizeof(int), stream));
          VGB_CUDA(cudaMemsetAsync(B.erun, 0x80, (size_t)(B.rows * nruns) * sizeof(int), stream));
        }
      }
      const int64_t ua = ceil_div(A.rows, slice_rows(q.Kp)) * nseg;
      const int64_t ub = new_b ? ceil_div(B.rows, slice_rows(q.Kp)) * nseg : 0;
      const unsigned sg = (unsigned)std::min<int64_t>(ua + ub, 64LL * sm_count());
      if (two) {
        launch_pdl(oz_slice_kernel, sg, 256, SLICE_SMEM, stream, A, B, (int)ua, (int)(ua + ub), 1, ip);
        VGB_LAUNCH_CHECK();
      }
      launch_pdl(oz_slice_kernel, sg, 256, SLICE_SMEM, stream, A, B, (int)ua, (int)(ua + ub), two ? 2 : 3,
                 ip);
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
      p.prof_a = A.prof;
      p.prof_b = B.prof;
      p.nprof = (int)(q.Kp / 4);
      p.mt = (int)ceil_div(p.M, BM);
      p.nt = (int)ceil_div(p.N, BN);
      p.ntiles = (int)(p.mt * p.nt * tn * q.splits);
      p.m_first = m0;
      p.b_first = t0;
      launch_pdl(oz_gemm_kernel, (unsigned)std::min(p.ntiles, sm_count()), kGemmThreads, SMEM_BYTES, stream,
                 p);
      VGB_LAUNCH_CHECK();
    }
  if (q.splits > 1) {
    const int64_t total = q.nbatch * q.M * q.N;
    launch_pdl(oz_reduce_kernel, (unsigned)std::min<int64_t>(ceil_div(total, 256), 8LL * sm_count()), 256, 0,
               stream, partial, q.M, q.N, q.nbatch, q.splits, q.crow, q.ccol, q.cbatch, d.C, d.alpha, d.beta);
    VGB_LAUNCH_CHECK();
  }
  return true;
}

}  // namespace vgb
