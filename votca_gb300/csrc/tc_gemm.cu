// tcgen05 BF16x3 GEMM (see tc_gemm.cuh).
#include "tc_gemm.cuh"

#include "tc_epilogue.cuh"
#include "tc_ptx.cuh"

#include <cuda_bf16.h>

#include <map>
#include <memory>
#include <mutex>

namespace vgb {

namespace {

constexpr int BM = 128;
constexpr int kEpiWarps = 8;   // two warps per TMEM lane quarter, each drains half the columns
constexpr int kThreads = 64 + 32 * kEpiWarps;  // warp 0: TMA, warp 1: MMA + TMEM owner, rest: epilogue
constexpr int kSmemRing = 196608;                     // bytes of operand ring per CTA

// BK = bf16 elements of K per stage row: 64 -> 128-byte rows (SWIZZLE_128B),
// 32 -> 64-byte rows (SWIZZLE_64B, half the stage size, twice the stages).
template <int BN, int BK>
struct Cfg {
  static constexpr int A_BYTES = BM * BK * 2;            // one of hi / lo (one plane)
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;
  static constexpr int STAGES = kSmemRing / STAGE_BYTES > 8 ? 8 : kSmemRing / STAGE_BYTES;
  // accumulator buffers in TMEM: four for the narrow tiles (short K splits: the epilogue of a
  // split may lag the MMAs of the next three), two for the wide ones
  static constexpr int NBUF = BN <= 64 ? 4 : 2;
  static constexpr int TMEM_COLS = NBUF * BN < 32 ? 32 : NBUF * BN;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static constexpr uint32_t SBO = BK == 64 ? 1024 : 512;     // 8 rows of one swizzle atom
  static constexpr uint64_t LAYOUT = BK == 64 ? 2 : 4;       // SWIZZLE_128B / SWIZZLE_64B
};

struct KParams {
  int64_t M, N, K;
  int products;  // 3: hi.hi + hi.lo + lo.hi;  4: + lo.lo
  int64_t nbatch, a_brows, b_brows;
  int ksplit, kc_per;
  int kacc;  // 1: one CTA runs the K splits of a tile and sums them as float pairs
  int64_t mt, nt, ntiles, nitems;
  TcEpilogue epi;
  int *err;
};

struct TileCoord {
  int64_t m, n, s, b;
};
__device__ __forceinline__ TileCoord decode(const KParams &p, int64_t t) {
  TileCoord c;
  QuotRem x;
  if (p.kacc) {  // the K splits of a tile are consecutive jobs of one CTA
    x = quot_rem(t, p.ksplit);
    c.s = x.r;
    x = quot_rem(x.q, p.mt);
    c.m = x.r;
    x = quot_rem(x.q, p.nt);
    c.n = x.r;
    c.b = x.q;
    return c;
  }
  x = quot_rem(t, p.mt);
  c.m = x.r;
  x = quot_rem(x.q, p.nt);
  c.n = x.r;
  x = quot_rem(x.q, p.ksplit);
  c.s = x.r;
  c.b = x.q;
  return c;
}

// Work items of the persistent kernel: an item is one tile job, or, for a problem with in-CTA K
// accumulation (kacc), the ksplit consecutive jobs of one output tile; items are strided over
// the CTAs and a CTA runs the jobs of its item in order.
__host__ __device__ __forceinline__ int64_t item_count(const KParams &p) {
  return p.kacc ? p.nitems : p.ntiles;
}
__device__ __forceinline__ int64_t item_len(const KParams &p) { return p.kacc ? p.ksplit : 1; }

// K blocks [kb, ke) of split s.
struct KRange {
  int kb, ke;
};
template <int BK>
__device__ __forceinline__ KRange k_range(const KParams &p, int64_t s) {
  KRange r;
  const int kchunks = (int)(p.K / BK);
  r.kb = (int)s * p.kc_per;
  r.ke = min(kchunks, r.kb + p.kc_per);
  return r;
}

// Problem sources of the persistent kernel: one problem, or a group of up to
// kGroupMax problems (same tile shape) whose item lists are concatenated.  Both
// live in the kernel parameter space, so every tensor map is a __grid_constant__.
struct SingleSrc {
  CUtensorMap maps[4];  // A hi, A lo, B hi, B lo
  KParams p;
  __device__ __forceinline__ int64_t total() const { return item_count(p); }
  __device__ __forceinline__ int locate(int64_t t, int64_t &local, int &) const {
    local = t;
    return 0;
  }
  __device__ __forceinline__ const KParams &params(int) const { return p; }
  __device__ __forceinline__ const CUtensorMap *map(int, int w) const { return &maps[w]; }
  __device__ __forceinline__ int *err() const { return p.err; }
};

constexpr int kGroupMax = 32;
struct GroupSrc {
  CUtensorMap maps[4 * kGroupMax];
  KParams p[kGroupMax];
  int64_t begin[kGroupMax + 1];  // first global item of each problem; begin[n] = total
  int n;
  int *err_ptr;
  __device__ __forceinline__ int64_t total() const { return begin[n]; }
  // t grows along a CTA's walk, so the problem index only moves forward from the hint
  __device__ __forceinline__ int locate(int64_t t, int64_t &local, int &hint) const {
    while (hint + 1 < n && begin[hint + 1] <= t) ++hint;
    local = t - begin[hint];
    return hint;
  }
  __device__ __forceinline__ const KParams &params(int i) const { return p[i]; }
  __device__ __forceinline__ const CUtensorMap *map(int i, int w) const { return &maps[4 * i + w]; }
  __device__ __forceinline__ int *err() const { return err_ptr; }
};
static_assert(sizeof(GroupSrc) <= 32000, "grouped GEMM parameters exceed the kernel parameter space");

template <int BN, int BK, class Src>
__global__ void __launch_bounds__(kThreads, 1) tc_gemm_kernel(const __grid_constant__ Src src) {
  pdl_wait();
  using C = Cfg<BN, BK>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *full = (uint64_t *)(smem + C::STAGES * C::STAGE_BYTES);
  uint64_t *empty = full + C::STAGES;
  uint64_t *accf = empty + C::STAGES;
  uint64_t *acce = accf + C::NBUF;
  TcControl *ctl = (TcControl *)(acce + C::NBUF);
  volatile int *abort_flag = &ctl->abort;

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int i = 0; i < C::STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < C::NBUF; ++i) {
      mbar_init(&accf[i], 1);
      mbar_init(&acce[i], kEpiWarps);  // one arrive per epilogue warp
    }
    ctl->init(kWaitUs);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ctl->tmem)),
                 "r"((uint32_t)C::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = ctl->tmem;
  int *const err = src.err();
  const int64_t nitems = src.total();  // item R: jobs li * len + u, u < len (see item_len)

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- TMA producer ----------------
      int stage = 0;
      uint32_t phase = 0;
      int hint = 0;
      for (int64_t R = blockIdx.x; R < nitems; R += gridDim.x) {
        int64_t li;
        const int pi = src.locate(R, li, hint);
        const KParams p = src.params(pi);  // registers: no reloads behind the stores
        const int64_t len = item_len(p);
        const CUtensorMap *mAhi = src.map(pi, 0), *mAlo = src.map(pi, 1);
        const CUtensorMap *mBhi = src.map(pi, 2), *mBlo = src.map(pi, 3);
        // the jobs of an item share the tile; only the K split advances (decode once per item)
        TileCoord tc = decode(p, li * len);
        const int ya = (int)(tc.b * p.a_brows + tc.m * BM);
        const int yb = (int)(tc.b * p.b_brows + tc.n * BN);
        for (int64_t u = 0; u < len; ++u, ++tc.s) {
          const KRange kr = k_range<BK>(p, tc.s);
          for (int kc = kr.kb; kc < kr.ke; ++kc) {
            if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, err, 1)) goto producer_done;
            uint8_t *st = smem + stage * C::STAGE_BYTES;
            mbar_expect_tx(&full[stage], (uint32_t)C::STAGE_BYTES);
            tma_load_2d(smem_u32(st), mAhi, &full[stage], kc * BK, ya);
            tma_load_2d(smem_u32(st + C::A_BYTES), mAlo, &full[stage], kc * BK, ya);
            tma_load_2d(smem_u32(st + 2 * C::A_BYTES), mBhi, &full[stage], kc * BK, yb);
            tma_load_2d(smem_u32(st + 2 * C::A_BYTES + C::B_BYTES), mBlo, &full[stage], kc * BK, yb);
            if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
          }
        }
      }
      for (int j = 0; j < C::STAGES; ++j)  // every stage consumed before the CTA leaves
        if (!mbar_wait(&empty[j], j < stage ? phase : phase ^ 1, abort_flag, err, 5)) break;
    producer_done:
      drain_loads(full, C::STAGES, stage, phase);  // passes at once unless a wait gave up
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- MMA issuer ----------------
      constexpr uint32_t idesc = (1u << 4)                   // D: FP32
                                 | (1u << 7) | (1u << 10)     // A, B: BF16
                                 | ((uint32_t)(BN >> 3) << 17) // N
                                 | ((uint32_t)(BM >> 4) << 24); // M
      int stage = 0;
      uint32_t phase = 0;
      int buf = 0;
      uint32_t aphase = 0;
      int hint = 0;
      for (int64_t R = blockIdx.x; R < nitems; R += gridDim.x) {
        int64_t li;
        const KParams p = src.params(src.locate(R, li, hint));
        const int64_t len = item_len(p);
        // the jobs of an item share the tile; only the K split advances (decode once per item)
        TileCoord tc = decode(p, li * len);
        for (int64_t u = 0; u < len; ++u, ++tc.s) {
          const KRange kr = k_range<BK>(p, tc.s);
          const int kb = kr.kb, ke = kr.ke;
          if (!mbar_wait(&acce[buf], aphase ^ 1, abort_flag, err, 2)) goto mma_done;
          fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
          for (int kc = kb; kc < ke; ++kc) {
            if (!mbar_wait(&full[stage], phase, abort_flag, err, 3)) goto mma_done;
            fence_after();
            const uint32_t st = smem_u32(smem + stage * C::STAGE_BYTES);
            // descriptors are linear in the address: + 2 per 16 bf16 (32 bytes) along K
            const uint64_t dah0 = sdesc(st, C::SBO, C::LAYOUT);
            const uint64_t dal0 = dah0 + (C::A_BYTES >> 4);
            const uint64_t dbh0 = dah0 + ((2 * C::A_BYTES) >> 4);
            const uint64_t dbl0 = dbh0 + (C::B_BYTES >> 4);
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
              const uint32_t acc0 = (kc > kb || kk > 0) ? 1u : 0u;
              const uint64_t dah = dah0 + 2 * kk, dal = dal0 + 2 * kk;
              const uint64_t dbh = dbh0 + 2 * kk, dbl = dbl0 + 2 * kk;
              mma_bf16(d_tmem, dah, dbh, idesc, acc0);
              mma_bf16(d_tmem, dah, dbl, idesc, 1u);
              mma_bf16(d_tmem, dal, dbh, idesc, 1u);
              if (p.products == 4) mma_bf16(d_tmem, dal, dbl, idesc, 1u);
            }
            mma_commit(&empty[stage]);  // frees the smem stage when these MMAs complete
            if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
          }
          mma_commit(&accf[buf]);  // accumulator ready for the epilogue
          if (++buf == C::NBUF) { buf = 0; aphase ^= 1; }
        }
      }
    mma_done:
      drain_mmas(&ctl->mma_done);  // the epilogue may have given up before the last of them
    }
  } else {
    // ---------------- epilogue warps ----------------
    // A warp may only read the TMEM lane quarter 32 * (warp % 4); the warps of each quarter split
    // the tile's columns.
    const int q = warp % 4;
    const int part = (warp - 2) / 4;
    constexpr int COLS = BN >= 64 ? BN / 2 : BN;
    const int cbeg = min(part * COLS, BN);
    const int cend = min(cbeg + COLS, BN);
    // float-pair sums over the K splits of a tile (kacc; BN <= 64: at most 32 columns per thread)
    constexpr int KACC = BN <= 64 ? 32 : 1;
    float kh[KACC], kl[KACC];
    int buf = 0;
    uint32_t aphase = 0;
    int hint = 0;
    for (int64_t R = blockIdx.x; R < nitems; R += gridDim.x) {
      int64_t li;
      // a register copy: the stores below cannot alias it, so nothing is reloaded per element
      const KParams p = src.params(src.locate(R, li, hint));
      const TcEpilogue &e = p.epi;
      const int64_t len = item_len(p);
      // the jobs of an item share the tile: row terms once per item
      TileCoord tc = decode(p, li * len);
      const int64_t i = tc.m * BM + q * 32 + lane;
      const QuotRem ix = quot_rem(i, e.rd);
      const bool row_ok = i < p.M && ix.r < e.rlim;
      // partial offset: the K split (F32 partials); none with kacc
      const int64_t rbase = ix.q * e.ro1 + ix.r * e.ro2 + tc.b * e.bo + (p.kacc ? 0 : tc.s * e.so);
      for (int64_t u = 0; u < len; ++u, ++tc.s) {
      if (!mbar_wait_warp(&accf[buf], aphase, abort_flag, err, 4)) goto epi_done;
      fence_after();
      if constexpr (BN <= 64) {
        if (p.kacc) {
          // this thread's 32 columns (cbeg == cend for the idle half of a BN = 32 tile)
          if (cbeg < cend) {
            uint32_t r[32];
            tmem_ld(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + cbeg), r);
            pair_add(kh, kl, r, u == 0);
            if (row_ok && u == len - 1) pair_write(kh, kl, e, p.N, tc.n * BN + cbeg, rbase);  // split order
          }
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[buf]);
          if (++buf == C::NBUF) { buf = 0; aphase ^= 1; }
          continue;
        }
      }
#pragma unroll 1
      for (int c0 = cbeg; c0 < cend; c0 += 32) {
        uint32_t r[32];
        tmem_ld(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + c0), r);
        if (!row_ok) continue;
        const int64_t n0 = tc.n * BN + c0;
        const QuotRem nx = quot_rem(n0, e.cd);
        const int64_t nq0 = nx.q, nr0 = nx.r;
        if (nr0 + 32 <= e.cd && n0 + 32 <= p.N && nr0 + 32 <= e.clim) {
          // fast path: the 32 columns are one arithmetic run of offsets
          const int64_t base = rbase + nq0 * e.co1 + nr0 * e.co2;
          const int64_t st = e.co2;
          if (e.kind == TcEpilogue::SPLIT_BF16) {
            uint16_t *oh = e.out_hi + base, *ol = e.out_lo + base;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float v = __uint_as_float(r[j]);
              const __nv_bfloat16 h = __float2bfloat16_rn(v);
              const __nv_bfloat16 l = __float2bfloat16_rn(v - __bfloat162float(h));
              oh[j * st] = __bfloat16_as_ushort(h);
              ol[j * st] = __bfloat16_as_ushort(l);
            }
          } else if (e.kind == TcEpilogue::STORE_F32) {
            float *o = e.out_f32 + base;
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j * st] = __uint_as_float(r[j]);
          } else {
            double *o = e.out_f64 + base;
            const double al = e.alpha, be = e.beta;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const double rv = al * (double)__uint_as_float(r[j]);
              o[j * st] = (be == 0.0) ? rv : fma(be, o[j * st], rv);
            }
          }
        } else {
          int64_t n = n0, nq = nq0, nr = nr0;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (n < p.N && nr < e.clim)
              epi_store(e, rbase + nq * e.co1 + nr * e.co2, __uint_as_float(r[j]));
            ++n;
            if (++nr == e.cd) { nr = 0; ++nq; }
          }
        }
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acce[buf]);
      if (++buf == C::NBUF) { buf = 0; aphase ^= 1; }
      }
    }
  epi_done:;
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((uint32_t)C::TMEM_COLS));
  }
}

// ---------------- helpers ----------------

__device__ __forceinline__ void split_range(const double *x, int64_t rows, int64_t cols,
                                            const SplitMap &m, uint16_t *__restrict__ hi,
                                            uint16_t *__restrict__ lo, int64_t ldo, int64_t t0,
                                            int64_t step) {
  const int64_t total = rows * cols;
  for (int64_t t = t0; t < total; t += step) {
    const QuotRem tx = quot_rem(t, cols);
    const int64_t r = tx.q, c = tx.r;
    const QuotRem rx = quot_rem(r, m.rdiv);
    const int64_t rq = rx.q, rr = rx.r;
    if (rr >= m.rlim) continue;
    const double v = x[rq * m.rs1 + rr * m.rs2 + c * m.cs];
    const __nv_bfloat16 h = __double2bfloat16(v);
    const __nv_bfloat16 l = __double2bfloat16(v - (double)__bfloat162float(h));
    hi[r * ldo + c] = __bfloat16_as_ushort(h);
    lo[r * ldo + c] = __bfloat16_as_ushort(l);
  }
}

__global__ void split_kernel(const double *x, int64_t rows, int64_t cols,
                             const SplitMap m, uint16_t *__restrict__ hi, uint16_t *__restrict__ lo,
                             int64_t ldo) {
  pdl_wait();
  split_range(x, rows, cols, m, hi, lo, ldo, blockIdx.x * (int64_t)blockDim.x + threadIdx.x,
              (int64_t)gridDim.x * blockDim.x);
}

constexpr int kJobsMax = 96;  // jobs per grouped elementwise launch (parameter space)
struct SplitGroup {
  SplitJob j[kJobsMax];
  int n;
};
struct ReduceGroup {
  ReduceJob j[kJobsMax];
  int n;
};
static_assert(sizeof(SplitGroup) <= 32000 && sizeof(ReduceGroup) <= 32000, "grouped job lists too large");

__global__ void split_group_kernel(const __grid_constant__ SplitGroup g) {
  pdl_wait();
  const SplitJob q = g.j[blockIdx.y];
  split_range(q.x, q.rows, q.cols, q.map, q.hi, q.lo, q.ldo,
              blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

__device__ __forceinline__ void reduce_range(const float *part, int64_t M, int64_t N,
                                             int ksplit, const TcEpilogue &e, int64_t t0, int64_t step) {
  const int64_t total = M * N;
  for (int64_t t = t0; t < total; t += step) {
    const QuotRem tx = quot_rem(t, N);
    const QuotRem ix = quot_rem(tx.q, e.rd), nx = quot_rem(tx.r, e.cd);
    if (ix.r >= e.rlim || nx.r >= e.clim) continue;
    const unsigned *p = reinterpret_cast<const unsigned *>(part) + t;
    double acc;
    if (ksplit <= kSplitRegs) {
      SplitRegs<kSplitRegs> r;
#pragma unroll
      for (int s = 0; s < kSplitRegs; ++s) r.w[s] = s < ksplit ? __ldcg(p + s * total) : 0u;
      acc = sum_splits(ksplit, r);
    } else {
      acc = sum_splits(ksplit, SplitMem{p, total});
    }
    // the partial sums are added in FP64; the final value enters the epilogue
    // as FP64 for AXPBY (no extra rounding) and as FP32 for the bf16 split
    const int64_t off = ix.q * e.ro1 + ix.r * e.ro2 + nx.q * e.co1 + nx.r * e.co2;
    if (e.kind == TcEpilogue::AXPBY_F64) {
      double *y = e.out_f64 + off;
      const double r = e.alpha * acc;
      *y = (e.beta == 0.0) ? r : fma(e.beta, *y, r);
    } else {
      epi_store(e, off, (float)acc);
    }
  }
}

__global__ void reduce_partials_kernel(const float *part, int64_t M, int64_t N,
                                       int ksplit, const TcEpilogue e) {
  pdl_wait();
  reduce_range(part, M, N, ksplit, e, blockIdx.x * (int64_t)blockDim.x + threadIdx.x,
               (int64_t)gridDim.x * blockDim.x);
}

constexpr int kMaxDigits = 5;

// One warp per (row, run of chunk columns): the run's maximum, then its digits, all in integer
// arithmetic on the FP64 bit patterns (the FP64 pipe of GB300 is slow; these are INT32/INT64
// operations): the run scale is 2^e with e the frexp exponent of the largest |x|, an element is
// m = round(x 2^(B - e)) with B = 7 nsl (|m| <= 2^B, a 64-bit integer from its mantissa), and the
// digits are its balanced base-2^7 digits, d_t = round(r / 2^(B - 7t)), r -= d_t 2^(B - 7t).
__device__ __forceinline__ long long fixed_point(unsigned long long bits, int e, int B) {
  const int ef = (int)((bits >> 52) & 0x7FF);
  if (ef == 0) return 0;  // zero or subnormal: below 2^-1022, far under the run scale
  const long long mant = (long long)((bits & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull);
  // value = mant 2^(ef - 1075), m = mant 2^(ef - 1075 + B - e): a right shift by sh >= 53 - B
  const int sh = 1075 + e - ef - B;
  long long m = 0;
  if (sh < 63) m = (mant + (1LL << (sh - 1))) >> sh;
  return (bits >> 63) ? -m : m;
}

// The same fixed point for a float given by its bits: value = mant 2^(ef - 150), m = mant
// 2^(ef - 150 + B - e).  The mantissa is shifted to 2 m with one guard bit (right by at least
// 26 - B + 12 >= 1 for B <= 35; amounts beyond 63 give 0), then rounded half up.
__device__ __forceinline__ long long fixed_point_f32(unsigned bits, int e, int B) {
  const int ef = (int)((bits >> 23) & 0xFF);
  const unsigned mant = ef ? (bits & 0x7FFFFFu) | 0x800000u : 0u;
  unsigned long long t;
  asm("shr.u64 %0, %1, %2;" : "=l"(t) : "l"((unsigned long long)mant << 13), "r"((unsigned)(162 + e - ef - B)));
  const long long m = (long long)((t + 1) >> 1);
  return (int)bits < 0 ? -m : m;
}

// Input element access of the slicer: FP64 values, or float pairs (hi, lo) with value hi + lo.
struct F64In {
  const unsigned long long *p;
  __device__ __forceinline__ unsigned long long abs_bits(int64_t i) const {
    return p[i] & 0x7FFFFFFFFFFFFFFFull;
  }
  // frexp exponent of a maximum (abs_bits): mx < 2^e; subnormal maxima as 2^-1022
  __device__ __forceinline__ static int exponent(unsigned long long mx) {
    return mx == 0 ? 0 : max((int)(mx >> 52), 1) - 1022;
  }
  __device__ __forceinline__ long long fixed(int64_t i, int e, int B) const {
    return fixed_point(p[i], e, B);
  }
  // four consecutive elements (32-byte aligned): raw words, |x| bits, fixed point of a word
  __device__ __forceinline__ void load4(int64_t i, unsigned long long (&w)[4]) const {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(p + i);
    const ulonglong2 b = reinterpret_cast<const ulonglong2 *>(p + i)[1];
    w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
  }
  __device__ __forceinline__ static unsigned long long abs_word(unsigned long long w) {
    return w & 0x7FFFFFFFFFFFFFFFull;
  }
  __device__ __forceinline__ static long long fixed_word(unsigned long long w, int e, int B) {
    return fixed_point(w, e, B);
  }
};
struct PairIn {
  const unsigned long long *p;  // float2 elements
  __device__ __forceinline__ unsigned long long abs_bits(int64_t i) const {
    return (unsigned long long)((unsigned)p[i] & 0x7FFFFFFFu);  // |hi|; hi holds the sum
  }
  __device__ __forceinline__ static int exponent(unsigned long long mx) {
    return mx == 0 ? 0 : max((int)(mx >> 23), 1) - 126;
  }
  __device__ __forceinline__ long long fixed(int64_t i, int e, int B) const {
    return fixed_word(p[i], e, B);
  }
  __device__ __forceinline__ void load4(int64_t i, unsigned long long (&w)[4]) const {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(p + i);
    const ulonglong2 b = reinterpret_cast<const ulonglong2 *>(p + i)[1];
    w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
  }
  __device__ __forceinline__ static unsigned long long abs_word(unsigned long long w) {
    return (unsigned long long)((unsigned)w & 0x7FFFFFFFu);
  }
  __device__ __forceinline__ static long long fixed_word(unsigned long long v, int e, int B) {
    // little-endian float2: hi in the low word
    return fixed_point_f32((unsigned)v, e, B) + fixed_point_f32((unsigned)(v >> 32), e, B);
  }
};

// The bf16 bits of digit d (|d| <= 128) of a run with scale exponent e at digit position t >= 1:
// d 2^(e - 7 t), exact; scales below the FP32 normal range flush to 0.
__device__ __forceinline__ uint16_t digit_bits(long long d, int e, int t) {
  const int pe = e - 7 * t + 127;
  float v = 0.f;
  if (pe >= 1 && pe <= 254) v = (float)(int)d * __int_as_float(pe << 23);
  return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// The digits of one element (fixed point rem of B = 7 nsl bits) into d[0 .. nsl).
__device__ __forceinline__ void digits(long long rem, int nsl, long long (&d)[kMaxDigits]) {
#pragma unroll
  for (int sl = 0; sl < kMaxDigits; ++sl) {
    const int shift = 7 * (nsl - 1 - sl);  // digit sl + 1 has weight 2^(B - 7 (sl + 1))
    long long v = sl < nsl ? rem : 0;      // the last digit: the remaining |rem| <= 64
    if (shift > 0) {
      v = (rem + (1LL << (shift - 1))) >> shift;  // round half up (arithmetic shift: floor)
      rem -= v << shift;
    }
    d[sl] = v;
  }
}

// VEC = 4: a lane handles 4 consecutive columns (one 32-byte load, one 8-byte store per plane);
// needs unit column stride, runs and row bases aligned to 4 elements.
// NSL > 0: the digit count as a compile-time constant (constant shifts); 0: nsl at run time.
template <class In, int VEC, int NSL>
__global__ void slice_kernel(const In in, int64_t rows, int64_t cols, const SplitMap m, int nsl_rt, int64_t chunk,
                             uint16_t *__restrict__ out, int64_t ldo, int64_t plane) {
  pdl_wait();
  const int nsl = NSL > 0 ? NSL : nsl_rt;
  const int lane = threadIdx.x & 31;
  const int64_t nchunks = (cols + chunk - 1) / chunk;
  const int64_t units = rows * nchunks;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < units; u += nwarps) {
    const QuotRem ux = quot_rem(u, nchunks), rx = quot_rem(ux.q, m.rdiv);
    const int64_t r = ux.q, q = ux.r, rq = rx.q, rr = rx.r;
    if (rr >= m.rlim) continue;  // uniform over the warp
    const int64_t base = rq * m.rs1 + rr * m.rs2;
    const int64_t c0 = q * chunk, c1 = min(cols, c0 + chunk);
    unsigned long long mx = 0;  // largest |x| as a bit pattern (ordered like the values)
    if constexpr (VEC == 4) {
      for (int64_t c = c0 + 4 * lane; c < c1; c += 128) {
        if (c + 4 <= c1) {
          unsigned long long w[4];
          in.load4(base + c, w);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const unsigned long long a = In::abs_word(w[v]);
            mx = a > mx ? a : mx;
          }
        } else {
          for (int64_t cc = c; cc < c1; ++cc) {
            const unsigned long long a = In::abs_word(in.p[base + cc]);
            mx = a > mx ? a : mx;
          }
        }
      }
    } else {
      for (int64_t c = c0 + lane; c < c1; c += 32) {
        const unsigned long long a = in.abs_bits(base + c * m.cs);
        mx = a > mx ? a : mx;
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = y > mx ? y : mx;
    }
    const int e = In::exponent(mx);
    uint16_t *orow = out + r * ldo;
    if constexpr (VEC == 4) {
      for (int64_t c = c0 + 4 * lane; c < c1; c += 128) {
        const int nv = (int)min((int64_t)4, c1 - c);
        unsigned long long w[4] = {0, 0, 0, 0};
        if (nv == 4) {
          in.load4(base + c, w);
        } else {
#pragma unroll
          for (int v = 0; v < 4; ++v)
            if (v < nv) w[v] = in.p[base + c + v];
        }
        long long d[4][kMaxDigits];
#pragma unroll
        for (int v = 0; v < 4; ++v) digits((v < nv && mx != 0) ? In::fixed_word(w[v], e, 7 * nsl) : 0, nsl, d[v]);
#pragma unroll
        for (int sl = 0; sl < kMaxDigits; ++sl) {
          if (sl >= nsl) break;
          uint16_t *o = orow + sl * plane + c;
          if (nv == 4) {
            const unsigned long long bits = (unsigned long long)digit_bits(d[0][sl], e, sl + 1) |
                                            ((unsigned long long)digit_bits(d[1][sl], e, sl + 1) << 16) |
                                            ((unsigned long long)digit_bits(d[2][sl], e, sl + 1) << 32) |
                                            ((unsigned long long)digit_bits(d[3][sl], e, sl + 1) << 48);
            *reinterpret_cast<unsigned long long *>(o) = bits;
          } else {
#pragma unroll
            for (int v = 0; v < 4; ++v)
              if (v < nv) o[v] = digit_bits(d[v][sl], e, sl + 1);
          }
        }
      }
    } else {
      for (int64_t c = c0 + lane; c < c1; c += 32) {
        long long d[kMaxDigits];
        digits(mx == 0 ? 0 : in.fixed(base + c * m.cs, e, 7 * nsl), nsl, d);
#pragma unroll
        for (int sl = 0; sl < kMaxDigits; ++sl) {
          if (sl >= nsl) break;
          orow[sl * plane + c] = digit_bits(d[sl], e, sl + 1);
        }
      }
    }
  }
}

// Single pass of the same slicing for runs of at most 1024 columns and NSL digits: a lane
// holds its (up to) 8 groups of 4 consecutive elements of the run in registers, so every load
// of the run is in flight at once and the input is read from memory once (the two-pass kernel
// above re-reads the run for its digits and keeps one load per lane in flight).  The digits and
// their bf16 bits are those of slice_kernel, element for element: digit t is round(m / 2^s_t) less
// 2^7 round(m / 2^s_(t-1)), in 32 bits from m >> 6, and becomes a float by one addition and one
// multiplication.
constexpr int kRunGroups = 8;  // 8 groups x 4 elements x 32 lanes = 1024 columns per run
template <class In, int NSL>
__global__ void __launch_bounds__(256) slice_run_kernel(const In in, int64_t rows, int64_t cols, const SplitMap m,
                                                        int64_t chunk, uint16_t *__restrict__ out, int64_t ldo,
                                                        int64_t plane) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int64_t nchunks = (cols + chunk - 1) / chunk;
  const int64_t units = rows * nchunks;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < units; u += nwarps) {
    const QuotRem ux = quot_rem(u, nchunks), rx = quot_rem(ux.q, m.rdiv);
    const int64_t r = ux.q, q = ux.r, rq = rx.q, rr = rx.r;
    if (rr >= m.rlim) continue;  // uniform over the warp
    const int64_t base = rq * m.rs1 + rr * m.rs2;
    const int64_t c0 = q * chunk, c1 = min(cols, c0 + chunk);
    unsigned long long w[kRunGroups][4];
    unsigned long long mx = 0;
#pragma unroll
    for (int g = 0; g < kRunGroups; ++g) {
      const int64_t c = c0 + 128 * g + 4 * lane;
#pragma unroll
      for (int v = 0; v < 4; ++v) w[g][v] = 0;
      if (c + 4 <= c1) {
        in.load4(base + c, w[g]);
      } else if (c < c1) {
#pragma unroll
        for (int v = 0; v < 3; ++v)
          if (c + v < c1) w[g][v] = in.p[base + c + v];
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const unsigned long long a = In::abs_word(w[g][v]);
        mx = a > mx ? a : mx;
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = y > mx ? y : mx;
    }
    const int e = In::exponent(mx);
    float sc[NSL];  // digit scales; those below the FP32 normal range flush to 0, as digit_bits
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) {
      const int pe = e - 7 * (sl + 1) + 127;
      sc[sl] = pe >= 1 && pe <= 254 ? __int_as_float(pe << 23) : 0.f;
    }
    uint16_t *orow = out + r * ldo;
#pragma unroll
    for (int g = 0; g < kRunGroups; ++g) {
      const int64_t c = c0 + 128 * g + 4 * lane;
      if (c >= c1) continue;
      uint32_t packed[NSL][2];
#pragma unroll
      for (int v = 0; v < 4; v += 2) {
        // zero-filled words past the run's end slice to zero digits and are not stored
        float f[2][NSL];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const long long m = In::fixed_word(w[g][v + h], e, 7 * NSL);
          const int u = (int)(m >> 6);
          int above = 0;  // m rounded (half up) to the digits before this one
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) {
            const int shift = 7 * (NSL - 1 - sl);
            const int cur = shift > 0 ? (u + (1 << (shift - 7 & 31))) >> (shift - 6 & 31) : (int)m;
            // the digit (|d| <= 128) as a float: 1.5 2^23 + d, less 1.5 2^23
            f[h][sl] = (__int_as_float(0x4B400000 + cur - (above << 7)) - 12582912.f) * sc[sl];
            above = cur;
          }
        }
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl)
          asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed[sl][v / 2]) : "f"(f[1][sl]), "f"(f[0][sl]));
      }
      if (c + 4 <= c1) {
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl)
          *reinterpret_cast<uint2 *>(orow + sl * plane + c) = make_uint2(packed[sl][0], packed[sl][1]);
      } else {
        const int nv = (int)(c1 - c);
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl)
#pragma unroll
          for (int v = 0; v < 3; ++v)
            if (v < nv) orow[sl * plane + c + v] = (uint16_t)(packed[sl][v / 2] >> (16 * (v & 1)));
      }
    }
  }
}

// Digits of float pairs (values hi + lo) for runs of at most 128 NG columns and five digits: a lane
// holds its NG groups of 4 consecutive elements of the run in registers, so every load of the run
// is in flight at once and the input is read once.  The digits come from additions (Ozaki et al.'s
// extraction: adding and taking back 1.5 2^23 units of a digit rounds to it): digit t of r in
// units of 2^(1 - 7 t) for r = value 2^(1 - e), e the exponent of the run's largest value, three
// from hi and two more after adding lo; two elements per instruction.  Bound: HBM (8 bytes read,
// 10 written per element).  5120 x 32768 pairs in runs of 1024: 868 us with 64-bit integer digits,
// 668 us with 32-bit ones, 428 us; 9000 x 40000 in runs of 320: 2090 us with the registers of 1024
// columns, 946 us.
template <int NG>
__global__ void __launch_bounds__(256) slice_pairs_kernel(const float *x2, int64_t rows, int64_t cols,
                                                          const SplitMap m, int64_t chunk, uint16_t *__restrict__ out,
                                                          int64_t ldo, int64_t plane) {
  pdl_wait();
  constexpr int S = kMaxDigits;
  const int lane = threadIdx.x & 31;
  const int64_t nchunks = (cols + chunk - 1) / chunk;
  const int64_t units = rows * nchunks;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < units; u += nwarps) {
    const QuotRem ux = quot_rem(u, nchunks), rx = quot_rem(ux.q, m.rdiv);
    if (rx.r >= m.rlim) continue;  // uniform over the warp
    const float4 *src = reinterpret_cast<const float4 *>(x2) + (rx.q * m.rs1 + rx.r * m.rs2) / 2;
    const int64_t c0 = ux.r * chunk, c1 = min(cols, c0 + chunk);
    float2 h[NG][2], l[NG][2];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int64_t c = c0 + 128 * g + 4 * lane;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
      if (c + 4 <= c1) {
        a = src[c / 2];
        b = src[c / 2 + 1];
      } else if (c < c1) {
        const float2 *p = reinterpret_cast<const float2 *>(src) + c;
        const float2 y0 = *p;
        a.x = y0.x; a.y = y0.y;
        if (c + 1 < c1) { const float2 y = p[1]; a.z = y.x; a.w = y.y; }
        if (c + 2 < c1) { const float2 y = p[2]; b.x = y.x; b.y = y.y; }
      }
      h[g][0] = make_float2(a.x, a.z); l[g][0] = make_float2(a.y, a.w);
      h[g][1] = make_float2(b.x, b.z); l[g][1] = make_float2(b.y, b.w);
    }
    unsigned mx = 0;
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        // normalised pairs (TwoSum): |lo| <= 2^-24 |hi|
        const float2 s = add2(h[g][v], l[g][v]), bb = sub2(s, h[g][v]);
        l[g][v] = add2(sub2(h[g][v], sub2(s, bb)), sub2(l[g][v], bb));
        h[g][v] = s;
        mx = max(mx, max(__float_as_uint(s.x) & 0x7FFFFFFFu, __float_as_uint(s.y) & 0x7FFFFFFFu));
      }
    mx = __reduce_max_sync(0xffffffffu, mx);
    const int e = min(max((int)(mx >> 23), 1) - 126, 127);  // mx < 2^e; infinities and NaN stay what they are
    const float down = __int_as_float((127 + 1 - e) << 23), up = mx ? __int_as_float((127 + e - 1) << 23) : 0.f;
    const float2 dn2 = make_float2(down, down), up2 = make_float2(up, up);
    uint16_t *orow = out + ux.q * ldo;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int64_t c = c0 + 128 * g + 4 * lane;
      if (c >= c1) continue;
      uint32_t packed[S][2];
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        float2 r = mul2(h[g][v], dn2);
#pragma unroll
        for (int t = 1; t <= S; ++t) {
          if (t == 4) r = add2(r, mul2(l[g][v], dn2));
          const float mg = 12582912.f / (float)(1ull << (7 * t - 1));  // 1.5 2^23 units of 2^(1 - 7 t)
          const float2 mg2 = make_float2(mg, mg);
          const float2 d = sub2(add2(r, mg2), mg2);
          r = sub2(r, d);
          const float2 f = mul2(d, up2);
          asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed[t - 1][v]) : "f"(f.y), "f"(f.x));
        }
      }
      if (c + 4 <= c1) {
#pragma unroll
        for (int t = 0; t < S; ++t)
          *reinterpret_cast<uint2 *>(orow + t * plane + c) = make_uint2(packed[t][0], packed[t][1]);
      } else {
        const int nv = (int)(c1 - c);
#pragma unroll
        for (int t = 0; t < S; ++t)
#pragma unroll
          for (int v = 0; v < 3; ++v)
            if (v < nv) orow[t * plane + c + v] = (uint16_t)(packed[t][v / 2] >> (16 * (v & 1)));
      }
    }
  }
}

__global__ void reduce_group_kernel(const __grid_constant__ ReduceGroup g) {
  pdl_wait();
  const ReduceJob q = g.j[blockIdx.y];
  reduce_range(q.part, q.M, q.N, q.ksplit, q.epi, blockIdx.x * (int64_t)blockDim.x + threadIdx.x,
               (int64_t)gridDim.x * blockDim.x);
}

template <int BN, int BK, class Src>
void launch_src(const Src &src, int64_t ntiles, cudaStream_t s) {
  using C = Cfg<BN, BK>;
  static PerDevice attr;
  attr.run(current_device(), [] {
    VGB_CUDA(cudaFuncSetAttribute(tc_gemm_kernel<BN, BK, Src>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
  });
  const int64_t grid = std::min<int64_t>(ntiles, sm_count());
  launch_pdl(tc_gemm_kernel<BN, BK, Src>, (unsigned)grid, kThreads, C::SMEM, s, src);
  VGB_LAUNCH_CHECK();
}

template <class Src>
void launch_any(int bn, int bk, const Src &src, int64_t ntiles, cudaStream_t s) {
  if (bk == 64) {
    switch (bn) {
      case 32: launch_src<32, 64>(src, ntiles, s); break;
      case 64: launch_src<64, 64>(src, ntiles, s); break;
      case 128: launch_src<128, 64>(src, ntiles, s); break;
      default: launch_src<256, 64>(src, ntiles, s); break;
    }
  } else {
    switch (bn) {
      case 32: launch_src<32, 32>(src, ntiles, s); break;
      case 64: launch_src<64, 32>(src, ntiles, s); break;
      case 128: launch_src<128, 32>(src, ntiles, s); break;
      default: launch_src<256, 32>(src, ntiles, s); break;
    }
  }
}

unsigned grid_1d(int64_t n) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), 16LL * 152));
}

}  // namespace

TcMat make_tc_mat(const uint16_t *hi, const uint16_t *lo, int64_t rows, int64_t K, int64_t ld,
                  int box_rows, int bk) {
  TcMat m;
  m.hi = hi;
  m.lo = lo;
  m.rows = rows;
  m.K = K;
  m.ld = ld;
  m.box_rows = box_rows;
  m.bk = bk;
  encode_kmajor(&m.map_hi, hi, rows, K, ld, box_rows, bk);
  encode_kmajor(&m.map_lo, lo, rows, K, ld, box_rows, bk);
  return m;
}

namespace {

// Validated kernel parameters of one problem (tiles == 0 when there is nothing to do).
KParams make_params(const TcMat &A, const TcMat &B, const TcShape &sh, const TcEpilogue &epi, int bn,
                    int *err) {
  VGB_REQUIRE(bn == 32 || bn == 64 || bn == 128 || bn == 256, "tc_gemm: unsupported tile N");
  VGB_REQUIRE(A.box_rows == BM && B.box_rows == bn, "tc_gemm: operand boxes do not match the tile");
  VGB_REQUIRE(A.bk == B.bk, "tc_gemm: operands staged with different K boxes");
  const int BK = A.bk;
  VGB_REQUIRE(sh.K % BK == 0 && A.K >= sh.K && B.K >= sh.K, "tc_gemm: K not padded");
  VGB_REQUIRE(epi.rd >= 1 && epi.cd >= 1, "tc_gemm: bad epilogue map");
  KParams p;
  p.ntiles = 0;
  p.ksplit = 0;
  if (sh.M <= 0 || sh.N <= 0 || sh.nbatch <= 0) return p;
  // rows addressed by the last batch must exist in the operands (TMA fills beyond with zeros,
  // but row coordinates must stay within the int32 range of the descriptor)
  VGB_REQUIRE((sh.nbatch - 1) * sh.a_batch_rows + sh.M <= A.rows + BM, "tc_gemm: A rows");
  VGB_REQUIRE((sh.nbatch - 1) * sh.b_batch_rows + sh.N <= B.rows + bn, "tc_gemm: B rows");
  VGB_REQUIRE(A.rows < (1LL << 31) && B.rows < (1LL << 31), "tc_gemm: too many rows");
  p.M = sh.M; p.N = sh.N; p.K = sh.K;
  p.products = sh.products == 4 ? 4 : 3;
  p.nbatch = sh.nbatch;
  p.a_brows = sh.a_batch_rows;
  p.b_brows = sh.b_batch_rows;
  const int kchunks = (int)(sh.K / BK);
  VGB_REQUIRE(kchunks >= 1, "tc_gemm: K must be positive");
  const int ks = std::max(1, std::min(sh.ksplit, kchunks));
  p.kc_per = (int)ceil_div(kchunks, ks);
  p.ksplit = (int)ceil_div(kchunks, p.kc_per);
  p.kacc = (sh.kacc && p.ksplit > 1) ? 1 : 0;
  VGB_REQUIRE(epi.kind != TcEpilogue::PAIR_F32, "tc_gemm: float-pair output is for slice products");
  VGB_REQUIRE(!p.kacc || (bn <= 64 && epi.kind != TcEpilogue::STORE_F32),
              "tc_gemm: in-CTA K accumulation needs BN <= 64 and a final (split or FP64) epilogue");
  VGB_REQUIRE(p.ksplit == 1 || p.kacc || epi.kind == TcEpilogue::STORE_F32,
              "tc_gemm: K split needs F32 partials or in-CTA accumulation");
  p.mt = ceil_div(sh.M, BM);
  p.nt = ceil_div(sh.N, bn);
  p.ntiles = p.mt * p.nt * p.ksplit * sh.nbatch;
  p.nitems = p.ntiles / p.ksplit;
  p.epi = epi;
  p.err = err;
  return p;
}

}  // namespace

int tc_gemm(const TcMat &A, const TcMat &B, const TcShape &sh, const TcEpilogue &epi, int bn,
            int *err, cudaStream_t s) {
  const KParams p = make_params(A, B, sh, epi, bn, err);
  if (p.ntiles == 0) return 0;
  SingleSrc src;
  src.maps[0] = A.map_hi;
  src.maps[1] = A.map_lo;
  src.maps[2] = B.map_hi;
  src.maps[3] = B.map_lo;
  src.p = p;
  launch_any(bn, A.bk, src, item_count(p), s);
  return p.ksplit;
}

namespace {

// Non-blocking auxiliary streams per device (created once, kept for the process): the launches
// of one grouped product spread over them so that the tail of one launch overlaps the start of
// the next.
std::vector<cudaStream_t> aux_streams(int n) {
  static std::mutex mu;
  static std::map<int, std::vector<cudaStream_t>> pool;
  int dev = 0;
  VGB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  auto &v = pool[dev];
  while ((int)v.size() < n) {
    cudaStream_t st;
    VGB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    v.push_back(st);
  }
  return std::vector<cudaStream_t>(v.begin(), v.begin() + n);
}

}  // namespace

void tc_gemm_grouped(const std::vector<const TcProblem *> &probs, int bn, int *err, cudaStream_t s,
                     int *ksplit_out, int group_max, int nstreams) {
  std::unique_ptr<GroupSrc> src(new GroupSrc());
  const int gmax = std::max(1, std::min(group_max, kGroupMax));
  // more than one launch and several streams: launch l on stream l % nstreams, ordered after the
  // work already on s, and s waits for all of them at the end
  std::vector<cudaStream_t> sts;
  cudaEvent_t fork = nullptr;
  if (nstreams > 1 && (int64_t)probs.size() > gmax) {
    sts = aux_streams(std::min(nstreams, 8));
    VGB_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    VGB_CUDA(cudaEventRecord(fork, s));
    for (cudaStream_t st : sts) VGB_CUDA(cudaStreamWaitEvent(st, fork, 0));
  }
  int launches = 0;
  int bk = 0;
  size_t i = 0;
  while (i < probs.size()) {
    src->n = 0;
    src->err_ptr = err;
    int64_t total = 0;
    for (; i < probs.size() && src->n < gmax; ++i) {
      const TcProblem &q = *probs[i];
      const KParams p = make_params(q.A, q.B, q.shape, q.epi, bn, err);
      if (ksplit_out) ksplit_out[i] = p.ksplit;
      if (p.ntiles == 0) continue;
      VGB_REQUIRE(bk == 0 || bk == q.A.bk, "tc_gemm_grouped: problems with different K boxes");
      bk = q.A.bk;
      const int g = src->n++;
      src->maps[4 * g + 0] = q.A.map_hi;
      src->maps[4 * g + 1] = q.A.map_lo;
      src->maps[4 * g + 2] = q.B.map_hi;
      src->maps[4 * g + 3] = q.B.map_lo;
      src->p[g] = p;
      src->begin[g] = total;
      total += item_count(p);
    }
    if (src->n == 0) continue;
    src->begin[src->n] = total;
    launch_any(bn, bk, *src, total, sts.empty() ? s : sts[launches % sts.size()]);
    ++launches;
  }
  if (!sts.empty()) {
    for (cudaStream_t st : sts) {
      cudaEvent_t join;
      VGB_CUDA(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
      VGB_CUDA(cudaEventRecord(join, st));
      VGB_CUDA(cudaStreamWaitEvent(s, join, 0));
      VGB_CUDA(cudaEventDestroy(join));
    }
    VGB_CUDA(cudaEventDestroy(fork));
  }
}

void split_f64_to_bf16(const double *x, int64_t rows, int64_t cols, const SplitMap &m, uint16_t *hi,
                       uint16_t *lo, int64_t ldo, cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return;
  VGB_REQUIRE(m.rdiv >= 1, "split: bad row map");
  launch_pdl(split_kernel, grid_1d(rows * cols), 256, 0, s, x, rows, cols, m, hi, lo, ldo);
  VGB_LAUNCH_CHECK();
}

namespace {
// blocks per job of a grouped elementwise launch: about 4 waves of 256-thread blocks in total
unsigned group_blocks(int64_t max_elems, int njobs) {
  const int64_t want = ceil_div(max_elems, 256);
  const int64_t cap = std::max<int64_t>(1, (4LL * 8 * sm_count()) / std::max(1, njobs));
  return (unsigned)std::max<int64_t>(1, std::min(want, std::max<int64_t>(cap, 4)));
}
}  // namespace

void split_grouped(const std::vector<SplitJob> &jobs, cudaStream_t s) {
  std::unique_ptr<SplitGroup> g(new SplitGroup());
  size_t i = 0;
  while (i < jobs.size()) {
    g->n = 0;
    int64_t mx = 0;
    for (; i < jobs.size() && g->n < kJobsMax; ++i) {
      if (jobs[i].rows <= 0 || jobs[i].cols <= 0) continue;
      VGB_REQUIRE(jobs[i].map.rdiv >= 1, "split: bad row map");
      g->j[g->n++] = jobs[i];
      mx = std::max(mx, jobs[i].rows * jobs[i].cols);
    }
    if (g->n == 0) continue;
    launch_pdl(split_group_kernel, dim3(group_blocks(mx, g->n), (unsigned)g->n), 256, 0, s, *g);
    VGB_LAUNCH_CHECK();
  }
}

void reduce_grouped(const std::vector<ReduceJob> &jobs, cudaStream_t s) {
  std::unique_ptr<ReduceGroup> g(new ReduceGroup());
  size_t i = 0;
  while (i < jobs.size()) {
    g->n = 0;
    int64_t mx = 0;
    for (; i < jobs.size() && g->n < kJobsMax; ++i) {
      if (jobs[i].M <= 0 || jobs[i].N <= 0 || jobs[i].ksplit <= 0) continue;
      g->j[g->n++] = jobs[i];
      mx = std::max(mx, jobs[i].M * jobs[i].N);
    }
    if (g->n == 0) continue;
    launch_pdl(reduce_group_kernel, dim3(group_blocks(mx, g->n), (unsigned)g->n), 256, 0, s, *g);
    VGB_LAUNCH_CHECK();
  }
}

void slice_f64(const double *x, int64_t rows, int64_t cols, const SplitMap &m, int nslices, int64_t chunk,
               uint16_t *out, int64_t ldo, int64_t plane, cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return;
  VGB_REQUIRE(m.rdiv >= 1 && nslices >= 1 && nslices <= kMaxDigits && chunk >= 1 && chunk <= 1024 &&
                  ldo >= cols && plane >= rows * ldo,
              "slice: bad map or sizes");
  const int64_t warps = rows * ceil_div(cols, chunk);
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(warps, 8), 64LL * sm_count()));
  const F64In in{reinterpret_cast<const unsigned long long *>(x)};
  if (m.cs == 1 && chunk % 4 == 0 && m.rs1 % 4 == 0 && m.rs2 % 4 == 0 && ldo % 4 == 0 && plane % 4 == 0 &&
      ((uintptr_t)x & 31) == 0 && ((uintptr_t)out & 7) == 0) {
    if (nslices == 5) launch_pdl(slice_run_kernel<F64In, 5>, blocks, 256, 0, s, in, rows, cols, m, chunk, out,
                                 ldo, plane);
    else launch_pdl(slice_kernel<F64In, 4, 0>, blocks, 256, 0, s, in, rows, cols, m, nslices, chunk, out, ldo,
                    plane);
  } else {
    launch_pdl(slice_kernel<F64In, 1, 0>, blocks, 256, 0, s, in, rows, cols, m, nslices, chunk, out, ldo,
               plane);
  }
  VGB_LAUNCH_CHECK();
}

void slice_pairs(const float *x2, int64_t rows, int64_t cols, const SplitMap &m, int nslices, int64_t chunk,
                 uint16_t *out, int64_t ldo, int64_t plane, cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return;
  VGB_REQUIRE(((uintptr_t)x2 & 7) == 0 && m.rdiv >= 1 && nslices >= 1 && nslices <= kMaxDigits && chunk >= 1 &&
                  chunk <= 1024 && ldo >= cols && plane >= rows * ldo,
              "slice: bad map or sizes");
  const int64_t warps = rows * ceil_div(cols, chunk);
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(warps, 8), 64LL * sm_count()));
  const PairIn in{reinterpret_cast<const unsigned long long *>(x2)};
  if (m.cs == 1 && chunk % 4 == 0 && m.rs1 % 4 == 0 && m.rs2 % 4 == 0 && ldo % 4 == 0 && plane % 4 == 0 &&
      ((uintptr_t)x2 & 31) == 0 && ((uintptr_t)out & 7) == 0) {
    if (nslices == 5) {
      const int ng = (int)ceil_div(std::min(chunk, cols), 128);
#define VGB_SLICE(NG) launch_pdl(slice_pairs_kernel<NG>, blocks, 256, 0, s, x2, rows, cols, m, chunk, out, ldo, plane)
      switch (ng) {
        case 1: VGB_SLICE(1); break;
        case 2: VGB_SLICE(2); break;
        case 3: VGB_SLICE(3); break;
        case 4: VGB_SLICE(4); break;
        case 5: VGB_SLICE(5); break;
        case 6: VGB_SLICE(6); break;
        default: VGB_SLICE(8); break;
      }
#undef VGB_SLICE
    } else launch_pdl(slice_kernel<PairIn, 4, 0>, blocks, 256, 0, s, in, rows, cols, m, nslices, chunk, out,
                      ldo, plane);
  } else {
    launch_pdl(slice_kernel<PairIn, 1, 0>, blocks, 256, 0, s, in, rows, cols, m, nslices, chunk, out, ldo,
               plane);
  }
  VGB_LAUNCH_CHECK();
}

void reduce_partials(const float *partial, int64_t M, int64_t N, int ksplit, const TcEpilogue &epi,
                     cudaStream_t s) {
  launch_pdl(reduce_partials_kernel, grid_1d(M * N), 256, 0, s, partial, M, N, ksplit, epi);
  VGB_LAUNCH_CHECK();
}

}  // namespace vgb
