// Slice products: FP64-accurate GEMM from 7-bit digit planes on the tensor cores (slice_gemm.cuh).
#include "slice_gemm.cuh"


#include "slice_plan.hpp"
#include "tc_epilogue.cuh"
#include "tc_ptx.cuh"

namespace vgb {

namespace {

constexpr int BM = kSliceTileM;
constexpr int BK = kSliceStageK;  // 64-byte swizzle rows
constexpr int DRAIN = kSliceDrain;
constexpr int A_BYTES = BM * BK * 2;
constexpr int kEpi = 16;  // epilogue warps: four per TMEM lane quarter
constexpr int kGemmThreads = 64 + 32 * kEpi;  // warp 0: TMA, warp 1: MMA + TMEM owner, rest: epilogue

// A stage holds the S planes of A (128 rows) and of B (BN rows) for 32 K elements; one MMA
// multiplies A plane a with stacked B planes into the adjacent accumulators of levels a + b, so the
// pairs of a digit level add up in the tensor core.
template <int BN, int S>
struct Cfg {
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = S * (A_BYTES + B_BYTES);
  static constexpr int STAGES = 204800 / STAGE_BYTES > 8 ? 8 : 204800 / STAGE_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  // Accumulators: the levels [0, H) twice, so that a drain overlaps the next run's MMAs, and, for
  // BN 64, the levels [H, S) once between the two (they are issued last in a stage).
  static constexpr int H = BN == 64 ? (S < 3 ? S : 3) : S;
  static constexpr int L = S - H;
  static constexpr int HW = H * BN;          // columns of one H buffer
  static constexpr int H1 = (H + L) * BN;    // column of the second one
  static constexpr int EC = BN / 4;          // columns of an epilogue thread
  static_assert(H1 + HW <= 512 && SMEM <= 232448, "tile exceeds the SM");
};

struct Args {
  CUtensorMap map_a, map_b;
  int64_t M, N;
  int a_plane, b_plane;     // operand rows between planes
  int run;                  // K stages per digit run
  int nkb, kb_per, groups;  // K stages, stages per item (whole runs), items per tile
  int mt, nitems;
  TcEpilogue epi;
  int *err;
};

struct Item {
  int m, n, g, kb0, n_kb;
};
__device__ __forceinline__ Item item_of(const Args &p, int t) {
  Item c;
  const uint32_t u = (uint32_t)t / (uint32_t)p.groups;
  c.g = (int)((uint32_t)t - u * (uint32_t)p.groups);
  c.n = (int)(u / (uint32_t)p.mt);
  c.m = (int)(u - (uint32_t)c.n * (uint32_t)p.mt);
  c.kb0 = c.g * p.kb_per;
  c.n_kb = min(p.nkb, c.kb0 + p.kb_per) - c.kb0;
  return c;
}

// Position of stage i of an item (a whole number of runs) in its drain interval.
struct Drain {
  int pos = 0;     // stage of the run
  bool first, last;
  __device__ __forceinline__ void step(int run) {
    first = pos % DRAIN == 0;
    last = (pos + 1) % DRAIN == 0 || pos + 1 == run;
    pos = pos + 1 == run ? 0 : pos + 1;
  }
};

// The MMAs of levels [l0, l1) of a stage: A plane a times the stacked B planes of those levels.
template <int BN, int S>
__device__ __forceinline__ void mma_levels(int l0, int l1, uint32_t d, uint64_t a0, uint64_t b0, bool fresh) {
  using C = Cfg<BN, S>;
#pragma unroll
  for (int kk = 0; kk < BK / 16; ++kk) {
#pragma unroll
    for (int a = 0; a < S; ++a) {
      const int bs = l0 > a ? l0 - a : 0, be = l1 - a;  // B planes [bs, be)
      if (be <= bs) continue;
      // at most 256 columns per MMA
      constexpr int W = 256 / BN;
#pragma unroll
      for (int b = bs; b < be; b += W) {
        const int nb = be - b < W ? be - b : W;
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((nb * BN) >> 3) << 17) |
                               ((uint32_t)(BM >> 4) << 24);
        // the first pair of the interval that reaches a level clears it: plane 0 of A for the
        // levels that it reaches, all of them (it is issued first)
        mma_bf16(d + (uint32_t)((a + b - l0) * BN), a0 + (uint64_t)(a * (A_BYTES >> 4) + 2 * kk),
                 b0 + (uint64_t)(b * (C::B_BYTES >> 4) + 2 * kk), idesc, fresh && kk == 0 && a == 0 ? 0u : 1u);
      }
    }
  }
}

// The levels' sums of a thread's columns at TMEM address t into its float pairs.
template <int BN, int W>
__device__ __forceinline__ void add_levels(int n, float (&kh)[W], float (&kl)[W], uint32_t t) {
#pragma unroll
  for (int l = 0; l < n; ++l) {
    uint32_t r[W];
    tmem_ld(t + (uint32_t)(l * BN), r);
    pair_add(kh, kl, r, false);
  }
}

// Persistent kernel, one CTA per SM.  Bound: the L2 to SM feed and shared memory, 120 KB per 64 K
// elements of a 128 x 64 tile: every plane of a stage is loaded once for its S (S + 1) / 2 pairs, and
// the levels of a drain interval are added once.  With one accumulator and epilogue pass per pair,
// and A plane a loaded with the B planes of its pairs (216 KB): 640 x 262144 x 256 1510 us, 1070 us
// here; 5120 x 32 x 32768 460 us, 255 us here (of which 100 us for K runs shared out by waves).
template <int BN, int S>
__global__ void __launch_bounds__(kGemmThreads, 1) slice_gemm_kernel(const __grid_constant__ Args p) {
  pdl_wait();
  using C = Cfg<BN, S>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *full = (uint64_t *)(smem + C::STAGES * C::STAGE_BYTES);
  uint64_t *empty = full + C::STAGES;
  uint64_t *accf = empty + C::STAGES;  // [0], [1]: H buffers complete, [2]: L
  uint64_t *acce = accf + 3;           // drained
  TcControl *ctl = (TcControl *)(acce + 3);
  volatile int *abort_flag = &ctl->abort;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int i = 0; i < C::STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 3; ++i) {
      mbar_init(&accf[i], 1);
      mbar_init(&acce[i], kEpi);
    }
    ctl->init(kWaitUs);
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
      for (int R = blockIdx.x; R < p.nitems; R += gridDim.x) {
        const Item it = item_of(p, R);
        const int ya = it.m * BM, yb = it.n * BN;
        for (int kb = it.kb0; kb < it.kb0 + it.n_kb; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.err, 1)) goto tma_done;
          const uint32_t st = smem_u32(smem + stage * C::STAGE_BYTES);
          mbar_expect_tx(&full[stage], (uint32_t)C::STAGE_BYTES);
#pragma unroll
          for (int t = 0; t < S; ++t) {
            tma_load_2d(st + t * A_BYTES, &p.map_a, &full[stage], kb * BK, ya + t * p.a_plane);
            tma_load_2d(st + S * A_BYTES + t * C::B_BYTES, &p.map_b, &full[stage], kb * BK, yb + t * p.b_plane);
          }
          if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
        }
      }
      for (int j = 0; j < C::STAGES; ++j)  // every stage consumed before the CTA leaves
        if (!mbar_wait(&empty[j], j < stage ? phase : phase ^ 1, abort_flag, p.err, 5)) break;
    tma_done:
      drain_loads(full, C::STAGES, stage, phase);  // passes at once unless a wait gave up
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0, hb = 0;
      uint32_t phase = 0, ph = 0, pl = 0;  // phases of the ring, of the H buffers (per round of two), of L
      for (int R = blockIdx.x; R < p.nitems; R += gridDim.x) {
        const int n = item_of(p, R).n_kb;
        Drain dr;
        for (int i = 0; i < n; ++i) {
          dr.step(p.run);
          if (!mbar_wait(&full[stage], phase, abort_flag, p.err, 3)) goto mma_done;
          if (dr.first && !mbar_wait(&acce[hb], ph ^ 1, abort_flag, p.err, 2)) goto mma_done;
          fence_after();
          const uint32_t st = smem_u32(smem + stage * C::STAGE_BYTES);
          // descriptors are linear in the address (units of 16 bytes): + 2 per 16 K elements
          const uint64_t a0 = sdesc(st, 512, 4), b0 = sdesc(st + S * A_BYTES, 512, 4);
          mma_levels<BN, S>(0, C::H, tmem + (uint32_t)(hb ? C::H1 : 0), a0, b0, dr.first);
          if (dr.last) mma_commit(&accf[hb]);
          if constexpr (C::L > 0) {
            if (dr.first) {
              if (!mbar_wait(&acce[2], pl ^ 1, abort_flag, p.err, 6)) goto mma_done;
              fence_after();
            }
            mma_levels<BN, S>(C::H, S, tmem + (uint32_t)C::HW, a0, b0, dr.first);
            if (dr.last) {
              mma_commit(&accf[2]);
              pl ^= 1;
            }
          }
          mma_commit(&empty[stage]);
          if (dr.last) {
            ph ^= (uint32_t)hb;
            hb ^= 1;
          }
          if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
        }
      }
    mma_done:
      drain_mmas(&ctl->mma_done);  // the epilogue may have given up before the last of them
    }
  } else {
    const int q = warp % 4, part = (warp - 2) / 4;
    const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * C::EC);
    int hb = 0;
    uint32_t ph = 0, pl = 0;
    float kh[C::EC], kl[C::EC];  // the sum over runs and levels, as float pairs
    for (int R = blockIdx.x; R < p.nitems; R += gridDim.x) {
      const Item it = item_of(p, R);
      const TcEpilogue e = p.epi;
      const int64_t row = (int64_t)it.m * BM + q * 32 + lane;
      const QuotRem ix = quot_rem(row, e.rd);
      const bool row_ok = row < p.M && ix.r < e.rlim;
#pragma unroll
      for (int j = 0; j < C::EC; ++j) kh[j] = kl[j] = 0.f;
      Drain dr;
      for (int i = 0; i < it.n_kb; ++i) {
        dr.step(p.run);
        if (!dr.last) continue;
        if (!mbar_wait_warp(&accf[hb], ph, abort_flag, p.err, 4)) goto epi_done;
        fence_after();
        add_levels<BN>(C::H, kh, kl, tl + (uint32_t)(hb ? C::H1 : 0));
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acce[hb]);
        if constexpr (C::L > 0) {
          if (!mbar_wait_warp(&accf[2], pl, abort_flag, p.err, 7)) goto epi_done;
          pl ^= 1;
          fence_after();
          add_levels<BN>(C::L, kh, kl, tl + (uint32_t)C::HW);
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[2]);
        }
        ph ^= (uint32_t)hb;
        hb ^= 1;
      }
      if (row_ok)
        pair_write(kh, kl, e, p.N, (int64_t)it.n * BN + part * C::EC,
                   ix.q * e.ro1 + ix.r * e.ro2 + it.g * e.so);
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

// FP64 sum of element t over the groups' float pairs, the high and the low parts each exactly where
// sum_splits can; N >= groups.
template <int N>
__device__ __forceinline__ double sum_pairs(const float2 *part, int64_t total, int groups) {
  SplitRegs<N> h, l;
#pragma unroll
  for (int g = 0; g < N; ++g) {
    const float2 x = g < groups ? __ldcg(part + g * total) : make_float2(0.f, 0.f);
    h.w[g] = __float_as_uint(x.x);
    l.w[g] = __float_as_uint(x.y);
  }
  return sum_splits(groups, h) + sum_splits(groups, l);
}

// Y = epi(sum over the groups' float pairs), part[g][n][i].
__global__ void reduce_pairs_kernel(const float2 *part, int64_t M, int64_t N, int groups, const TcEpilogue e) {
  pdl_wait();
  const int64_t total = M * N;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const QuotRem tx = quot_rem(t, M);
    const QuotRem ix = quot_rem(tx.r, e.rd), nx = quot_rem(tx.q, e.cd);
    if (ix.r >= e.rlim || nx.r >= e.clim) continue;
    const unsigned *p = reinterpret_cast<const unsigned *>(part + t);
    double sum;
    if (groups <= 4) sum = sum_pairs<4>(part + t, total, groups);
    else if (groups <= 8) sum = sum_pairs<8>(part + t, total, groups);
    else if (groups <= 16) sum = sum_pairs<16>(part + t, total, groups);
    else sum = sum_splits(groups, SplitMem{p, 2 * total}) + sum_splits(groups, SplitMem{p + 1, 2 * total});
    double *y = e.out_f64 + ix.q * e.ro1 + ix.r * e.ro2 + nx.q * e.co1 + nx.r * e.co2;
    const double r = e.alpha * sum;
    *y = (e.beta == 0.0) ? r : fma(e.beta, *y, r);
  }
}

template <int BN, int S>
void launch(const Args &p, cudaStream_t s) {
  using C = Cfg<BN, S>;
  static PerDevice attr;
  attr.run(current_device(), [] {
    VGB_CUDA(cudaFuncSetAttribute(slice_gemm_kernel<BN, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
  });
  launch_pdl(slice_gemm_kernel<BN, S>, (unsigned)std::min(p.nitems, sm_count()), kGemmThreads, C::SMEM, s, p);
  VGB_LAUNCH_CHECK();
}

template <int BN>
void launch_digits(int digits, const Args &p, cudaStream_t s) {
  switch (digits) {
    case 2: launch<BN, 2>(p, s); break;
    case 3: launch<BN, 3>(p, s); break;
    case 4: launch<BN, 4>(p, s); break;
    default: launch<BN, 5>(p, s); break;
  }
}

}  // namespace

void slice_gemm(const SliceMat &A, const SliceMat &B, int64_t M, int64_t N, int64_t K, int64_t chain, int digits,
                const TcEpilogue &fe, DeviceBuffer<double> &gpart, int *err, cudaStream_t s) {
  if (M <= 0 || N <= 0) return;
  VGB_REQUIRE(digits >= 2 && digits <= 5, "slice_gemm: 2 to 5 digits");
  VGB_REQUIRE(chain >= BK && chain <= 1024 && chain % BK == 0 && K > 0 && K % chain == 0, "slice_gemm: bad run");
  VGB_REQUIRE(A.plane >= M && B.plane >= N, "slice_gemm: planes smaller than the problem");
  VGB_REQUIRE(fe.rd >= 1 && fe.cd >= 1, "slice_gemm: bad epilogue map");
  VGB_REQUIRE(fe.kind == TcEpilogue::AXPBY_F64 || fe.kind == TcEpilogue::PAIR_F32, "slice_gemm: bad epilogue");
  VGB_REQUIRE((int64_t)digits * std::max(A.plane, B.plane) < (1LL << 31) && K < (1LL << 31),
              "slice_gemm: planes too large");
  const int bn = N > 32 ? 64 : 32;
  Args p;
  p.M = M;
  p.N = N;
  p.a_plane = (int)A.plane;
  p.b_plane = (int)B.plane;
  p.run = (int)(chain / BK);
  p.nkb = (int)(K / BK);
  SlicePlan plan;
  plan.rpg = p.nkb / p.run;
  if (fe.kind == TcEpilogue::AXPBY_F64)  // float-pair outputs are written by the CTA that owns the tile
    plan = slice_plan(M, N, bn, p.nkb / p.run, p.run, sm_count());
  p.groups = plan.groups;
  p.kb_per = plan.rpg * p.run;
  const int64_t mt = ceil_div(M, BM), items = mt * ceil_div(N, bn) * p.groups;
  VGB_REQUIRE(items < (1LL << 31) - sm_count(), "slice_gemm: too many tiles");
  p.mt = (int)mt;
  p.nitems = (int)items;
  p.epi = fe;
  p.err = err;
  if (p.groups > 1) {  // float-pair partials [group][column][row]
    gpart.resize((size_t)p.groups * M * N);
    p.epi.kind = TcEpilogue::PAIR_F32;
    p.epi.rd = M; p.epi.ro1 = 0; p.epi.ro2 = 1; p.epi.rlim = M;
    p.epi.cd = N; p.epi.co1 = 0; p.epi.co2 = M; p.epi.clim = N;
    p.epi.so = M * N;
    p.epi.out_f32 = reinterpret_cast<float *>(gpart.get());
  }
  encode_kmajor(&p.map_a, A.p, digits * A.plane - A.first, K, A.ld, BM, BK);
  encode_kmajor(&p.map_b, B.p, digits * B.plane - B.first, K, B.ld, bn, BK);
  if (bn == 64) launch_digits<64>(digits, p, s);
  else launch_digits<32>(digits, p, s);
  if (p.groups > 1) {
    launch_pdl(reduce_pairs_kernel, (unsigned)std::min<int64_t>(ceil_div(M * N, 256), 16LL * sm_count()), 256,
               0, s, reinterpret_cast<const float2 *>(gpart.get()), M, N, p.groups, fe);
    VGB_LAUNCH_CHECK();
  }
}

}  // namespace vgb
