// FP64 strided batched GEMM (see dgemm.cuh for the design note).
#include "dgemm.cuh"

#include <mutex>
#include <vector>

#include "fma_plan.hpp"
#include "oz_gemm.cuh"

namespace vgb {

namespace {

constexpr int TK = kFmaStep;
constexpr int THREADS = 256;

struct Grid {
  int64_t mt, nt, nbatch, splits, kchunk;
};

// C = alpha * sum_s p[s mn] + beta * C of one element, in split order (deterministic).
__device__ __forceinline__ void add_splits(const GemmDesc &d, int64_t b1, int64_t b2, int64_t i, int64_t n,
                                           const double *p, int64_t mn, int64_t splits) {
  double acc = 0.0;
#pragma unroll 8
  for (int64_t s = 0; s < splits; ++s) acc += __ldcg(p + s * mn);  // the loads overlap
  double *c = d.C + b1 * d.c_b1 + b2 * d.c_b2 + i * d.c_rs + n * d.c_cs;
  const double v = d.alpha * acc;
  *c = (d.beta == 0.0) ? v : fma(d.beta, *c, v);
}

// TM x TN outputs per 256-thread block, (TM / 16) x (TN / 16) per thread; the next K step's
// operands are in flight while the current one is multiplied.  The FP64 pipe bounds it: a block
// of 64 x 64 x 16 products keeps its SM busy for 32768 clocks (17 us), so small products want many
// small tiles (fma_plan.hpp).  The sum of an output does not depend on the tile: one chain of FMAs
// in K order per split.  The splits of a 16 x 16 tile are added by the block that finishes last
// (arrived: one counter per tile, back at zero afterwards) instead of by a launch of 4 us.
template <int TM, int TN>
__global__ void __launch_bounds__(THREADS)
    dgemm_kernel(const GemmDesc d, const Grid g, double *partial, unsigned *arrived, int a_icontig, int b_lcontig) {
  pdl_wait();
  constexpr int RM = TM / 16, RN = TN / 16;
  __shared__ double As[2][TK][TM + 1];
  __shared__ double Bs[2][TK][TN + 1];

  // flat block index -> (split, batch, n-tile, m-tile)
  const int64_t bid = blockIdx.x;
  QuotRem x = quot_rem(bid, g.mt);
  const int64_t mtile = x.r;
  x = quot_rem(x.q, g.nt);
  const int64_t ntile = x.r;
  x = quot_rem(x.q, g.splits);
  const int64_t s = x.r, batch = x.q;
  x = quot_rem(batch, d.nb2);
  const int64_t b1 = x.q, b2 = x.r;

  const double *A = d.A + b1 * d.a_b1 + b2 * d.a_b2;
  const double *B = d.B + b1 * d.b_b1 + b2 * d.b_b2;

  const int64_t m0 = mtile * TM, n0 = ntile * TN;
  const int64_t kbeg = s * g.kchunk;
  const int64_t kend = min(d.K, kbeg + g.kchunk);

  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  double acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = 0.0;

  double ra[RM], rb[RN];
  auto load = [&](int64_t k0) {
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int e = tid + THREADS * r;
      const int i = a_icontig ? e & (TM - 1) : e >> 4, l = a_icontig ? e / TM : e & (TK - 1);
      const int64_t gi = m0 + i, gl = k0 + l;
      ra[r] = (gi < d.M && gl < kend) ? A[gi * d.a_rs + gl * d.a_cs] : 0.0;
    }
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const int e = tid + THREADS * r;
      const int l = b_lcontig ? e & (TK - 1) : e / TN, n = b_lcontig ? e >> 4 : e & (TN - 1);
      const int64_t gn = n0 + n, gl = k0 + l;
      rb[r] = (gn < d.N && gl < kend) ? B[gl * d.b_rs + gn * d.b_cs] : 0.0;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int e = tid + THREADS * r;
      As[buf][a_icontig ? e / TM : e & (TK - 1)][a_icontig ? e & (TM - 1) : e >> 4] = ra[r];
    }
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      const int e = tid + THREADS * r;
      Bs[buf][b_lcontig ? e & (TK - 1) : e / TN][b_lcontig ? e >> 4 : e & (TN - 1)] = rb[r];
    }
  };

  load(kbeg);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int64_t k0 = kbeg; k0 < kend; k0 += TK) {
    const bool more = k0 + TK < kend;
    if (more) load(k0 + TK);
#pragma unroll
    for (int l = 0; l < TK; ++l) {
      double a[RM], b[RN];
#pragma unroll
      for (int i = 0; i < RM; ++i) a[i] = As[buf][l][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < RN; ++j) b[j] = Bs[buf][l][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    if (more) store(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }

  double *C = g.splits == 1 ? d.C + b1 * d.c_b1 + b2 * d.c_b2
                                         : partial + (batch * g.splits + s) * d.M * d.N;
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int64_t gi = m0 + ty + 16 * i;
    if (gi >= d.M) continue;
#pragma unroll
    for (int j = 0; j < RN; ++j) {
      const int64_t gn = n0 + tx + 16 * j;
      if (gn >= d.N) continue;
      if (g.splits == 1) {
        double *c = C + gi * d.c_rs + gn * d.c_cs;
        const double v = d.alpha * acc[i][j];
        *c = (d.beta == 0.0) ? v : fma(d.beta, *c, v);
      } else {
        C[gi + gn * d.M] = acc[i][j];
      }
    }
  }
  if constexpr (TM * TN > THREADS) return;
  if (g.splits == 1 || !arrived) return;
  // the tile's last block adds its splits
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (tid == 0)
    last = atomicInc(arrived + (batch * g.nt + ntile) * g.mt + mtile, (unsigned)g.splits - 1) == (unsigned)g.splits - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int64_t mn = d.M * d.N;
  const int64_t gi = m0 + tid % TM, gn = n0 + tid / TM;  // lanes along the columns of the partials
  if (gi < d.M && gn < d.N)
    add_splits(d, b1, b2, gi, gn, partial + batch * g.splits * mn + gi + gn * d.M, mn, g.splits);
}

// The same for all outputs in a launch of its own, for callers without counters.
__global__ void splitk_reduce_kernel(const GemmDesc d, const Grid g, const double *partial) {
  pdl_wait();
  const int64_t mn = d.M * d.N;
  const int64_t total = mn * g.nbatch;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const QuotRem tx = quot_rem(t, mn), ex = quot_rem(tx.r, d.M), bx = quot_rem(tx.q, d.nb2);
    add_splits(d, bx.q, bx.r, ex.r, ex.q, partial + tx.q * g.splits * mn + tx.r, mn, g.splits);
  }
}

__global__ void scale_kernel(const GemmDesc d, int64_t nbatch) {
  pdl_wait();
  const int64_t mn = d.M * d.N, total = mn * nbatch;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const QuotRem tx = quot_rem(t, mn), ex = quot_rem(tx.r, d.M);
    const int64_t batch = tx.q, i = ex.r, n = ex.q;
    const QuotRem bx = quot_rem(batch, d.nb2);
    const int64_t b1 = bx.q, b2 = bx.r;
    double *c = d.C + b1 * d.c_b1 + b2 * d.c_b2 + i * d.c_rs + n * d.c_cs;
    *c = (d.beta == 0.0) ? 0.0 : d.beta * *c;
  }
}

template <int TM, int TN>
void launch_tile(const GemmDesc &d, const Grid &g, double *partial, unsigned *arrived, cudaStream_t stream) {
  const int64_t blocks = g.mt * g.nt * g.nbatch * g.splits;
  VGB_REQUIRE(blocks < (1LL << 31), "dgemm: grid too large");
  launch_pdl(dgemm_kernel<TM, TN>, (unsigned)blocks, THREADS, 0, stream, d, g, partial, arrived,
             d.a_rs == 1 ? 1 : 0, d.b_rs == 1 ? 1 : 0);
  VGB_LAUNCH_CHECK();
}

void launch(const GemmDesc &d, const FmaPlan &f, double *partial, GemmWorkspace *ws, cudaStream_t stream) {
  Grid g;
  g.mt = ceil_div(d.M, f.tm);
  g.nt = ceil_div(d.N, f.tn);
  g.nbatch = d.nb1 * d.nb2;
  g.splits = f.splits;
  g.kchunk = f.kchunk;
  unsigned *arrived = nullptr;
  // only the smallest tiles, one output per thread: with two, over 150 splits, the last blocks took
  // 23 us longer, the launch 13 us
  if (ws && f.splits > 1 && f.tm == 16) {
    const int64_t tiles = g.mt * g.nt * g.nbatch;
    if ((int64_t)ws->arrived.count < tiles) {
      ws->arrived.resize((size_t)tiles);
      VGB_CUDA(cudaMemsetAsync(ws->arrived.get(), 0, tiles * sizeof(unsigned), stream));
    }
    arrived = ws->arrived.get();
  }
  if (f.tm == 64) {
    if (f.tn == 64) launch_tile<64, 64>(d, g, partial, arrived, stream);
    else if (f.tn == 32) launch_tile<64, 32>(d, g, partial, arrived, stream);
    else launch_tile<64, 16>(d, g, partial, arrived, stream);
  } else if (f.tm == 32) {
    if (f.tn == 32) launch_tile<32, 32>(d, g, partial, arrived, stream);
    else launch_tile<32, 16>(d, g, partial, arrived, stream);
  } else {
    launch_tile<16, 16>(d, g, partial, arrived, stream);
  }
  if (f.splits > 1 && !arrived) {
    const int64_t total = d.M * d.N * g.nbatch;
    launch_pdl(splitk_reduce_kernel, (unsigned)std::min<int64_t>(ceil_div(total, 256), 8 * sm_count()), 256,
               0, stream, d, g, partial);
    VGB_LAUNCH_CHECK();
  }
}

}  // namespace

cudaStream_t &alloc_stream() {
  static thread_local cudaStream_t s = nullptr;
  return s;
}

namespace {
// Freed blocks stay in the device's default pool instead of being returned to
// the driver at every synchronisation (the Davidson loop synchronises once per
// iteration); bse_op_destroy trims the pool.
void keep_pool_blocks() {
  static PerDevice once;
  const int dev = current_device();
  once.run(dev, [&] {
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
      uint64_t thr = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
  });
}
}  // namespace

cudaMemPool_t &alloc_pool() {
  static thread_local cudaMemPool_t p = nullptr;
  return p;
}

namespace {
std::mutex g_scratch_mu;
cudaMemPool_t g_scratch[64] = {};
}  // namespace

cudaMemPool_t scratch_pool() {
  int dev = 0;
  VGB_CUDA(cudaGetDevice(&dev));
  if (dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (!g_scratch[dev]) {
    cudaMemPoolProps pp = {};
    pp.allocType = cudaMemAllocationTypePinned;
    pp.location.type = cudaMemLocationTypeDevice;
    pp.location.id = dev;
    cudaMemPool_t pool;
    VGB_CUDA(cudaMemPoolCreate(&pool, &pp));
    uint64_t keep = kScratchKeep;
    VGB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    g_scratch[dev] = pool;
  }
  return g_scratch[dev];
}

void *device_alloc(size_t bytes, cudaStream_t &used) {
  used = alloc_stream();
  auto get = [&](void **p) {
    if (!used) return cudaMalloc(p, bytes);
    if (cudaMemPool_t pool = alloc_pool()) return cudaMallocFromPoolAsync(p, bytes, pool, used);
    keep_pool_blocks();
    return cudaMallocAsync(p, bytes, used);
  };
  void *p = nullptr;
  cudaError_t e = get(&p);
  for (int again = 1; e == cudaErrorMemoryAllocation && again >= 0; --again) {
    // the pools' unused blocks may be what is missing, and what was reserved for the attempt that failed
    // (it can be all of the GPU's memory) would be missing elsewhere
    cudaGetLastError();
    trim_pool();
    if (again) e = get(&p);
  }
  VGB_CUDA(e);
  return p;
}

// A stream-ordered block is freed on the stream of the running call, which is
// ordered after every use in this call; uses in earlier calls on other streams
// are complete by the handle's contract.  Outside a stream scope the free waits
// for the device first, as cudaFree does.
void device_free(void *p, cudaStream_t used) {
  if (!used) {
    cudaFree(p);
  } else if (cudaStream_t cur = alloc_stream()) {
    cudaFreeAsync(p, cur);
  } else {
    cudaDeviceSynchronize();  // nothing is in flight: any stream may take the free
    cudaFreeAsync(p, 0);
  }
}

void trim_pool() {
  int dev = 0;
  cudaMemPool_t pool;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (dev < 64 && g_scratch[dev]) cudaMemPoolTrimTo(g_scratch[dev], 0);
}

int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    VGB_CUDA(cudaGetDevice(&dev));
    VGB_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    return v;
  }();
  return n;
}

namespace {

// Error slots of the workspaces: ints of one page-locked allocation that is kept for the process,
// handed out and taken back.
struct SlotPool {
  std::mutex mu;
  std::vector<int *> free;
} g_slots;
constexpr int kSlotPage = 1024;

}  // namespace

int *GemmWorkspace::error_slot() {
  if (slot_) return slot_;
  std::lock_guard<std::mutex> lk(g_slots.mu);
  if (g_slots.free.empty()) {
    int *page = nullptr;
    VGB_CUDA(cudaHostAlloc((void **)&page, kSlotPage * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
    for (int i = 0; i < kSlotPage; ++i) g_slots.free.push_back(page + i);
  }
  slot_ = g_slots.free.back();
  g_slots.free.pop_back();
  *slot_ = 0;
  return slot_;
}

GemmWorkspace::~GemmWorkspace() {
  if (!slot_) return;
  std::lock_guard<std::mutex> lk(g_slots.mu);
  g_slots.free.push_back(slot_);
}

void GemmWorkspace::check() {
  if (!slot_) return;
  const int code = *(volatile int *)slot_;
  if (code == 0) return;
  *slot_ = 0;
  fail(BSE_ERR_TIMEOUT, "tensor-core FP64 GEMM: a bounded pipeline wait gave up (code " + std::to_string(code) + ")");
}

void dgemm(const GemmDesc &d, cudaStream_t stream, GemmWorkspace *ws, int splitk) {
  VGB_REQUIRE(d.M >= 0 && d.N >= 0 && d.K >= 0, "dgemm: negative size");
  const int64_t nbatch = d.nb1 * d.nb2;
  if (d.M == 0 || d.N == 0 || nbatch == 0) return;
  if (splitk == 0 && oz_dgemm(d, stream, ws)) return;
  if (d.K == 0) {  // C = beta * C
    const int64_t total = d.M * d.N * nbatch;
    launch_pdl(scale_kernel, (unsigned)std::min<int64_t>(ceil_div(total, 256), 65535), 256, 0, stream, d,
               nbatch);
    VGB_LAUNCH_CHECK();
    return;
  }
  const FmaPlan f = fma_plan(d, sm_count(), splitk);
  double *partial = nullptr;
  if (f.splits > 1) {
    VGB_REQUIRE(ws != nullptr, "dgemm: split-K needs a workspace");
    ws->partial.resize((size_t)(nbatch * f.splits * d.M * d.N));
    partial = ws->partial.get();
  }
  launch(d, f, partial, ws, stream);
}

void dgemm_prealloc(const GemmDesc &d, cudaStream_t stream, double *ws, int64_t ws_count) {
  VGB_REQUIRE(d.M >= 0 && d.N >= 0 && d.K >= 0, "dgemm: negative size");
  const int64_t nbatch = d.nb1 * d.nb2;
  if (d.M == 0 || d.N == 0 || nbatch == 0) return;
  if (d.K == 0) {
    const int64_t total = d.M * d.N * nbatch;
    launch_pdl(scale_kernel, (unsigned)std::min<int64_t>(ceil_div(total, 256), 65535), 256, 0, stream, d,
               nbatch);
    VGB_LAUNCH_CHECK();
    return;
  }
  int64_t splits = fma_chain_splits(d, sm_count());
  if (!ws) splits = 1;
  else splits = std::max<int64_t>(1, std::min(splits, ws_count / std::max<int64_t>(1, nbatch * d.M * d.N)));
  launch(d, fma_plan(d, sm_count(), (int)splits), ws, nullptr, stream);
}

}  // namespace vgb
