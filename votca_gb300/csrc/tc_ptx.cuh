// PTX wrappers of the 5th-generation tensor-core kernels (mbarrier, TMA, tcgen05, TMEM loads) and
// the tensor-map encoder, shared by tc_gemm.cu and oz_gemm.cu.
#pragma once

#include <cuda.h>

#include <mutex>

#include "common.cuh"

namespace vgb {

constexpr int kWaitUs = 2000000;  // bounded waits: 2 s

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// What follows the barriers of a kernel in shared memory.
struct alignas(8) TcControl {
  uint32_t tmem;            // base of the TMEM allocation
  int abort, wait_us;       // set when a wait gave up; the limit of the waits
  uint64_t mma_done;        // barrier of drain_mmas
  __device__ void init(int limit_us) {
    abort = 0;
    wait_us = limit_us;
    mbar_init(&mma_done, 1);
  }
};
static_assert(sizeof(TcControl) == 24, "abort and wait_us are read as an array of two");
// Bounded wait: gives up after abort_flag[1] microseconds (at once for 0) or when another role aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                          int *err, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = now_ns(), limit = 1000ull * (uint64_t)abort_flag[1];
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255) == 0 || limit == 0) {
      if (*abort_flag) return false;
      if (now_ns() - t0 > limit || limit == 0) {
        *abort_flag = 1;
        atomicExch(err, code);
        return false;
      }
    }
  }
}
// The same for a warp that goes on together: TMEM loads need all of its lanes.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *err,
                                               int code) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, err, code));
}
// A role's wait for what it has in flight itself, before the CTA may leave: not cut short by an abort.
__device__ __forceinline__ void mbar_wait_own(uint64_t *bar, uint32_t parity) {
  const uint64_t t0 = now_ns();
  while (!mbar_try_wait(bar, parity) && now_ns() - t0 <= 1000ull * kWaitUs) {}
}
// The loads of a ring of stages, of which `stage` is the next to fill in the round with parity phase (a
// barrier that was never filled passes).
__device__ __forceinline__ void drain_loads(uint64_t *full, int stages, int stage, uint32_t phase) {
  for (int j = 0; j < stages; ++j) mbar_wait_own(&full[j], j < stage ? phase : phase ^ 1);
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint64_t *bar,
                                            int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3}], [%4];" ::"r"(dst),
      "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Swizzled K-major shared-memory matrix descriptor (8-row core groups sbo bytes apart).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t sbo, uint64_t layout) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)(16 >> 4) << 16;  // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(sbo >> 4) << 32; // stride byte offset
  d |= (uint64_t)1 << 46;          // descriptor version (tcgen05)
  d |= layout << 61;               // swizzle mode
  return d;
}
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}
// The MMAs that this thread has issued; bar: of its own, unused before.
__device__ __forceinline__ void drain_mmas(uint64_t *bar) {
  mma_commit(bar);
  mbar_wait_own(bar, 0);
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
      "%30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    VGB_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !p) fail(BSE_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    fn = (EncodeTiledFn)p;
  });
  return fn;
}

// Tensor map of a K-major bf16 matrix (rows x K, row stride ld): boxes of box_rows x bk elements,
// 128-byte (bk 64) or 64-byte (bk 32) swizzle, rows past the end read as zeros.
inline void encode_kmajor(CUtensorMap *m, const uint16_t *base, int64_t rows, int64_t K, int64_t ld, int box_rows,
            int bk) {
  VGB_REQUIRE(((uintptr_t)base & 15) == 0, "tc operand base must be 16-byte aligned");
  VGB_REQUIRE(bk == 32 || bk == 64, "tc operand: K box must be 32 or 64");
  VGB_REQUIRE(K % bk == 0 && (ld * 2) % 16 == 0 && ld >= K, "tc operand K/ld not padded");
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * 2)};
  cuuint32_t box[2] = {(cuuint32_t)bk, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_fn()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void *)base, dims, strides, box,
                           estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           bk == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(BSE_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
}

}  // namespace vgb
