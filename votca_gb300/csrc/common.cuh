// Shared host/device helpers of the GB300 BSE library.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <exception>
#include <stdexcept>
#include <string>
#include <utility>

#include "../../include/votca_gb300_bse.h"
#include "per_device.hpp"

namespace vgb {

// Error carried from the C++ core to the C ABI (mapped to a bse_status code).
struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string &msg) : std::runtime_error(msg), code(c) {}
};

[[noreturn]] inline void fail(int code, const std::string &msg) { throw Error(code, msg); }

// Several checks of which each takes back what it reports: all of them run, and the first error is raised,
// so that none is left for a later call.
struct FirstError {
  std::exception_ptr first;
  template <class F>
  void run(F &&f) {
    try {
      f();
    } catch (...) {
      if (!first) first = std::current_exception();
    }
  }
  void raise() const {
    if (first) std::rethrow_exception(first);
  }
};

inline void cuda_check(cudaError_t e, const char *what, const char *file, int line) {
  if (e != cudaSuccess) {
    int code = (e == cudaErrorMemoryAllocation) ? BSE_ERR_OUT_OF_MEMORY : BSE_ERR_CUDA;
    fail(code, std::string(what) + " failed at " + file + ":" + std::to_string(line) + ": " +
                   cudaGetErrorString(e));
  }
}
#define VGB_CUDA(x) ::vgb::cuda_check((x), #x, __FILE__, __LINE__)
#define VGB_LAUNCH_CHECK() ::vgb::cuda_check(cudaGetLastError(), "kernel launch", __FILE__, __LINE__)
#define VGB_REQUIRE(cond, msg)                                   \
  do {                                                           \
    if (!(cond)) ::vgb::fail(BSE_ERR_ARGUMENT, std::string(msg)); \
  } while (0)

// Stream on which DeviceBuffer allocates and frees on the calling thread (set by
// the C ABI entry points to the handle's stream).  With a stream set, buffers
// use the stream-ordered allocator (cudaMallocAsync / cudaFreeAsync), which does
// not synchronise the device, so independent handles can work concurrently.
cudaStream_t &alloc_stream();
struct AllocStreamScope {
  cudaStream_t saved;
  explicit AllocStreamScope(cudaStream_t s) : saved(alloc_stream()) { alloc_stream() = s; }
  ~AllocStreamScope() { alloc_stream() = saved; }
};
// The pool of such allocations on the calling thread; null: the device's default pool, in which the
// handles keep their freed blocks.
cudaMemPool_t &alloc_pool();
// The pool of calls without a handle, one per device: at most kScratchKeep of it stays reserved between
// them, until trim_pool.
constexpr uint64_t kScratchKeep = 1ull << 30;
cudaMemPool_t scratch_pool();
void *device_alloc(size_t bytes, cudaStream_t &used);
void device_free(void *p, cudaStream_t used);
void trim_pool();  // return the unused blocks of both pools to the driver

// Owning device buffer.
template <typename T>
struct DeviceBuffer {
  T *ptr = nullptr;
  size_t count = 0;
  cudaStream_t stream = nullptr;  // stream of the stream-ordered allocation (null: cudaMalloc)
  DeviceBuffer() = default;
  explicit DeviceBuffer(size_t n) { resize(n); }
  DeviceBuffer(const DeviceBuffer &) = delete;
  DeviceBuffer &operator=(const DeviceBuffer &) = delete;
  DeviceBuffer(DeviceBuffer &&o) noexcept : ptr(o.ptr), count(o.count), stream(o.stream) {
    o.ptr = nullptr;
    o.count = 0;
  }
  DeviceBuffer &operator=(DeviceBuffer &&o) noexcept {
    if (this != &o) {
      release();
      ptr = o.ptr; count = o.count; stream = o.stream;
      o.ptr = nullptr; o.count = 0;
    }
    return *this;
  }
  ~DeviceBuffer() { release(); }
  void resize(size_t n) {
    if (n <= count && ptr) return;
    release();
    if (n == 0) return;
    ptr = (T *)device_alloc(n * sizeof(T), stream);
    count = n;
  }
  void release() {
    if (ptr) device_free(ptr, stream);
    ptr = nullptr;
    count = 0;
  }
  T *get() const { return ptr; }
  size_t bytes() const { return count * sizeof(T); }
};

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

inline int current_device() {
  int dev = 0;
  VGB_CUDA(cudaGetDevice(&dev));
  return dev;
}
// Number of SMs of the current device (152 on GB300).
int sm_count();

// Measured FP64 FMA throughput of the current device in TFLOP/s.
double probe_fp64_tflops();

// Screening (screening.cu)
void rpa_epsilon(const bse_mmn_desc &desc, const double *const *slices, const double *energies,
                 int64_t rpatotal, int64_t homo, int64_t rpamin, int64_t rpamax, double wr, double wi,
                 double eta, double *eps_host, cudaStream_t s);
void cholesky_inverse(int64_t n, const double *a_host, int64_t lda, double *inv_host, int64_t ldi,
                      cudaStream_t s, bool in_place = false);
void positive_inverse(int64_t n, const double *a_host, int64_t lda, double cutoff, double *inv_host,
                      int64_t ldi, cudaStream_t s);
void mmn_multiply_right(const bse_mmn_desc &desc, double *const *slices, const double *U_host,
                        int64_t ldu, cudaStream_t s);

// Mmn producer (threecenter.cu)
void fill_3c_mo(const bse_mmn_desc &desc, double *const *slices, const double *ao3c, int64_t nbf,
                const double *C, int64_t ldc, int64_t nmo, cudaStream_t s);
void transition_dipoles(const double *ao_dip, int64_t nbf, const double *C, int64_t ldc, int64_t nmo,
                        int64_t vmin, int64_t vtotal, int64_t cmin, int64_t ctotal, const double *X,
                        const double *Y, int64_t ldx, int64_t nstates, double prefactor, bool accumulate,
                        double *dip, cudaStream_t s);
void aux_pseudo_inv_sqrt(int64_t n, const double *V, int64_t ldv, double etol, double *out, int64_t ldo,
                         int64_t *removed, cudaStream_t s);
void aux_pseudo_inv_sqrt_gwbse(int64_t n, const double *S, int64_t lds, const double *V, int64_t ldv,
                               double etol, double *out, int64_t ldo, int64_t *removed, cudaStream_t s);

#ifdef __CUDACC__
// Programmatic dependent launch: a kernel launched by launch_pdl is set up while the kernel before it
// in the stream still runs, and waits here, first of all, until that one has completed and its
// writes are visible.  Only kernels that begin with pdl_wait are launched this way, and they read with
// plain loads: the read-only path (__ldg, or a parameter that is const and __restrict__) asks for
// data that stays as it is from the start of the kernel, which lies before the wait.  A chain of
// small dependent kernels: 4.1 us a kernel launched normally, 1.4 us this way.  No kernel lets its
// successor start before its own end (griddepcontrol.launch_dependents): the chain is no faster
// with it, and blocks that wait beside a large product slow it (Hd products of 10 vectors, v32 c256
// Naux 1024: 763 us with it, 712 us without, 738 us with normal launches).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  VGB_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}

// Quotient and remainder of indices, in 32 bits where they fit: a 64-bit division converts through
// the FP64 pipe, where an instruction holds its SM quarter for 64 clocks.
struct QuotRem {
  int64_t q, r;
};
__device__ __forceinline__ QuotRem quot_rem(int64_t a, int64_t b) {
  if (((uint64_t)(a | b) >> 32) == 0) {
    const uint32_t x = (uint32_t)a, d = (uint32_t)b, q = x / d;
    return {(int64_t)q, (int64_t)(x - q * d)};
  }
  return {a / b, a % b};
}
#endif

}  // namespace vgb
