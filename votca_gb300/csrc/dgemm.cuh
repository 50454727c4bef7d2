// Strided, two-level-batched FP64 GEMM on CUDA cores with deterministic split-K.
//
// GB300 runs FP64 at ~1.2 TFLOP/s (2 DFMA/clk/SM), so every FP64 contraction
// of this library is DFMA-bound long before it is bandwidth-bound: large ones run
// as digit products on the tensor cores (oz_gemm.cuh); for the others the kernel
// needs only enough blocks and resident warps to keep every SM's DFMA pipe busy
// (tiles of 64 x 64 down to 16 x 16, fma_plan.hpp), and arbitrary element strides
// cost nothing that matters.  This lets one interface serve all FP64 contractions
// (the Hd/Hd2/Hx stages and the Davidson projections) by describing the operands
// with strides instead of materialising transposes.
#pragma once

#include "common.cuh"
#include "gemm_desc.hpp"

namespace vgb {

// Scratch owned by the caller (split-K partials; small digit planes, exponents and the error slot of
// the tensor-core path).  Grows on demand.
struct GemmWorkspace {
  DeviceBuffer<double> partial;
  DeviceBuffer<uint16_t> oz_a, oz_b;
  DeviceBuffer<int> oz_int;
  DeviceBuffer<unsigned> arrived;  // finished splits per tile, zero between products
  int64_t plane_budget = 3LL << 29;  // bytes of digit planes per operand and launch
  int wait_us = 2000000;           // after which a wait inside a product gives up
  GemmWorkspace() = default;
  GemmWorkspace(const GemmWorkspace &) = delete;
  GemmWorkspace &operator=(const GemmWorkspace &) = delete;
  ~GemmWorkspace();
  // Page-locked int a kernel sets when a bounded wait gives up.
  int *error_slot();
  // Raises if one did; call after a synchronisation with the products.
  void check();

 private:
  int *slot_ = nullptr;
};

// Launch.  splitk = 0 picks the path (FMA, or exact digit products on the tensor cores for the
// products that are faster there, oz_gemm.cuh) and a split so that the grid covers the GPU;
// splitk = kFmaSplits is the FMA path with that split, whose bits do not depend on the rule.
constexpr int kFmaSplits = -1;
void dgemm(const GemmDesc &d, cudaStream_t stream, GemmWorkspace *ws, int splitk = 0);

// Same kernels with caller-owned split-K scratch of ws_count doubles: the K
// split is reduced until its partials fit (no split when ws is null).  Never
// allocates.
void dgemm_prealloc(const GemmDesc &d, cudaStream_t stream, double *ws, int64_t ws_count);

}  // namespace vgb
