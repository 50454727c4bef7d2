// GEMM of matrices given as 7-bit digit planes (slice_f64, slice_pairs): every product of two
// digits is exact, and so is the FP32 sum of a digit level over 512 K elements with one scale.
#pragma once

#include "common.cuh"
#include "tc_gemm.cuh"

namespace vgb {

// Digit planes of an operand, K-major bf16: digit t of row r is row t * plane + r of p (row stride
// ld, 16-byte aligned).  p may start `first` rows into its first plane.
struct SliceMat {
  const uint16_t *p = nullptr;
  int64_t ld = 0, plane = 0, first = 0;
};

// C (M x N) = sum over the pairs a + b < digits of A plane a times B plane b, through fe (AXPBY_F64, or
// PAIR_F32: the sum as float pairs).  chain: the K elements of one digit scale in both operands, at
// most 1024, dividing K.  A digit level a + b accumulates in the tensor core for at most 512 K
// elements of one run: level 4 sums at most 512 (2 2^13 + 3 2^12) < 2^24 units, the others less, so
// the sums are exact; the runs and levels of a CTA are added as float pairs (about 48 bits), the
// sums of CTAs that share a tile's runs in FP64.  gpart: scratch for those.  err: device int, set when a
// bounded wait gives up.
void slice_gemm(const SliceMat &A, const SliceMat &B, int64_t M, int64_t N, int64_t K, int64_t chain, int digits,
                const TcEpilogue &fe, DeviceBuffer<double> &gpart, int *err, cudaStream_t s);

}  // namespace vgb
