// FP64 GEMM on the 5th-generation tensor cores: exact products of digit planes.
//
// GB300 runs FP64 at 2 FMA per clock and SM (1.2 TFLOP/s), 1600 times slower than its bf16 tensor
// rate, so an FP64 contraction large enough to fill the chip is cheaper as many exact bf16 products
// (Ozaki, Ogita, Oishi, Rump, Numer. Algorithms 59 (2012) 95-118; Mukunoki, Ozaki, Ogita, Imamura,
// ISC 2020).  Every row of either operand is cut, per run of 1024 K elements, into seven balanced
// base-256 digits (55 bits and sign below the run's largest element) held as bf16 planes; the
// products of planes a and b with a + b <= 7 (34 of 49) are accumulated in FP32, exactly, and the
// level sums are added as float pairs and written as FP64 values.
//
// Accuracy.  The error's 2-norm over the result's is 6e-17 to 2e-16 on Gaussian, graded and six-decade
// inputs, below that of the FMA chain it replaces (2e-16 to 1e-15 on the same inputs), which is why 34
// pairs are kept: the 28 pairs with a + b <= 6 lose to the chain on inputs graded over both operands
// (1.3e-15 and 1.8e-15 against 7.7e-16).  Element by element the bound is K 2^-53 max|a| max|b| of the row
// and the column, where the chain has K 2^-53 sum |a||b|: an element is cut 2^-56 below the largest of
// its run.  In units of the chain's bound, the largest error over the cc products of v30 c220, v8 c64
// and v17 c131 is 0.004 to 0.015 for Gaussian vectors (chain 0.03 to 0.09), 2.8 to 21 for vectors of one
// large and many small elements (0.08 to 0.27), and 220 to 5000 for unit vectors (a chain is exact),
// where a small element of A stands alone.  Operands graded in opposite directions along K lose as many
// bits as they are graded: where the first digits of the two, with the rows scaled to one, nowhere
// meet in a product above 2^-12, the tiles run as FMA.
//
// Measured on a GB300, FMA kernel against this one (L2 flushed between runs): 4096^3 110 ms and
// 2.82 ms (49 TFLOP/s of FP64 results), the Hd stage 1 of eight vectors of v64 c512 and 256
// auxiliary functions 55.1 and 1.76 ms, its stage 2 (K = 32768) 13.8 and 1.17 ms, 1000^3 1.71 and
// 0.08 ms.
#pragma once

#include "dgemm.cuh"

namespace vgb {

// Runs d on the tensor cores when it is large enough and of a form they take (see oz_gemm.cu);
// false: nothing was launched.  Stream-ordered; takes its scratch from ws (grown on demand).
bool oz_dgemm(const GemmDesc &d, cudaStream_t stream, GemmWorkspace *ws);

}  // namespace vgb
