// Epilogue helpers of the tensor-core kernels: bf16 split stores, float-pair sums, sums of partials.
#pragma once

#include <cuda_bf16.h>

#include "tc_gemm.cuh"

namespace vgb {

// v - float(hi) is exact in FP32 (hi is v rounded to 8 significant bits), so
// the split costs no FP64 work in the epilogue.
__device__ __forceinline__ void epi_store(const TcEpilogue &e, int64_t off, float v) {
  if (e.kind == TcEpilogue::SPLIT_BF16) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    const __nv_bfloat16 l = __float2bfloat16_rn(v - __bfloat162float(h));
    e.out_hi[off] = __bfloat16_as_ushort(h);
    e.out_lo[off] = __bfloat16_as_ushort(l);
  } else if (e.kind == TcEpilogue::STORE_F32) {
    e.out_f32[off] = v;
  } else {
    double *y = e.out_f64 + off;
    const double r = e.alpha * (double)v;
    *y = (e.beta == 0.0) ? r : fma(e.beta, *y, r);
  }
}

// Two FP32 operations per instruction, each rounded to nearest.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 x, x, y;\n"
      " mov.b64 {%0, %1}, x;\n}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.f32x2 x, x, y;\n"
      " mov.b64 {%0, %1}, x;\n}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mul.rn.f32x2 x, x, y;\n"
      " mov.b64 {%0, %1}, x;\n}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// The K splits' FP32 sums of a tile are added as an unevaluated pair of floats (Knuth's TwoSum,
// error-free; about 48 significant bits) in kh[j] + kl[j]: no FP64 instruction per split (the
// FP64 pipe of GB300 runs at 2 operations per clock and SM).  The sums of slice
// products are exact, so their result is the exact sum to that precision.
template <int W>
__device__ __forceinline__ void pair_add(float (&kh)[W], float (&kl)[W], const uint32_t (&r)[W], bool first) {
  if (first) {
#pragma unroll
    for (int j = 0; j < W; ++j) {
      kh[j] = __uint_as_float(r[j]);
      kl[j] = 0.f;
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < W; j += 2) {  // two columns per instruction
    const float2 x = make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1]));
    const float2 hi = make_float2(kh[j], kh[j + 1]);
    const float2 sum = add2(hi, x);
    const float2 bb = sub2(sum, hi);
    const float2 lo = add2(make_float2(kl[j], kl[j + 1]), add2(sub2(hi, sub2(sum, bb)), sub2(x, bb)));
    kh[j] = sum.x;
    kh[j + 1] = sum.y;
    kl[j] = lo.x;
    kl[j + 1] = lo.y;
  }
}

// Writes a thread's float-pair sums (columns n0 ..) of row base rbase through the epilogue map.
template <int W>
__device__ __forceinline__ void pair_write(const float (&kh)[W], const float (&kl)[W], const TcEpilogue &e,
                                           int64_t N, int64_t n0,
                                           int64_t rbase) {
  const QuotRem nx = quot_rem(n0, e.cd);
  int64_t n = n0, nq = nx.q, nr = nx.r;
#pragma unroll
  for (int j = 0; j < W; ++j) {
    if (n < N && nr < e.clim) {
      const int64_t off = rbase + nq * e.co1 + nr * e.co2;
      const float hi = kh[j], lo = kl[j];
      if (e.kind == TcEpilogue::PAIR_F32) {
        reinterpret_cast<float2 *>(e.out_f32)[off] = make_float2(hi, lo);
      } else {
        const double val = (double)hi + (double)lo;
        if (e.kind == TcEpilogue::AXPBY_F64) {
          double *y = e.out_f64 + off;
          const double rv = e.alpha * val;
          *y = (e.beta == 0.0) ? rv : fma(e.beta, *y, rv);
        } else {
          epi_store(e, off, (float)val);
        }
      }
    }
    ++n;
    if (++nr == e.cd) { nr = 0; ++nq; }
  }
}

// The FP64 sum of the ksplit floats p[s * stride], in split order.  Every addition is exact while the
// floats' exponents lie within 29 - log2(ksplit) of each other (24-bit mantissas, at most 53 bits
// altogether), so the sum is taken in 64-bit integers then and converted once; otherwise (and with
// infinities or NaN) in FP64.  The same bits either way: a conversion and an addition per float
// hold an SM quarter for 128 clocks a warp.  163840 sums of 32 floats: 41 us in FP64, 22 us; 20480: 9.2 us, 5.2 us.
template <class Load>
__device__ __forceinline__ double sum_splits(int ksplit, const Load &load) {
  int emax = 0, emin = 255;
#pragma unroll(Load::kUnroll)
  for (int s = 0; s < Load::kMax; ++s) {
    if (!Load::kPadded && s >= ksplit) break;
    const unsigned b = load(s) & 0x7FFFFFFFu;
    const int ex = max((int)(b >> 23), 1);  // subnormals as exponent 1 without the hidden bit
    emax = max(emax, b ? ex : 0);
    emin = min(emin, b ? ex : 255);
  }
  if (emax == 0) return 0.0;
  if (emax == 255 || emax - emin > 29 - (32 - __clz(ksplit - 1))) {
    double acc = 0.0;
#pragma unroll(Load::kUnroll)
    for (int s = 0; s < Load::kMax; ++s) {
      if (!Load::kPadded && s >= ksplit) break;
      acc += (double)__uint_as_float(load(s));
    }
    return acc;
  }
  long long a = 0;
#pragma unroll(Load::kUnroll)
  for (int s = 0; s < Load::kMax; ++s) {
    if (!Load::kPadded && s >= ksplit) break;
    const unsigned b = load(s);
    const int ex = (int)(b >> 23) & 0xFF;
    const unsigned m = (b & 0x7FFFFFu) | (ex ? 0x800000u : 0u);
    const long long t = (long long)m << max(max(ex, 1) - emin, 0);  // zeros: m = 0
    a += (int)b < 0 ? -t : t;
  }
  if (a == 0) return 0.0;
  const double v = __ll2double_rn(a);  // exact; units of 2^(emin - 150)
  return __hiloint2double(__double2hiint(v) + ((emin - 150) << 20), __double2loint(v));
}
constexpr int kSplitRegs = 32;
template <int N>
struct SplitRegs {  // up to N splits, the rest zeros, all loads in flight at once
  static constexpr bool kPadded = true;
  static constexpr int kMax = N, kUnroll = N;
  unsigned w[N];
  __device__ __forceinline__ unsigned operator()(int s) const { return w[s]; }
};
struct SplitMem {  // more: read again in each pass
  static constexpr bool kPadded = false;
  static constexpr int kMax = 1 << 30, kUnroll = 8;
  const unsigned *p;
  int64_t stride;
  __device__ __forceinline__ unsigned operator()(int s) const { return __ldcg(p + s * stride); }
};

}  // namespace vgb
