// Host-side plan of an FP64 GEMM on digit products (oz_gemm.cu): which batches become rows or
// columns of one large product, tiles, K splits, chunks, and whether it is faster than FMA.
#pragma once

#include <algorithm>
#include <cstdint>
#include <utility>
#include <vector>

#include "fma_plan.hpp"
#include "gemm_desc.hpp"

#ifdef __CUDACC__
#define VGB_HD __host__ __device__ __forceinline__
#else
#define VGB_HD inline
#endif

namespace vgb {

constexpr int kOzDigits = 7;
constexpr int kOzTileM = 128, kOzTileN = 64, kOzStageK = 32;
constexpr int kOzRun = 1024;     // K elements of one digit scale
constexpr int kOzDrain = 8;      // stages between full drains: K splits are multiples of it
constexpr int64_t kOzOne = 1LL << 62;  // a map of one level

// Index r = (q2 * n1 + q1) * n0 + q0 at q2 s2 + q1 s1 + q0 s0.
struct OzMap {
  int64_t n0 = 1, n1 = 1, s0 = 0, s1 = 0, s2 = 0;
  // 32-bit divisions where the index fits (64-bit ones convert through the FP64 pipe)
  VGB_HD int64_t at(int64_t r) const {
    if (r < n0) return r * s0;
    if (r >> 32) {
      const int64_t q0 = r % n0, q = r / n0;
      return (q / n1) * s2 + (q % n1) * s1 + q0 * s0;
    }
    const uint32_t x = (uint32_t)r, d = (uint32_t)n0, q = x / d, q0 = x - q * d;  // n0 <= r
    if (q < n1) return (int64_t)q * s1 + (int64_t)q0 * s0;
    const uint32_t e = (uint32_t)n1, q2 = q / e;
    return (int64_t)q2 * s2 + (int64_t)(q - q2 * e) * s1 + (int64_t)q0 * s0;
  }
};

// C[cbatch(b) + crow(i) + ccol(n)] = beta C + alpha sum_k A[amap(b M + i) + k ka] B[bmap(b N + n) + k kb]
struct OzPlan {
  const double *A = nullptr, *B = nullptr;
  int64_t ka = 1, kb = 1;
  int64_t M = 0, N = 0, nbatch = 1;  // rows and columns per batch
  OzMap amap, bmap, crow, ccol, cbatch;
  int64_t Kp = 0;                    // K padded to whole stages
  int nkb = 0, kb_per = 0, splits = 1;
  int64_t m_chunk = 0, tb_chunk = 1; // rows of A (one batch), or batches, per launch
  bool faster = false;
};

inline int64_t oz_ceil(int64_t a, int64_t b) { return (a + b - 1) / b; }

// false: a form that stays with the FMA kernel (a batch that moves neither operand, sizes beyond
// the 32-bit row coordinates or the scratch budget).
inline bool oz_plan(const GemmDesc &d, int sms, int64_t plane_budget, OzPlan &q) {
  if (d.M < 1 || d.N < 1 || d.K < 1 || d.nb1 < 1 || d.nb2 < 1) return false;
  struct Dim { int64_t n, s, c; };  // count, operand stride, C stride
  // a batch that moves only A is more rows, one that moves only B more columns (the other operand
  // is then shared by the whole product); one that moves both is a batch of products
  std::vector<Dim> ra, rb, ta, tb;  // outer to inner
  const int64_t bn[2] = {d.nb1, d.nb2}, ba[2] = {d.a_b1, d.a_b2}, bb[2] = {d.b_b1, d.b_b2}, bc[2] = {d.c_b1, d.c_b2};
  for (int x = 0; x < 2; ++x) {
    if (bn[x] == 1) continue;
    if (ba[x] != 0 && bb[x] != 0) {
      ta.push_back({bn[x], ba[x], bc[x]});
      tb.push_back({bn[x], bb[x], bc[x]});
    } else if (ba[x] != 0) {
      ra.push_back({bn[x], ba[x], bc[x]});
    } else if (bb[x] != 0) {
      rb.push_back({bn[x], bb[x], bc[x]});
    } else {
      return false;
    }
  }
  ra.push_back({d.M, d.a_rs, d.c_rs});
  rb.push_back({d.N, d.b_cs, d.c_cs});
  auto count = [](const std::vector<Dim> &v) {
    int64_t n = 1;
    for (const Dim &x : v) n *= x.n;
    return n;
  };
  auto map = [](const std::vector<Dim> &v, bool of_c) {
    OzMap m;
    const size_t n = v.size();
    if (n > 0) { m.n0 = v[n - 1].n; m.s0 = of_c ? v[n - 1].c : v[n - 1].s; }
    if (n > 1) { m.n1 = v[n - 2].n; m.s1 = of_c ? v[n - 2].c : v[n - 2].s; }
    if (n > 2) m.s2 = of_c ? v[n - 3].c : v[n - 3].s;
    return m;
  };
  q.A = d.A; q.B = d.B; q.ka = d.a_cs; q.kb = d.b_rs;
  q.M = count(ra); q.N = count(rb); q.nbatch = count(ta);
  // orientation: fewer padded tiles; a warp of the epilogue stores one column's 32 rows, four
  // times the sectors when C is contiguous along the columns
  const double fwd = (double)oz_ceil(q.M, kOzTileM) * oz_ceil(q.N, kOzTileN) * (d.c_rs == 1 ? 1.0 : 1.25);
  const double bwd = (double)oz_ceil(q.N, kOzTileM) * oz_ceil(q.M, kOzTileN) * (d.c_cs == 1 ? 1.0 : 1.25);
  if (bwd < fwd) {
    std::swap(ra, rb);
    std::swap(ta, tb);
    std::swap(q.M, q.N);
    std::swap(q.A, q.B);
    std::swap(q.ka, q.kb);
  }
  std::vector<Dim> fa = ta, fb = tb;
  fa.insert(fa.end(), ra.begin(), ra.end());
  fb.insert(fb.end(), rb.begin(), rb.end());
  q.amap = map(fa, false); q.bmap = map(fb, false);
  q.crow = map(ra, true); q.ccol = map(rb, true); q.cbatch = map(ta, true);
  q.Kp = oz_ceil(d.K, kOzStageK) * kOzStageK;
  if (q.Kp >= (1LL << 31) || q.M >= (1LL << 27) || q.N >= (1LL << 27)) return false;
  const int64_t tiles = oz_ceil(q.M, kOzTileM) * oz_ceil(q.N, kOzTileN) * q.nbatch;
  if (tiles >= (1LL << 24)) return false;  // tile indices (times at most 64 splits) in 32 bits
  q.nkb = (int)(q.Kp / kOzStageK);
  // chunks: equal shares of the batches, or of the row tiles of A, within the budget of planes
  const int64_t plane_row = (int64_t)kOzDigits * q.Kp * 2;
  q.m_chunk = q.M;
  q.tb_chunk = q.nbatch;
  if (q.nbatch > 1) {
    const int64_t fit = std::max<int64_t>(1, plane_budget / (plane_row * std::max(q.M, q.N)));
    q.tb_chunk = oz_ceil(q.nbatch, oz_ceil(q.nbatch, fit));
  } else if (q.M * plane_row > plane_budget) {
    const int64_t mt = oz_ceil(q.M, kOzTileM), fit = std::max<int64_t>(1, plane_budget / plane_row / kOzTileM);
    q.m_chunk = std::min(q.M, oz_ceil(mt, oz_ceil(mt, fit)) * kOzTileM);
  }
  const int64_t most = std::max(q.m_chunk, q.N) * q.tb_chunk;
  if (most * plane_row > 4 * plane_budget || most * kOzDigits >= (1LL << 31)) return false;
  if ((most / 16 + 2) * (q.Kp / 256 + 1) >= (1LL << 31)) return false;  // units of the slicer
  // K splits (whole drain intervals): the fewest waves of work items over the SMs, against the FP64
  // partials they write.  Times in microseconds, from measurements on a GB300: 2400 clocks per
  // stage, 6000 per item.
  const int64_t nchunks = q.nbatch > 1 ? oz_ceil(q.nbatch, q.tb_chunk) : oz_ceil(q.M, q.m_chunk);
  const int64_t ctiles = oz_ceil(q.m_chunk, kOzTileM) * oz_ceil(q.N, kOzTileN) * q.tb_chunk;
  double t_gemm = 1e300;
  for (int s = 1; s <= std::max(1, std::min(64, q.nkb / kOzDrain)); ++s) {
    const int per = s == 1 ? q.nkb : (int)(oz_ceil(oz_ceil(q.nkb, s), kOzDrain) * kOzDrain);
    const int sp = (int)oz_ceil(q.nkb, per);
    const double t = nchunks * (double)oz_ceil(ctiles * sp, sms) * (per * 2400.0 + 6000.0) / 1.9e3 +
                     (sp > 1 ? 5.0 + 16.0 * sp * q.M * q.N * q.nbatch / 4e6 : 0.0);
    if (t < 0.98 * t_gemm) {
      t_gemm = t;
      q.splits = sp;
      q.kb_per = per;
    }
    if (ctiles * sp >= 8LL * sms) break;
  }
  // the slicer: 5e-6 us per element (read once or twice, planes written), and the launches
  const double elems = (double)(q.M + q.N) * q.nbatch * d.K;
  const double t_oz = nchunks * (q.Kp > 256 ? 20.0 : 15.0) + elems * 5.2e-6 + t_gemm;
  q.faster = t_oz < fma_plan(d, sms, 0).time_us;
  return true;
}

}  // namespace vgb
