// Tile and K split of the FP64 FMA GEMM (dgemm.cu), and its time.
#pragma once

#include <algorithm>
#include <cstdint>

#include "gemm_desc.hpp"

namespace vgb {

constexpr int kFmaStep = 16;  // K elements per shared-memory step

struct FmaPlan {
  int tm = 64, tn = 64;
  int64_t splits = 1, kchunk = 0;
  double time_us = 0.0;
};

// The K splits of the rule that fixes the chain of every output (splitk = kFmaSplits): counted in
// 64 x 64 tiles whatever the tile, at least 128 elements each.
inline int64_t fma_chain_splits(const GemmDesc &d, int sms) {
  const int64_t tiles = ((d.M + 63) / 64) * ((d.N + 63) / 64) * d.nb1 * d.nb2, target = 3LL * sms;
  if (tiles >= target || d.K <= 4 * kFmaStep) return 1;
  const int64_t s = std::min((target + tiles - 1) / tiles, (d.K + 8 * kFmaStep - 1) / (8 * kFmaStep));
  return std::max<int64_t>(1, std::min<int64_t>(s, 256));
}

// splitk > 0: that many splits; < 0: fma_chain_splits; 0: chosen with the tile.  The FP64 pipe runs
// 2 FMA per clock and SM (0.001 us per 4 of them), so a plan costs what its busiest SM multiplies,
// padding included: the smallest such maximum wins, the larger tile among equals.  60 x 15 x 8192
// (a Davidson projection): 154 us with 64 x 64 tiles, 36 us with 16 x 16 ones (cold cache);
// 256 x 15 x 512: 140 and 17 us.
inline FmaPlan fma_plan(const GemmDesc &d, int sms, int splitk) {
  static const int kTiles[6][2] = {{64, 64}, {64, 32}, {32, 32}, {64, 16}, {32, 16}, {16, 16}};
  const int64_t nb = d.nb1 * d.nb2;
  const int64_t fixed = splitk > 0 ? splitk : splitk < 0 ? fma_chain_splits(d, sms) : 0;
  FmaPlan best;
  best.time_us = 1e300;
  for (const auto &t : kTiles) {
    const int64_t tiles = ((d.M + t[0] - 1) / t[0]) * ((d.N + t[1] - 1) / t[1]) * nb;
    int64_t lo = fixed, hi = fixed;
    if (!fixed) {
      lo = 1;
      hi = tiles >= 2LL * sms ? 1 : std::max<int64_t>(1, std::min<int64_t>(64, d.K / (4 * kFmaStep)));
    }
    for (int64_t s = lo; s <= hi; s = s < 8 ? s + 1 : s + s / 4) {
      const int64_t kc = ((d.K + s - 1) / s + kFmaStep - 1) / kFmaStep * kFmaStep;
      const int64_t sp = (d.K + kc - 1) / kc, blocks = tiles * sp;
      const double per_sm = (double)((blocks + sms - 1) / sms) * t[0] * t[1] * kc;
      // a step costs its block at least a load's latency; partials are written and read
      const double time = 4.0 + std::max(per_sm / 3800.0, 0.7 * kc / kFmaStep) +
                          (sp > 1 ? 2.5 + 16.0 * sp * d.M * d.N * nb / 3e6 : 0.0);
      if (time < 0.97 * best.time_us) {
        best.tm = t[0]; best.tn = t[1];
        best.splits = sp; best.kchunk = kc;
        best.time_us = time;
      }
    }
  }
  return best;
}

}  // namespace vgb
