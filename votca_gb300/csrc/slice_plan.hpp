// Host-side split of a slice product's K runs over CTAs (slice_gemm.cu).
#pragma once

#include <algorithm>
#include <cstdint>

namespace vgb {

constexpr int kSliceTileM = 128, kSliceStageK = 32;
constexpr int kSliceDrain = 16;  // stages (512 K elements) whose level sums are exact in FP32

struct SlicePlan {
  int groups = 1;  // work items per tile
  int rpg = 1;     // K runs per item (the last one of a tile may have fewer)
};

// The K runs of a tile go to several CTAs where the tiles alone leave SMs idle in the last wave of
// work items.  Clocks from measurements on a GB300: 1450 (BN 64) or 1220 (BN 32) per stage, 4000
// per item, and the float-pair partials written and read at 2100 bytes per clock.
inline SlicePlan slice_plan(int64_t M, int64_t N, int bn, int runs, int stages_per_run, int sms) {
  const int64_t tiles = ((M + kSliceTileM - 1) / kSliceTileM) * ((N + bn - 1) / bn);
  SlicePlan best;
  double t_best = 1e300;
  for (int g = 1; g <= std::min(runs, 64); ++g) {
    const int rpg = (runs + g - 1) / g, n = (runs + rpg - 1) / rpg;
    const double waves = (double)((tiles * n + sms - 1) / sms);
    const double t = waves * ((double)rpg * stages_per_run * (bn == 64 ? 1450.0 : 1220.0) + 4000.0) +
                     (n > 1 ? 8000.0 + 16.0 * (double)M * (double)N * n / 2100.0 : 0.0);
    if (t < 0.98 * t_best) {
      t_best = t;
      best.groups = n;
      best.rpg = rpg;
    }
    if (tiles * n >= 8LL * sms) break;
  }
  return best;
}

}  // namespace vgb
