// range_variants.h -- the range kernel's variants, and the body that a launch runs with (host only).
#pragma once
#include <stdint.h>

namespace cz {

// jw: steps of a window.  A warp gives its idle lanes new entries once rl of them are idle in runs of at
// least 64 rows, rs in shorter ones.  warps per block: 0, by the launch's rows (range_pick).  6 and 7 fix
// what 0 chooses from.
struct RangeVariant {
  uint32_t jw, rl, rs, warps;
};
constexpr int RANGE_VARIANTS = 8;
constexpr RangeVariant RANGE_VARIANT[RANGE_VARIANTS] = {{13, 4, 10, 0}, {13, 4, 8, 0},  {13, 4, 14, 0},  {13, 2, 12, 0},
                                                        {13, 6, 10, 0}, {12, 4, 10, 0}, {13, 4, 10, 32}, {13, 4, 10, 24}};

// Launches with fewer than 512 rows to a warp run with 24 warps per block, whichever thresholds are
// set: they spend much of their time opening runs and on the exact path's last seeds, and fewer warps
// open fewer.  2^28 seeds at 2^40: 115 us with 32 warps, 103 with 24; 2^30: 163 and 152; 2^32: 285
// and 271; 2^30 at 2^60: 178 and 165.  Long launches need the 32 (2^36: 2.36 and 2.57 ms).
inline RangeVariant range_pick(int variant, unsigned long long rows, uint32_t sm_count) {
  RangeVariant v = RANGE_VARIANT[variant];
  if (v.warps == 0) v.warps = rows < 512ull * 32 * sm_count ? 24 : 32;
  return v;
}

}  // namespace cz
