// case_limits.h -- up to which value and how many look-ups a seed of a cases line may go without its
// exact run (cases_win.cu); compiles for the host as well.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define CZ_HD __host__ __device__ __forceinline__
#else
#define CZ_HD inline
#endif

namespace cz {

constexpr int CP_STEPS = 12;  // most steps of a look-up

// The limits on values are kept in units of 2^(32 + this), below 2^23 units.  A line whose maximum is
// below 256 units runs every seed exactly, and so does a seed that reaches 2^23 units: the unit
// grows with N, so that the largest start of a checkpoint loop, n 1.5^(N - 10) < 2^(1.585 N - 5.8), lies
// a factor of 2^5 below that, up to N = 45, from where on it is 2^48.  With 2^48 for every N, 2000
// lines of N = 36 took 3.28 ms on the device and 1370 larger ones 7.1, so 1.06 and 2.74.  With units of
// 2^41 at N = 45, the lines of the largest starts took 0.41 ms and not 0.24.
CZ_HD uint32_t line_unit(uint32_t maxbits) {
  const uint32_t top = (maxbits * 317u + 199u) / 200u;  // 1.585 N, rounded up
  return top < 55u ? 0u : top < 71u ? top - 55u : 16u;
}

// A line's limits from the keys of its maxima (key_of): the least value that goes to the exact path, in
// units of 2^(32 + unit) (below 2^24; 0: every value), 1/256 of the maximum or 2^23 units, and above it
// the look-ups that a seed may take (at most 200).
CZ_HD uint32_t line_limits(unsigned long long st_key, unsigned long long e_key, uint32_t mbi, uint32_t iter_cap,
                           uint32_t unit) {
  const int bl = (int)(e_key >> 54) - (int)unit;  // of the maximum in units of 2^unit
  const uint32_t hi = bl > 63   ? 1u << 23
                      : bl < 41 ? 0u
                                : (uint32_t)((e_key & ((1ull << 54) - 1)) >> (94 - bl));
  const uint32_t st = (uint32_t)(st_key < (1ull << 24) ? st_key : 1ull << 24);
  int k = st > mbi ? (int)((st - 1u - mbi) / (uint32_t)CP_STEPS) : -1;
  const int cap = (int)(iter_cap < 201u ? iter_cap : 201u) - 1;  // (look-ups are at least the checkpoints)
  k = k < cap ? k : cap;
  return k < 0 ? 0u : hi | ((uint32_t)k << 24);
}

}  // namespace cz
