// The slot of a distance R in a lookup table of 164 quarter-bohr slots (the radial intervals
// of the CO2-Ar sample kernels): slot j covers [j / 4, (j + 1) / 4), the last one everything
// from 40.75 on.  Shared with the host so that it can be checked there.
#pragma once

#if defined(__CUDACC__)
#define HH_INTERVAL_FN __host__ __device__ __forceinline__
#else
#define HH_INTERVAL_FN inline
#endif

namespace hh {
constexpr int R_SLOTS = 164;

// R is |r| (not negative) or a NaN, which takes the last slot: the comparison comes before the
// conversion, because a NaN double converts to INT_MIN on the device (a NaN float to 0), an
// index 2 GB below the table.  The NaN then reaches the dipole and its status test.
template <typename T> HH_INTERVAL_FN int r_slot(T R) {
  return R < T(0.25 * (R_SLOTS - 1)) ? int(R * T(4)) : R_SLOTS - 1;
}
}  // namespace hh
