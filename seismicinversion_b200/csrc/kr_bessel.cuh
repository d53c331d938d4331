// The Bessel sum's choices that decide what it reads from the J0 table, compiled for the host too
// so that the CPU tests can walk them.
#pragma once

#include <string.h>

#include "kr_math.cuh"

namespace kr {

// The interval k = floor(x) of the J0 table for 0 <= x < n, and t = x - (k + 1/2), from one
// rounding (no conversions, which are slow for 64 bits; an integer x may take either neighbour).
// Below zero k is negative: only rising and falling tiles, whose x are not, call this without fabs.
KR_HD int j0_interval(double x, int n, double& t) {
  constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
  const double w = x - 0.5;
  const double z = w + kRound;
  t = w - (z - kRound);
#ifdef __CUDA_ARCH__
  const int k = __double2loint(z);
#else
  long long bits;
  memcpy(&bits, &z, sizeof bits);
  const int k = (int)bits;
#endif
  return k < n ? k : n - 1;
}

// Whether a tile's arguments x_j = omega r p_j rise from a first one that is not negative, so that
// its branches need no fabs: slownesses on an ascending progression that starts at or above zero,
// and omega r in the range where the tile's factors are finite (`regular`, never negative).
// Slownesses that rise through zero or end below it are summed term by term.  A falling tile counts
// as the rising one that starts at its last slowness, with the step's magnitude.
KR_HD bool rising_tile(bool on_line, double step, double p_first, bool regular) {
  return on_line && step > 0.0 && p_first >= 0.0 && regular;
}

}  // namespace kr
