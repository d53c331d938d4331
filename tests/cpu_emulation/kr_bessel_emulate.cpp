// Test-only CPU walk of the Bessel sum's tiles (seismicinversion_b200/csrc/kr_bessel.cuh): which
// intervals of the J0 table one (omega, offset) of the kernel would read.
#include <math.h>

#include "../../seismicinversion_b200/csrc/kr_bessel.cuh"

using namespace kr;

// range[0], range[1]: the least and largest interval read (n, -1 if none); range[2]: terms of
// rising tiles.  One slice of all n_p slownesses, tiles of 32.
extern "C" void emu_bessel_intervals(const double* p, int n_p, double om, double r, int n,
                                     int* range) {
  range[0] = n;
  range[1] = -1;
  range[2] = 0;
  const double omr = om * r;
  const bool regular = (omr >= 1e-100 && omr <= 1e100) || omr == 0.0;
  const double step = n_p >= 2 ? (p[n_p - 1] - p[0]) / (double)(n_p - 1) : 0.0;
  for (int j0 = 0; j0 < n_p; j0 += 32) {
    const int m = n_p - j0 < 32 ? n_p - j0 : 32;
    bool line = true;
    for (int k = 0; k < m; ++k)
      line = line && fabs(p[j0 + k] - fma((double)(j0 + k), step, p[0])) <= 1e-15 * fabs(p[j0 + k]);
    const bool rising = rising_tile(line, step, p[j0], regular);
    if (rising) range[2] += m;
    for (int k = 0; k < m; ++k) {
      const double x = (om * p[j0 + k]) * r;
      if (!(rising ? x < 25.0 : x < 25.0 && x > -25.0)) continue;
      double t;
      const int i = j0_interval(rising ? x : fabs(x), n, t);
      if (i < range[0]) range[0] = i;
      if (i > range[1]) range[1] = i;
    }
  }
}

// The same with falling tiles as the kernel takes them: rising ones from their other end.
extern "C" void emu_bessel_steady(const double* p, int n_p, double om, double r, int n, int* range) {
  range[0] = n;
  range[1] = -1;
  range[2] = 0;
  const double omr = om * r;
  const bool regular = (omr >= 1e-100 && omr <= 1e100) || omr == 0.0;
  const double step = n_p >= 2 ? (p[n_p - 1] - p[0]) / (double)(n_p - 1) : 0.0;
  for (int j0 = 0; j0 < n_p; j0 += 32) {
    const int m = n_p - j0 < 32 ? n_p - j0 : 32;
    bool line = true;
    for (int k = 0; k < m; ++k)
      line = line && fabs(p[j0 + k] - fma((double)(j0 + k), step, p[0])) <= 1e-15 * fabs(p[j0 + k]);
    const double p_low = p[j0 + (step > 0.0 ? 0 : m - 1)];
    const bool steady = rising_tile(line, fabs(step), p_low, regular);
    if (steady) range[2] += m;
    for (int k = 0; k < m; ++k) {
      const double x = (om * p[j0 + k]) * r;
      if (!(steady ? x < 25.0 : x < 25.0 && x > -25.0)) continue;
      double t;
      const int i = j0_interval(steady ? x : fabs(x), n, t);
      if (i < range[0]) range[0] = i;
      if (i > range[1]) range[1] = i;
    }
  }
}
