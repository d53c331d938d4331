// Test-only CPU build of csqrt_any (seismicinversion_b200/csrc/kr_math.cuh).
#include "../../seismicinversion_b200/csrc/kr_math.cuh"

extern "C" void emu_csqrt_any(const double* z, int n, double* out) {
  for (int i = 0; i < n; ++i) {
    const kr::cd r = kr::csqrt_any(kr::mk(z[2 * i], z[2 * i + 1]));
    out[2 * i] = r.x;
    out[2 * i + 1] = r.y;
  }
}
