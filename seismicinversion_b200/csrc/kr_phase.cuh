// Frequency grids that are lines: tabulated layer phase factors exp(omega_k c).
//
// The frequency axis is cut into tiles of 128 (tile u holds k = 128 u + t, t < 128).  When
// every frequency of tile u lies on the grid's line omega_k = omega_0 + k delta,
// delta = (omega_{n-1} - omega_0) / (n - 1), to within kUniformTol * max|omega| (rounding of
// an arange-built grid is ~1 ulp), then for each phase exponent c
//     exp(omega_k c) = (hi[u] * mid[t / 16]) * lo[t % 16],
//     lo[j] = exp(j delta c) (j < 16),  mid[m] = exp(16 m delta c) (m < 8),
//     hi[u] = exp(omega_{128 u} c)       (the tile's own first frequency)
// in the forward kernels (kr_sweep.cuh: as squares and products of a layer's two where it tabulates
// three phases); the derivative kernels (kr_adjsum.cuh) keep hi mid as one entry of the same
// rounding.  Each exponential is one direct exp of an exactly formed argument, and a product of
// table reads replaces an exp and a sincos per layer, phase and frequency.  A tile whose frequencies
// leave the line, or whose entries exceed 1e100 in magnitude (so that no product can overflow),
// evaluates its phases directly.
//
// R of kr_reflectivity and of the batch's forward items is the same bit for bit, and so is R of all
// derivative kernels; between the two families it agrees to rounding
// (tests/test_adjoint_from_forward_gpu.py bounds what that does to a gradient).
#pragma once

#include "kr_internal.cuh"

namespace kr {

constexpr int kPhTile = 128;
constexpr int kPhLo = 16;
constexpr int kPhMid = kPhTile / kPhLo;
constexpr int kPhHead = kPhLo + kPhMid;  // lo + mid entries ahead of the hi entries
constexpr double kUniformTol = 2e-15;
constexpr double kPhMaxMag = 1e100;

struct GridLine {
  double2 w0;
  cd d;
  double tol;
};

__device__ __forceinline__ GridLine grid_line(const double2* __restrict__ omega, int n_w) {
  const double2 a = omega[0], b = omega[n_w - 1];
  GridLine g;
  g.w0 = a;
  g.d = n_w > 1 ? mk((b.x - a.x) / (n_w - 1), (b.y - a.y) / (n_w - 1)) : mk(0.0, 0.0);
  g.tol = kUniformTol * fmax(fmax(fabs(a.x), fabs(a.y)), fmax(fabs(b.x), fabs(b.y)));
  return g;
}

}  // namespace kr
