// Complex FP64 arithmetic, layer slownesses, interface scattering coefficients and the
// Kennett 2x2 addition step, shared by every kernel of the library.
//
// Physics follows tmnestor/SeismicInversion, Kennett_Reflectivity/:
//   complex slowness      layer_model.py:15-45
//   vertical slowness     layer_model.py:48-74   (Im(eta) > 0 branch, flip when Im <= 0)
//   solid-solid coeffs    scattering_matrices.py:42-161
//   ocean-bottom coeffs   scattering_matrices.py:164-296
//   Kennett step          kennett_reflectivity.py:227-256
//   PP + free surface     kennett_reflectivity.py:264-326
//
// Storage choices (ours): Rd and Ru are symmetric and Tu = Td^T (reciprocity,
// scattering_matrices.py:150), so an interface is 10 complex coefficients, stored with 11
// derived constants of the Kennett step, which runs in a symmetric adjugate form (one
// reciprocal per step; see kennett_step).
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define KR_HD __host__ __device__ __forceinline__
#else
#define KR_HD inline
#endif

namespace kr {

struct alignas(16) cd {  // 16-byte aligned: one 128-bit load / store per complex value
  double x, y;
};

KR_HD cd mk(double x, double y) { cd r; r.x = x; r.y = y; return r; }
KR_HD cd operator+(cd a, cd b) { return mk(a.x + b.x, a.y + b.y); }
KR_HD cd operator-(cd a, cd b) { return mk(a.x - b.x, a.y - b.y); }
KR_HD cd operator-(cd a) { return mk(-a.x, -a.y); }
KR_HD cd operator*(cd a, cd b) {
  return mk(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
KR_HD cd operator*(double s, cd a) { return mk(s * a.x, s * a.y); }
KR_HD cd operator*(cd a, double s) { return mk(s * a.x, s * a.y); }
KR_HD cd operator+(cd a, double s) { return mk(a.x + s, a.y); }
KR_HD cd operator+(double s, cd a) { return mk(a.x + s, a.y); }
KR_HD cd operator-(double s, cd a) { return mk(s - a.x, -a.y); }
KR_HD cd operator-(cd a, double s) { return mk(a.x - s, a.y); }
KR_HD cd conj(cd a) { return mk(a.x, -a.y); }
// Fused complex multiply-accumulate: s + a b with two FMAs per component (one rounding per
// FMA, no separate product and sum), and a b + c d as one multiply and three FMAs per
// component.  Operand negations are free in an FMA, so s - a b is cmac(s, -a, b).
KR_HD cd cmac(cd s, cd a, cd b) {
  return mk(fma(a.x, b.x, fma(-a.y, b.y, s.x)), fma(a.x, b.y, fma(a.y, b.x, s.y)));
}
KR_HD cd cdot2(cd a, cd b, cd c, cd d) {
  return mk(fma(a.x, b.x, fma(-a.y, b.y, fma(c.x, d.x, -(c.y * d.y)))),
            fma(a.x, b.y, fma(a.y, b.x, fma(c.x, d.y, c.y * d.x))));
}
KR_HD double abs2(cd a) { return fma(a.x, a.x, a.y * a.y); }

// 1/z via the conjugate over |z|^2, with a prescale by 1e-150 or 1e150 so that |z|^2 neither
// overflows nor underflows for the magnitudes met here (down to ~1e-150).
KR_HD cd recip(cd z) {
  double m = fmax(fabs(z.x), fabs(z.y));
  double s = 1.0;
  if (m > 1e150) s = 1e-150; else if (m < 1e-150 && m > 0.0) s = 1e150;
  double zx = z.x * s, zy = z.y * s;
  double inv = 1.0 / fma(zx, zx, zy * zy);
  return mk(zx * inv * s, -zy * inv * s);
}

// 1/z of a step determinant (|z| near 1 in practice).  recip() spends ~20 FP64 instructions,
// most of them on range scaling and the correctly rounded division; here the range is tested
// on the exponent bits of |z|^2 (integer work) and 1/|z|^2 comes from the hardware's
// reciprocal estimate y (relative error e < 2^-19) refined once by the cubically convergent
// iteration y (1 + e + e^2), e = 1 - n y (Householder's method for 1/n: the new error is
// e^3 < 2^-57, then one rounding): 8 FP64 instructions, within 2 ulp of the quotient.
KR_HD cd recip_near(cd z) {
#ifdef __CUDA_ARCH__
  const double n = fma(z.x, z.x, z.y * z.y);
  // 2^-800 <= n < 2^800: neither n nor its estimate is near the ends of the range
  if ((unsigned)(__double2hiint(n) - (223 << 20)) < (unsigned)(1600 << 20)) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(n));
    const double e = fma(-n, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    return mk(z.x * y, -z.y * y);
  }
#endif
  return recip(z);
}
KR_HD cd operator/(cd a, cd b) { return a * recip(b); }
KR_HD cd operator/(cd a, double s) { return mk(a.x / s, a.y / s); }

// Principal square root, branch cut on the negative real axis, sqrt(conj z) = conj sqrt z
// (C99 csqrt semantics, the convention NumPy and torch use).  For slownesses and their products;
// near the ends of the range see csqrt_any.
KR_HD cd csqrt(cd z) {
  if (z.x == 0.0 && z.y == 0.0) return mk(0.0, z.y);
  double t = sqrt(0.5 * (fabs(z.x) + hypot(z.x, z.y)));
  if (z.x >= 0.0) return mk(t, z.y / (2.0 * t));
  return mk(fabs(z.y) / (2.0 * t), copysign(t, z.y));
}

// csqrt of any magnitude, scaled by a power of four near the ends of the range: of a subnormal,
// csqrt's half sum may round to zero and leave y / (2 t) infinite; of a value near the largest it
// may overflow.  For what data decide: the adjoint of an evanescent water phase underflows
// gradually.
KR_HD cd csqrt_any(cd z) {
  const double m = fmax(fabs(z.x), fabs(z.y));
  double s = 1.0, back = 1.0;
  if (m < 0x1p-960) {
    s = 0x1p120;
    back = 0x1p-60;
  } else if (m > 0x1p960) {
    s = 0.25;
    back = 2.0;
  }
  const cd r = csqrt(mk(z.x * s, z.y * s));
  return mk(r.x * back, r.y * back);
}

KR_HD cd cexp_(cd z) {
  double e = exp(z.x);
  double s, c;
#ifdef __CUDA_ARCH__
  sincos(z.y, &s, &c);
#else
  s = sin(z.y);
  c = cos(z.y);
#endif
  return mk(e * c, e * s);
}

// Complex slowness of a layer with velocity v and quality factor Q.  The multiply-add is an
// explicit fma so that every kernel rounds it alike whatever nvcc's contraction decides in
// the surrounding code (kernels that must agree bit for bit all call this).
KR_HD cd complex_slowness(double v, double Q) {
  double q2 = 2.0 * Q;
  double q2sq = q2 * q2;
  double den = fma(q2, q2, 1.0) * v;
  return mk(q2sq / den, q2 / den);
}

// eta = sqrt((s + p)(s - p)) with Im(eta) > 0.
KR_HD cd vertical_slowness(cd s, double p) {
  cd t = (s + p) * (s - p);
  cd e = csqrt(t);
  if (e.y <= 0.0) e = -e;
  return e;
}

KR_HD bool is_half_space(double h) { return !(h < 1e30); }  // +inf, >= 1e30 (and NaN)

// ---------------------------------------------------------------------------------------
// Per-layer quantities for one slowness.
// ---------------------------------------------------------------------------------------
struct LayerP {
  cd eta;    // vertical P slowness
  cd neta;   // vertical S slowness (0 in the ocean)
  cd betac;  // complex S velocity 1/s_s (0 where beta = 0)
  cd ca;     // i * eta * h   (0 for the half-space: phase factor exactly 1)
  cd cb;     // i * neta * h
  double rho;
  double pad;  // 96 bytes: arrays of LayerP are whole 16-byte units (vector copies)
};

// Whether |exp(omega i eta h)| may exceed 1: eta and neta lie in the first quadrant and h >= 0, so
// only for frequencies with a negative real or imaginary part.
KR_HD bool phases_grow(cd w) { return w.x < 0.0 || w.y < 0.0; }

// Phase factors exp(omega * i eta h) and exp(omega * i neta h) of layer l, evaluated directly
// (kernels on uniform frequency grids use a tabulated source with the same a(l) / b(l)).
struct PhaseDirect {
  cd w;
  const LayerP* lay;
  KR_HD cd a(int l) const { return cexp_(w * lay[l].ca); }
  KR_HD cd b(int l) const { return cexp_(w * lay[l].cb); }
  // whether a factor is cheaper to recompute than to keep (a tabulated source: two products)
  KR_HD bool cheap() const { return false; }
  // whether a phase may grow downwards (phases_grow)
  KR_HD bool grows() const { return phases_grow(w); }
};

// Layer table layout (device or host): 6 rows of n_layers doubles:
// alpha, beta, rho, thickness, Q_alpha, Q_beta.
//
// The P and the S half of a layer's terms are independent chains (two divisions, a complex
// root), so a block's prologue gives each its own thread.
KR_HD void layer_terms_p(const double* tab, int n_layers, int l, double p, LayerP& o) {
  const double h = tab[3 * n_layers + l];
  o.eta = vertical_slowness(complex_slowness(tab[l], tab[4 * n_layers + l]), p);
  o.ca = is_half_space(h) ? mk(0.0, 0.0) : mk(-o.eta.y * h, o.eta.x * h);
  o.rho = tab[2 * n_layers + l];
  o.pad = 0.0;
}
KR_HD void layer_terms_s(const double* tab, int n_layers, int l, double p, LayerP& o) {
  const double beta = tab[n_layers + l];
  const double h = tab[3 * n_layers + l];
  const cd ss = beta > 0.0 ? complex_slowness(beta, tab[5 * n_layers + l]) : mk(0.0, 0.0);
  o.betac = (ss.x != 0.0 || ss.y != 0.0) ? recip(ss) : mk(0.0, 0.0);
  o.neta = (l == 0) ? mk(0.0, 0.0) : vertical_slowness(ss, p);
  o.cb = is_half_space(h) ? mk(0.0, 0.0) : mk(-o.neta.y * h, o.neta.x * h);
}
KR_HD LayerP layer_terms(const double* tab, int n_layers, int l, double p) {
  LayerP o;
  layer_terms_p(tab, n_layers, l, p, o);
  layer_terms_s(tab, n_layers, l, p, o);
  return o;
}

// Square roots of a layer that its two interfaces' coefficients share: formed once per layer
// (four complex roots, ~150 instructions each, leave the coefficients' serial chain).
struct LayerRoots {
  cd eta, neta;  // sqrt(eta), sqrt(neta)
};

// ---------------------------------------------------------------------------------------
// Interface coefficients: Rd, Ru symmetric (3 entries each), Td full (Tu = Td^T).
// ---------------------------------------------------------------------------------------
template <class T>
struct IfaceT {
  T rd11, rd12, rd22;
  T ru11, ru12, ru22;
  T td11, td12, td21, td22;
};

// The coefficients plus the per-interface constants of kennett_step: 2 ru12, det Ru, and the
// quadratic forms of Td that give the entries (11, 12, 22) of Td^T X Td for a symmetric X
// from (x11, x12, x22): q[3 i + k] multiplies the k-th entry in output row i.
struct Iface : IfaceT<cd> {
  cd ru12x2, dru;
  cd q[9];
};

// Scalar-generic so that the same code yields values (T = cd) and forward-mode tangents
// (T = a dual number).  rho enters as T so its tangent can be seeded.
template <class T>
KR_HD void solid_solid(double p, T eta1, T neta1, T rho1, T beta1, T eta2, T neta2, T rho2,
                       T beta2, T rteta1, T rtneta1, T rtrho1, T rteta2, T rtneta2, T rtrho2,
                       IfaceT<T>& o) {
  T rtza1 = rteta1 * rtrho1, rtza2 = rteta2 * rtrho2;
  T rtzb1 = rtneta1 * rtrho1, rtzb2 = rtneta2 * rtrho2;
  const double psq = p * p;
  T dmu = rho2 * beta2 * beta2 - rho1 * beta1 * beta1;
  T d = 2.0 * dmu;
  T psqd = psq * d;
  T a = (rho2 - rho1) - psqd;
  T b = rho2 - psqd;
  T c = rho1 + psqd;
  T E = b * eta1 + c * eta2;
  T F = b * neta1 + c * neta2;
  T G = a - d * eta1 * neta2;
  T H = a - d * eta2 * neta1;
  T det = E * F + G * H * psq;
  T idet = recip(det);
  E = E * idet;
  F = F * idet;
  G = G * idet;
  H = H * idet;
  T Qv = (b * eta1 - c * eta2) * F;
  T Rv = (a + d * eta1 * neta2) * H * psq;
  T Sv = (a * b + c * d * eta2 * neta2) * p * idet;
  T Tv = (b * neta1 - c * neta2) * E;
  T Uv = (a + d * eta2 * neta1) * G * psq;
  T Vv = (a * c + b * d * eta1 * neta1) * p * idet;
  const cd m2i = mk(0.0, -2.0);
  o.rd11 = Qv - Rv;
  o.rd12 = m2i * (rteta1 * rtneta1 * Sv);
  o.rd22 = Tv - Uv;
  o.ru11 = -(Qv + Uv);
  o.ru12 = m2i * (rteta2 * rtneta2 * Vv);
  o.ru22 = -(Tv + Rv);
  o.td11 = 2.0 * (rtza1 * rtza2 * F);
  o.td12 = m2i * (rtzb1 * rtza2 * G * p);
  o.td21 = m2i * (rtza1 * rtzb2 * H * p);
  o.td22 = 2.0 * (rtzb1 * rtzb2 * E);
}

template <class T>
KR_HD void ocean_bottom(double p, T eta1, T rho1, T eta2, T neta2, T rho2, T beta2, T rteta1,
                        T rtrho1, T rteta2, T rtneta2, T rtrho2, IfaceT<T>& o) {
  T rtza1 = rtrho1 * rteta1, rtza2 = rtrho2 * rteta2, rtzb2 = rtrho2 * rtneta2;
  const double psq = p * p;
  T d = 2.0 * (rho2 * beta2 * beta2);
  T psqd = psq * d;
  T a = (rho2 - rho1) - psqd;
  T b = rho2 - psqd;
  T c = rho1 + psqd;
  T E = b * eta1 + c * eta2;
  T F = b;
  T G = a - d * eta1 * neta2;
  T H = -(d * eta2);
  T det = E * F + G * H * psq;
  T idet = recip(det);
  E = E * idet;
  F = F * idet;
  G = G * idet;
  H = H * idet;
  T T1 = (b * eta1 - c * eta2) * F;
  T T2 = (a + d * eta1 * neta2) * H * psq;
  T T4 = b * E;
  T T5 = d * eta2 * G * psq;
  T T6 = b * d * eta1 * p * idet;
  const cd mi = mk(0.0, -1.0);
  T zero = 0.0 * rho1;
  o.rd11 = T1 - T2;
  o.rd12 = zero;
  o.rd22 = zero;
  o.ru11 = -(T1 + T5);
  o.ru12 = mi * (2.0 * (rteta2 * rtneta2 * T6));
  o.ru22 = -(T2 + T4);
  o.td11 = 2.0 * (rtza1 * rtza2 * F);
  o.td12 = zero;
  o.td21 = mi * (2.0 * (rtza1 * rtzb2 * H * p));
  o.td22 = zero;
}

template <class T>
KR_HD void solid_solid(double p, T eta1, T neta1, T rho1, T beta1, T eta2, T neta2, T rho2,
                       T beta2, IfaceT<T>& o) {
  solid_solid(p, eta1, neta1, rho1, beta1, eta2, neta2, rho2, beta2, csqrt(eta1), csqrt(neta1),
              csqrt(rho1), csqrt(eta2), csqrt(neta2), csqrt(rho2), o);
}
template <class T>
KR_HD void ocean_bottom(double p, T eta1, T rho1, T eta2, T neta2, T rho2, T beta2,
                        IfaceT<T>& o) {
  ocean_bottom(p, eta1, rho1, eta2, neta2, rho2, beta2, csqrt(eta1), csqrt(rho1), csqrt(eta2),
               csqrt(neta2), csqrt(rho2), o);
}

KR_HD cd to_c(double r) { return mk(r, 0.0); }

// Coefficients of interface `iface` (between layers iface and iface+1) from layer terms and
// their square roots (the root of a real density is real).
KR_HD Iface interface_coeffs(double p, int iface, const LayerP& up, const LayerP& lo,
                             const LayerRoots& rup, const LayerRoots& rlo) {
  Iface o;
  const cd r1 = to_c(sqrt(up.rho)), r2 = to_c(sqrt(lo.rho));
  if (iface == 0)
    ocean_bottom<cd>(p, up.eta, to_c(up.rho), lo.eta, lo.neta, to_c(lo.rho), lo.betac, rup.eta,
                     r1, rlo.eta, rlo.neta, r2, o);
  else
    solid_solid<cd>(p, up.eta, up.neta, to_c(up.rho), up.betac, lo.eta, lo.neta, to_c(lo.rho),
                    lo.betac, rup.eta, rup.neta, r1, rlo.eta, rlo.neta, r2, o);
  const cd t11 = o.td11, t12 = o.td12, t21 = o.td21, t22 = o.td22;
  o.ru12x2 = 2.0 * o.ru12;
  o.dru = cdot2(o.ru11, o.ru22, -o.ru12, o.ru12);
  o.q[0] = t11 * t11;
  o.q[1] = 2.0 * (t11 * t21);
  o.q[2] = t21 * t21;
  o.q[3] = t11 * t12;
  o.q[4] = cdot2(t11, t22, t21, t12);
  o.q[5] = t21 * t22;
  o.q[6] = t12 * t12;
  o.q[7] = 2.0 * (t12 * t22);
  o.q[8] = t22 * t22;
  return o;
}

KR_HD Iface interface_coeffs(double p, int iface, const LayerP& up, const LayerP& lo) {
  return interface_coeffs(p, iface, up, lo, LayerRoots{csqrt(up.eta), csqrt(up.neta)},
                          LayerRoots{csqrt(lo.eta), csqrt(lo.neta)});
}

// ---------------------------------------------------------------------------------------
// One Kennett addition step: RRd <- Rd + Tu MT (I - Ru MT)^-1 Td with MT = E RRd E,
// E = diag(ea, eb) of the layer below the interface (kennett_reflectivity.py:235-256).
//
// Evaluated in a symmetric form (ours).  Rd, Ru and MT are symmetric and Tu = Td^T, so
// X = MT N^-1 (N = I - Ru MT) and RRd are symmetric, and for 2x2 matrices the adjugate is
// linear, adj(I - Ru MT) = I - adj(MT) adj(Ru), which gives
//     X = (MT - det(MT) adj(Ru)) / det N,   det N = 1 - tr(Ru MT) + det(Ru) det(MT),
//     RRd = Rd + Td^T X Td   (three entries, from per-interface quadratic forms of Td).
// The linearised step maps a perturbation dRRd to Td^T N^-T E dRRd E N^-1 Td, a congruence,
// so an antisymmetric part of the rounding never reaches R; the reference's full-matrix
// evaluation carries such a part, and carrying one of its off-diagonals for both positions
// turns it into error (1e-8 at large slowness).  The symmetric form has none by
// construction and avoids forming N's entries, whose products cancel when the interface
// determinants do: on the reference's 5-layer default model, at every 64th slowness of the
// 8192-slowness gather grid (every third frequency), its worst relative error against an
// 80-bit evaluation of the reference's form is 1.7e-10 (no free surface) and 8.1e-11 (free
// surface), against 8.9e-10 and 2.4e-10 for the full-matrix form in double; on 21-layer models
// both stay near 1e-12.  ~120 FP64 operations per step instead of ~190.
// RRd = [[a, b], [c, d]] with c = b.
// ---------------------------------------------------------------------------------------
struct M2 {
  cd a, b, c, d;
};

// X = MT (I - Ru MT)^-1 of the step (entries 11, 12, 22) from MT's entries; returns 1 / det N.
KR_HD cd step_x(cd m11, cd m12, cd m22, const Iface& f, cd& x11, cd& x12, cd& x22) {
  const cd dm = cdot2(m11, m22, -m12, m12);
  const cd one = mk(1.0, 0.0);
  const cd idet = recip_near(
      cmac(cmac(cmac(cmac(one, -f.ru11, m11), -f.ru12x2, m12), -f.ru22, m22), f.dru, dm));
  x11 = cmac(m11, -f.ru22, dm) * idet;
  x12 = cmac(m12, f.ru12, dm) * idet;
  x22 = cmac(m22, -f.ru11, dm) * idet;
  return idet;
}
// The same from the squared and mixed phase factors P = ea^2, Q = eb^2, S = ea eb.
KR_HD void step_x(const M2& r, cd P, cd Q, cd S, const Iface& f, cd& x11, cd& x12, cd& x22) {
  step_x(P * r.a, S * r.b, Q * r.d, f, x11, x12, x22);
}

// The step, which also hands out X: the reverse sweep of the derivatives needs nothing else of
// it (kr_adjoint.cuh).
KR_HD M2 kennett_step_x(const M2& r, cd P, cd Q, cd S, const Iface& f, cd& x11, cd& x12,
                        cd& x22) {
  step_x(r, P, Q, S, f, x11, x12, x22);
  M2 o;
  o.a = cmac(cmac(cmac(f.rd11, f.q[0], x11), f.q[1], x12), f.q[2], x22);
  o.b = cmac(cmac(cmac(f.rd12, f.q[3], x11), f.q[4], x12), f.q[5], x22);
  o.d = cmac(cmac(cmac(f.rd22, f.q[6], x11), f.q[7], x12), f.q[8], x22);
  o.c = o.b;
  return o;
}

KR_HD M2 kennett_step(const M2& r, cd ea, cd eb, const Iface& f) {
  cd x11, x12, x22;
  return kennett_step_x(r, ea * ea, eb * eb, ea * eb, f, x11, x12, x22);
}

// The last (ocean-bottom) step, returning only RRd_00 (that interface's Td has one column, so
// only q[0..2] are non-zero).
KR_HD cd kennett_last_step_pp(const M2& r, cd P, cd Q, cd S, const Iface& f) {
  cd x11, x12, x22;
  step_x(r, P, Q, S, f, x11, x12, x22);
  return cmac(cmac(cmac(f.rd11, f.q[0], x11), f.q[1], x12), f.q[2], x22);
}

// PP reflectivity at the surface from RRd_PP below the ocean and the squared ocean phase, or
// the ocean phase e0 itself.
KR_HD cd pp_surface2(cd rpp, cd e0e0, bool free_surface) {
  cd y = e0e0 * rpp;
  if (!free_surface) return y;
  return y * recip(1.0 + y);
}
KR_HD cd pp_surface(cd rpp, cd e0, bool free_surface) {
  return pp_surface2(rpp, e0 * e0, free_surface);
}

}  // namespace kr
