// The misfit's exact Hessian by pairs of layers.
//
// Along a ray (ray_step in kr_adjoint.cuh) dR = sum over the parameters of expressions bilinear
// in the rays' 2-vectors, so the second variation needs only the variations of those vectors.
// For a parameter j of layer l, which acts at step l - 1 as the lower layer's (coefficient
// tangents, phase exponent derivatives dl) and at step l as the upper layer's, let, with X, Td,
// Ru, E of step l - 1 and a subscript u for step l,
//     a = dRd g + dTd^T x,   b = dTd g + dRu x + dl z,   c = dl x,       (lower role)
//     au, bu likewise with the upper layer's tangents at step l,
//     q = c + E (au + Td_u^T X_u bu),   dx = X (b + Ru q) + q,   e = b + Ru dx.
// Then (a, b, ... carry the parameter's index; . is the product without conjugation)
//     T g        = a + Td^T dx            T = d(state l - 1) / d theta_j,  J = dR/dtheta = g . T g
//     g^(j)_l-1  = K_l-1 T g              the variation of g_l-1: a changed state changes the
//                                         steps above it, K_0 = 0,
//                                         K_i+1 = E (Ru + Ru X Ru) E + G_i K_i G_i^T,
//     g^(j)_l    = E e + G_l-1 g^(j)_l-1  the variation of the next step's vector,
//     g^(j)_l+1  = E_u (I + Ru_u X_u)(bu + Td_u g^(j)_l),
//     g^(j)_i+1  = G_i g^(j)_i            below: G_i = E (I + Ru X) Td of step i,
// and the second derivatives of R (through Y where R = Y / (1 + Y)), for k in layer m <= l:
//     l = m      2 [b_j . dx_k + q_j . e_k - sum_a dl_ja dl_ka x_a z_a + bu_j . X_u bu_k
//                   + T g_j . K T g_k],
//     l = m + 1  2 T g_j . g^(k)_m + 2 dx_j . bu_k,
//     l > m + 1  2 T g_j . g^(k)_l-1,
// plus, where j and k share an interface (or a phase), its second derivatives times the
// adjoints, whose frequency sums suffice because those derivatives do not depend on omega.
// The misfit's Hessian is the frequency sum of Re[seed d2Y + A_j J_k] with seed = 2 conj(res),
// A = 2 conj(J) + zeta J, zeta = -2 seed (1 + Y) with the free surface and 0 without (the
// curvature of Y / (1 + Y)).
//
// Work per (omega, p): ~1.9k FP64 operations per layer and ~180 per pair of layers, where one
// dual adjoint per direction took ~40k per direction: 21 layers (79 directions) ~70k against
// ~3.4 million.
#pragma once

#include "kr_hvp.cuh"

namespace kr {

KR_HD cd dot2(const Ray& a, const Ray& b) { return cdot2(a.a, b.a, a.b, b.b); }
KR_HD Ray operator+(const Ray& a, const Ray& b) { return Ray{a.a + b.a, a.b + b.b}; }
KR_HD Ray scale(cd s, const Ray& a) { return Ray{s * a.a, s * a.b}; }
KR_HD Ray zero_ray() { return Ray{mk(0.0, 0.0), mk(0.0, 0.0)}; }
// y + M v for a symmetric M (entries a, b, d), and for Td and Td^T
KR_HD Ray sym_mac(const Ray& y, cd a, cd b, cd d, const Ray& v) {
  return Ray{cmac(cmac(y.a, a, v.a), b, v.b), cmac(cmac(y.b, b, v.a), d, v.b)};
}
template <class F>
KR_HD Ray td_mac(const Ray& y, const F& f, const Ray& v) {
  return Ray{cmac(cmac(y.a, f.td11, v.a), f.td12, v.b), cmac(cmac(y.b, f.td21, v.a), f.td22, v.b)};
}
template <class F>
KR_HD Ray tdt_mac(const Ray& y, const F& f, const Ray& v) {
  return Ray{cmac(cmac(y.a, f.td11, v.a), f.td21, v.b), cmac(cmac(y.b, f.td12, v.a), f.td22, v.b)};
}

// The coefficients of an interface that these formulas read.
struct HessIface {
  cd ru11, ru12, ru22, td11, td12, td21, td22;
};

// What the ray sweep leaves of step i (interface i): X, the phases of layer i + 1, g and K.
struct HessStep {
  S3 X;
  cd ea, eb;
  Ray g;
  S3 K;
};

// E (I + Ru X) v of a step.
template <class F>
KR_HD Ray step_down(const S3& X, cd ea, cd eb, const F& f, const Ray& v) {
  const Ray u = sym_mac(v, f.ru11, f.ru12, f.ru22, sym_mac(zero_ray(), X.a, X.b, X.d, v));
  return Ray{ea * u.a, eb * u.b};
}

// K_i+1 from K_i over step i.
KR_HD S3 hess_next_k(const S3& K, const S3& X, cd ea, cd eb, const IfaceT<cd>& f) {
  // columns of E (I + Ru X) Ru E and of G = E (I + Ru X) Td
  const Ray r1 = step_down(X, ea, eb, f, Ray{f.ru11, f.ru12});
  const Ray r2 = step_down(X, ea, eb, f, Ray{f.ru12, f.ru22});
  const Ray g1 = step_down(X, ea, eb, f, Ray{f.td11, f.td21});
  const Ray g2 = step_down(X, ea, eb, f, Ray{f.td12, f.td22});
  // H = G K (columns h1, h2), G K G^T = h1 g1^T + h2 g2^T
  const Ray h1 = Ray{cdot2(g1.a, K.a, g2.a, K.b), cdot2(g1.b, K.a, g2.b, K.b)};
  const Ray h2 = Ray{cdot2(g1.a, K.b, g2.a, K.d), cdot2(g1.b, K.b, g2.b, K.d)};
  return S3{cmac(cdot2(h1.a, g1.a, h2.a, g2.a), ea, r1.a),
            cmac(cdot2(h1.a, g1.b, h2.a, g2.b), eb, r2.a),
            cmac(cdot2(h1.b, g1.b, h2.b, g2.b), eb, r2.b)};
}

// a = dRd g + dTd^T x, b = dTd g + dRu x for tangent column j (`full`: the step has x; the bottom
// interface has only Rd).
KR_HD void tangent_rays(const ScatTan& t, int j, const Ray& g, const Ray& x, bool full, Ray& a,
                        Ray& b) {
  a = sym_mac(zero_ray(), t.t[0][j], t.t[1][j], t.t[2][j], g);
  b = zero_ray();
  if (full) {
    a = Ray{cmac(cmac(a.a, t.t[6][j], x.a), t.t[8][j], x.b),
            cmac(cmac(a.b, t.t[7][j], x.a), t.t[9][j], x.b)};
    b = sym_mac(b, t.t[3][j], t.t[4][j], t.t[5][j], x);
    b = Ray{cmac(cmac(b.a, t.t[6][j], g.a), t.t[7][j], g.b),
            cmac(cmac(b.b, t.t[8][j], g.a), t.t[9][j], g.b)};
  }
}

// A layer at one (omega, p): what the layers above it read (published), and what its own pairs
// need.  Parameters in order alpha, beta, rho, h.
// HessPublic is the plain form; the kernel's publisher writes the same to shared memory.
struct HessPublic {
  Ray w[4];   // 2 seed T g
  cd G[4];    // rows (11, 12, 21, 22) of G of step l
  cd A[4];    // 2 conj(J) + zeta J
  Ray dx[4];  // 2 seed dx
  KR_HD void set_w(int j, const Ray& v) { w[j] = v; }
  KR_HD void set_G(int c, cd v) { G[c] = v; }
  KR_HD void set_A(int j, cd v) { A[j] = v; }
  KR_HD void set_dx(int j, const Ray& v) { dx[j] = v; }
};
struct HessOwn {
  Ray gl[4];   // g^(k) at level l
  Ray gn[4];   // g^(k) at level l + 1
  Ray bu[3];
  cd J[4];
  double s[10];  // the layer's own block (j >= k, row by row): Re[seed d2Y + A_j J_k]
};

// Layer l (1 <= l <= I) of a model of I interfaces: steps lo = l - 1 and up = l with their
// coefficients and tangents (`up` is not read for the half-space, l = I, where only Rd of the
// bottom interface depends on the layer).
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <class Pub, class F>
KR_HD void hess_layer(int l, int I, cd w, cd seed, cd zeta, const HessStep& lo, const HessStep& up,
                      const F& flo, const F& fup, const ScatTan& tlo, const ScatTan& tup,
                      const LayerD& d, Pub& pub, HessOwn& own) {
  const bool low_full = l <= I - 1;  // step l - 1 is a Kennett step, not the bottom interface
  const bool has_up = l <= I - 1, up_full = l <= I - 2;
  const cd zero = mk(0.0, 0.0);
  const cd seed2 = 2.0 * seed;
  Ray x = zero_ray(), z = zero_ray(), xu = zero_ray(), zu;
  if (low_full) ray_step(lo.X, flo, lo.g, x, z);
  if (up_full) ray_step(up.X, fup, up.g, xu, zu);
  const cd xza = x.a * z.a, xzb = x.b * z.b;
  Ray dxs[4], es[4], kts[4], xbu[3];
  cd das[4], dbs[4];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int j = 0; j < 4; ++j) {
    Ray a = zero_ray(), b = zero_ray(), au = zero_ray(), bu = zero_ray();
    if (j < 3) {
      tangent_rays(tlo, 3 + j, lo.g, x, low_full, a, b);
      if (has_up) tangent_rays(tup, j, up.g, xu, up_full, au, bu);
    }
    // dl = omega d(i eta h) / d theta, likewise neta: alpha and h act on the first, beta and h on
    // the second (all zero in the half-space)
    const bool in_a = j == 0 || j == 3, in_b = j == 1 || j == 3;
    cd da = zero, db = zero;
    Ray c = zero_ray();
    if (in_a) {
      da = w * (j == 0 ? d.ca_alpha : d.ca_h);
      c.a = da * x.a;
      b.a = cmac(b.a, da, z.a);
    }
    if (in_b) {
      db = w * (j == 1 ? d.cb_beta : d.cb_h);
      c.b = db * x.b;
      b.b = cmac(b.b, db, z.b);
    }
    Ray q = zero_ray(), dx = zero_ray(), e = zero_ray(), xb = zero_ray();
    if (low_full) {
      Ray ug = au;
      if (up_full && j < 3) {
        xb = sym_mac(zero_ray(), up.X.a, up.X.b, up.X.d, bu);
        ug = tdt_mac(ug, fup, xb);
      }
      q = c;
      if (j < 3) q = Ray{cmac(c.a, lo.ea, ug.a), cmac(c.b, lo.eb, ug.b)};
      dx = sym_mac(q, lo.X.a, lo.X.b, lo.X.d, sym_mac(b, flo.ru11, flo.ru12, flo.ru22, q));
      e = sym_mac(b, flo.ru11, flo.ru12, flo.ru22, dx);
    }
    const Ray tg = low_full ? tdt_mac(a, flo, dx) : a;
    const cd J = dot2(tg, lo.g);
    const cd A = cmac(mk(2.0 * J.x, -2.0 * J.y), zeta, J);
    pub.set_w(j, scale(seed2, tg));
    pub.set_dx(j, scale(seed2, dx));
    pub.set_A(j, A);
    own.J[j] = J;
    const Ray kt = sym_mac(zero_ray(), lo.K.a, lo.K.b, lo.K.d, tg);
    Ray gl = zero_ray();
    if (low_full) {
      gl = step_down(lo.X, lo.ea, lo.eb, flo, td_mac(zero_ray(), flo, kt));
      gl = Ray{cmac(gl.a, lo.ea, e.a), cmac(gl.b, lo.eb, e.b)};
    }
    own.gl[j] = gl;
    if (up_full) {
      own.gn[j] = step_down(up.X, up.ea, up.eb, fup, td_mac(bu, fup, gl));
    } else {
      own.gn[j] = zero_ray();
    }
    if (j < 3) {
      own.bu[j] = bu;
      xbu[j] = xb;
    }
    dxs[j] = dx;
    es[j] = e;
    kts[j] = kt;
    das[j] = da;
    dbs[j] = db;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = 0; k <= j; ++k) {
      cd s = dot2(b, dxs[k]) + dot2(q, es[k]) + dot2(tg, kts[k]);
      if (in_a && (k == 0 || k == 3)) s = cmac(s, -(da * das[k]), xza);
      if (in_b && (k == 1 || k == 3)) s = cmac(s, -(db * dbs[k]), xzb);
      if (j < 3) s = s + dot2(bu, xbu[k]);
      const cd v = seed2 * s;
      const cd u = A * own.J[k];
      own.s[j * (j + 1) / 2 + k] = v.x + u.x;
    }
  }
  // G of step l, column by column: E (I + Ru X) Td e_c
  if (up_full) {
    for (int c = 0; c < 2; ++c) {
      const Ray t = c == 0 ? Ray{fup.td11, fup.td21} : Ray{fup.td12, fup.td22};
      const Ray v = step_down(up.X, up.ea, up.eb, fup, t);
      pub.set_G(c, v.a);
      pub.set_G(2 + c, v.b);
    }
  } else {
    for (int c = 0; c < 4; ++c) pub.set_G(c, zero);
  }
}

KR_HD double re_dot2(const Ray& a, const Ray& b) {  // Re(a . b)
  return fma(a.a.x, b.a.x, fma(-a.a.y, b.a.y, fma(a.b.x, b.b.x, -a.b.y * b.b.y)));
}
KR_HD double re_mac(double s, cd a, cd b) { return fma(a.x, b.x, fma(-a.y, b.y, s)); }

// Entry (j of layer m + 1, k of layer m) and (j of layer l, k of layer m), l > m + 1, with
// g = g^(k) at level l - 1.
KR_HD double hess_adjacent(const Ray& w, const Ray& dx, cd A, const HessOwn& own, int k) {
  double v = re_mac(re_dot2(w, own.gl[k]), A, own.J[k]);
  if (k < 3) v += re_dot2(dx, own.bu[k]);
  return v;
}
KR_HD double hess_far(const Ray& w, cd A, const Ray& g, cd J) {
  return re_mac(re_dot2(w, g), A, J);
}
KR_HD Ray hess_down(const cd G[4], const Ray& g) {
  return Ray{cdot2(G[0], g.a, G[1], g.b), cdot2(G[2], g.a, G[3], g.b)};
}

// Second derivatives of interface i's coefficients against their adjoint sums S[10] (order of
// ScatTan): items 0..20, the pairs (a >= b) of the interface's six parameters, item
// a (a + 1) / 2 + b; and of layer i + 1's phases against S[10], S[11]: items 21..24 = (alpha,
// alpha), (alpha, h), (beta, beta), (beta, h).  d2: of layers i and i + 1.
constexpr int kHessItems = 25;
KR_HD double hess_curvature(const double* tab, int L, int i, double p, const LayerP* lay,
                            const LayerD* dlay, const LayerD2* d2, const cd* S, int item) {
  if (item >= 21) {
    const int l = i + 1;
    const double h = tab[3 * L + l];
    if (is_half_space(h)) return 0.0;
    const cd s = item < 23 ? S[10] : S[11];
    const cd v = item == 21 ? h * d2[1].eta_aa : item == 22 ? dlay[l].eta_alpha
               : item == 23 ? h * d2[1].neta_bb : dlay[l].neta_beta;
    const cd u = s * mk(-v.y, v.x);  // i v
    return u.x;
  }
  int a = 0;
  while ((a + 1) * (a + 2) / 2 <= item) ++a;
  const int b = item - a * (a + 1) / 2;
  double vu[4] = {0.0, 0.0, 0.0, 0.0}, vl[4] = {0.0, 0.0, 0.0, 0.0};
  if (b < 3) vu[b] = 1.0; else vl[b - 3] = 1.0;
  const LayerV up = layer_dot(tab, L, i, lay[i], dlay[i], d2[0], vu);
  const LayerV lo = layer_dot(tab, L, i + 1, lay[i + 1], dlay[i + 1], d2[1], vl);
  cd col[10];
  interface_dot_col(p, i, up, lo, a, nullptr, col);
  double r = 0.0;
  for (int k = 0; k < 10; ++k) r = re_mac(r, S[k], col[k]);
  return r;
}

}  // namespace kr
