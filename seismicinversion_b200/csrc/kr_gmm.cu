// Global Matrix Method reflectivity with the block-Riccati sweep: an FP64 evaluation of
// R(omega, p) from the layers' eigenvectors and the continuity of displacement and traction,
// without reflection / transmission coefficients, behind the same boundary as kr_reflectivity.
//
// Follows tmnestor/SeismicInversion, GlobalMatrix/:
//   layer eigenvectors     layer_matrix.py:201-258 (E_d, E_u 4x2; ocean e_d, e_u)
//   Riccati sweep          riccati_solver.py:200-283 (E_eff = E_d + E_u diag(ph) Y,
//                          F = [E_u | -E_eff], F X = -E_d diag(ph), Y = X[0:2])
//   ocean extraction       riccati_solver.py:297-330
//   entry point            gmm_torch.py:229-305 (R / (1 + R) with the free surface)
//
// The 4x4 systems do not depend on omega but through Z = diag(ph) Y of the layer below, so they
// are solved once per (slowness, interface): with E = [E_d E_u] of each layer,
//     [diag(ph_k); Y_k] = Q [I; Z_k+1] D,   Q = E_k^-1 E_k+1 (4x4),
// hence Y_k diag(ph_k)^-1 = (Q21 + Q22 Z)(Q11 + Q12 Z)^-1 and Z_k = diag(ph_k) (that) diag(ph_k).
// E^-1 is in closed form: in sums s = d + u and differences t = d - u of the amplitudes the rows
// decouple into (s_P, t_S) and (t_P, s_S), 2x2 blocks of determinants rho nu and rho eta.
// Per (omega, p, interface) that leaves two 2x2 products, one 2x2 inverse and one more product:
// ~156 FP64 operations where the pivoted elimination of the 4x4 system took ~600 (943
// instructions); 1024 x 1023 of a 21-layer model 949 -> 278 us.
#include "kr_forward.cuh"

namespace kr {

// Interface k >= 1: Q up to a factor per interface (it cancels in the quotient), row by row.
// Interface 0 (ocean bottom): the eigenvector terms of layer 1, the ocean's eta and density, p.
struct GmmCoef {
  cd q11[4], q12[4], q21[4], q22[4];
};

static __device__ __noinline__ void gmm_store(double p, int k, const LayerP* lay, GmmCoef* out) {
  const LayerP& u = lay[k];
  const LayerP& l = lay[k + 1];
  const cd mul = l.rho * (l.betac * l.betac);
  GmmCoef o;
  if (k == 0) {
    // E_d = [[p, neta], [eta, -p], [-gamma, a], [b, gamma]], E_u with eta and neta negated
    const cd gamma = l.rho - (2.0 * p * p) * mul;
    o.q11[0] = u.eta;
    o.q11[1] = mk(u.rho, p);
    o.q11[2] = l.eta;
    o.q11[3] = gamma;
    o.q12[0] = (2.0 * p) * (mul * l.neta);
    o.q12[1] = (2.0 * p) * (mul * l.eta);
    o.q12[2] = o.q12[3] = mk(0.0, 0.0);
    for (int e = 0; e < 4; ++e) o.q21[e] = o.q22[e] = mk(0.0, 0.0);
    *out = o;
    return;
  }
  const cd d = 2.0 * (mul - u.rho * (u.betac * u.betac));
  const cd pd = (p * p) * d;
  const cd a = (l.rho - u.rho) - pd, b = l.rho - pd, c = u.rho + pd;
  // A fluid layer at p = 0 has neta = 0: its S amplitudes decouple from P there (every mixed entry has
  // a factor p) and are left without their coupling to the layer below instead of dividing by zero.
  const cd ie = recip(u.eta);
  const cd in = (u.neta.x == 0.0 && u.neta.y == 0.0) ? mk(0.0, 0.0) : recip(u.neta);
  const cd cp = (c * l.eta) * ie, cs = (c * l.neta) * in;   // c eta2 / eta1, c neta2 / neta1
  const cd ap = p * (a * ie), as = p * (a * in);            // p a / eta1, p a / neta1
  const cd dn = p * (d * l.neta), de = p * (d * l.eta);     // p d neta2, p d eta2
  o.q11[0] = b + cp;  o.q11[1] = ap - dn;  o.q11[2] = de - as;     o.q11[3] = b + cs;
  o.q12[0] = b - cp;  o.q12[1] = ap + dn;  o.q12[2] = -(de + as);  o.q12[3] = b - cs;
  o.q21[0] = b - cp;  o.q21[1] = -(ap + dn);  o.q21[2] = de + as;  o.q21[3] = b - cs;
  o.q22[0] = b + cp;  o.q22[1] = dn - ap;  o.q22[2] = as - de;     o.q22[3] = b + cs;
  *out = o;
}

// s + M Z for 2x2 matrices given row by row.
__device__ __forceinline__ void mac22(const cd s[4], const cd m[4], const cd z[4], cd o[4]) {
  o[0] = cmac(cmac(s[0], m[0], z[0]), m[1], z[2]);
  o[1] = cmac(cmac(s[1], m[0], z[1]), m[1], z[3]);
  o[2] = cmac(cmac(s[2], m[2], z[0]), m[3], z[2]);
  o[3] = cmac(cmac(s[3], m[2], z[1]), m[3], z[3]);
}
// A B^-1
__device__ __forceinline__ void div22(const cd a[4], const cd b[4], cd y[4]) {
  const cd id = recip_near(cdot2(b[0], b[3], -b[1], b[2]));
  y[0] = cdot2(a[0], b[3], -a[1], b[2]) * id;
  y[1] = cdot2(a[1], b[0], -a[0], b[1]) * id;
  y[2] = cdot2(a[2], b[3], -a[3], b[2]) * id;
  y[3] = cdot2(a[3], b[0], -a[2], b[1]) * id;
}

struct GmmForm {
  typedef GmmCoef Coef;
  static __device__ __forceinline__ void store(double p, int i, const LayerP* lay,
                                               const LayerRoots*, const LayerRoots*, Coef* out) {
    gmm_store(p, i, lay, out);
  }
  template <int F, class Ph>
  static __device__ __forceinline__ void sweep(int n_layers, const Coef* coef, const Ph& ph,
                                               bool fs, cd R[F]) {
    const int M = n_layers - 2;  // interfaces M .. 1 between solids
    cd P[F], Q[F], S[F], E[F];
    cd y[F][4];
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
      for (int e = 0; e < 4; ++e) y[f][e] = mk(0.0, 0.0);
    if (M >= 1) {  // nothing comes back from the half-space
      cd y0[4];
      div22(coef[M].q21, coef[M].q11, y0);
#pragma unroll
      for (int f = 0; f < F; ++f)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[f][e] = y0[e];
    }
#pragma unroll 1
    for (int k = M - 1; k >= 1; --k) {
      ph.pqs(k + 1, P, Q, S);
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const cd z[4] = {P[f] * y[f][0], S[f] * y[f][1], S[f] * y[f][2], Q[f] * y[f][3]};
        cd a[4], b[4];
        mac22(coef[k].q21, coef[k].q22, z, a);
        mac22(coef[k].q11, coef[k].q12, z, b);
        div22(a, b, y[f]);
      }
    }
    if (M >= 1) ph.pqs(1, P, Q, S);
    ph.ocean(E);
    // ocean bottom: layer 1's displacement and traction rows [u_z], [sigma], [tau] of
    // E_d + E_u Z; tau = 0 and continuity of u_z and sigma with e_d = (eta0, -rho0),
    // e_u = (-eta0, -rho0)
    const GmmCoef& o = coef[0];
    const cd eta0 = o.q11[0], eta = o.q11[2], gamma = o.q11[3], ea = o.q12[0], eb = o.q12[1];
    const double rho0 = o.q11[1].x, p = o.q11[1].y;
#pragma unroll
    for (int f = 0; f < F; ++f) {
      cd z[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) z[e] = mk(0.0, 0.0);
      if (M >= 1) {
        z[0] = P[f] * y[f][0];
        z[1] = S[f] * y[f][1];
        z[2] = S[f] * y[f][2];
        z[3] = Q[f] * y[f][3];
      }
      // rows 1 (u_z), 2 (sigma), 3 (tau) of E_d + E_u Z
      const cd u0 = cmac(eta, -eta, z[0]) - p * z[2], u1 = cmac(mk(-p, 0.0), -eta, z[1]) - p * z[3];
      const cd s0 = cmac(cmac(-gamma, -gamma, z[0]), -ea, z[2]);
      const cd s1 = cmac(cmac(ea, -gamma, z[1]), -ea, z[3]);
      const cd t0 = cmac(cmac(eb, -eb, z[0]), gamma, z[2]);
      const cd t1 = cmac(cmac(gamma, -eb, z[1]), gamma, z[3]);
      // D = (t1, -t0) up to a factor makes the traction vanish; eliminating the factor from
      // u_z = eta0 (1 - r), sigma = -rho0 (1 + r) (amplitudes at the ocean bottom) gives r
      const cd uz = cdot2(u0, t1, -u1, t0), sg = cdot2(s0, t1, -s1, t0);
      const cd en = eta0 * sg, ru = rho0 * uz;
      const cd r = (en + ru) * recip_near(en - ru);
      const cd v = E[f] * r;
      R[f] = fs ? v * recip(1.0 + v) : v;
    }
  }
};

}  // namespace kr

using namespace kr;

extern "C" kr_status kr_gmm_reflectivity(const double* layers, int32_t n_layers, const double* p,
                                         int32_t n_p, const double* omega, int32_t n_w,
                                         uint32_t flags, double* R, void* stream) {
  if (n_p < 0 || n_w < 0 || (flags & ~KR_FREE_SURFACE)) return KR_ERR_INVALID_ARGUMENT;
  if (n_layers < 2) return KR_ERR_INVALID_MODEL;
  if (n_layers > kMaxLayers) return KR_ERR_TOO_LARGE;
  if (n_p == 0 || n_w == 0) return KR_OK;
  if (!layers || !p || !omega || !R) return KR_ERR_INVALID_ARGUMENT;
  if (!aligned16(omega) || !aligned16(R)) return KR_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  constexpr const char* kWhat = "kr_gmm_reflectivity";
  if (n_layers > kPqsLayers)
    return launch_forward_deep<GmmForm>(kWhat, layers, n_layers, p, n_p, omega, n_w, flags, R, st);
  return launch_forward<GmmForm, 3, 1, 4, 4>(kWhat, layers, n_layers, p, n_p, omega, n_w, flags, R,
                                             st);
}
