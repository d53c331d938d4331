// Test-only CPU build of the pairwise Hessian (seismicinversion_b200/csrc/kr_hess.cuh): the
// per-(omega, p) arithmetic of the Hessian kernels, summed on the host.
#include <vector>

#include "../../seismicinversion_b200/csrc/kr_hess.cuh"

using namespace kr;

namespace {
struct RayStore {
  HessStep* st;
  cd robs, seed, zeta;
  bool fs;
  int last;  // the bottom interface
  const Iface* coef;
  S3 K;
  std::vector<cd>* sums;
  cd reflectivity(cd R) {
    const cd r = R - robs;
    seed = mk(2.0 * r.x, -2.0 * r.y);
    // 1 + Y = 1 / (1 - R) with the free surface
    zeta = fs ? (-2.0 * seed) * recip(1.0 - R) : mk(0.0, 0.0);
    return mk(1.0, 0.0);
  }
  void top(cd) {}
  void ray(int i, const Ray& g, const Ray& x, const Ray& wz, const S3& X, cd ea, cd eb) {
    st[i] = HessStep{X, ea, eb, g, K};
    if (i < last) K = hess_next_k(K, X, ea, eb, coef[i]);
    cd c[12];
    ray_adjoints(g, x, c);
    c[10] = 2.0 * (wz.a * x.a);
    c[11] = 2.0 * (wz.b * x.b);
    for (int k = 0; k < 12; ++k) (*sums)[12 * i + k] = (*sums)[12 * i + k] + seed * c[k];
  }
};
}  // namespace

// H [4 I][4 I] over layers 1..I, index k I + (l - 1), k = alpha, beta, rho, h.
extern "C" void emu_hessian(const double* tab, int L, const double* p, int n_p, const double* w,
                            int nw, int fs, const double* R_obs, double* H) {
  const int I = L - 1, n = 4 * I;
  for (int q = 0; q < n * n; ++q) H[q] = 0.0;
  std::vector<LayerP> lay(L);
  std::vector<LayerD> dl(L);
  std::vector<LayerD2> d2(L);
  std::vector<Iface> f(I + 1);
  std::vector<ScatTan> t(I + 1);
  std::vector<HessStep> st(I + 1);
  std::vector<HessPublic> pub(I + 1);
  std::vector<HessOwn> own(I + 1);
  auto add = [&](int l, int j, int m, int k, double v) {
    const int r = j * I + l - 1, c = k * I + m - 1;
    H[r * n + c] += v;
    if (r != c) H[c * n + r] += v;
  };
  for (int ip = 0; ip < n_p; ++ip) {
    for (int l = 0; l < L; ++l) {
      lay[l] = layer_terms(tab, L, l, p[ip]);
      dl[l] = layer_derivs(tab, L, l, p[ip], lay[l]);
      d2[l] = layer_derivs2(tab, L, l, lay[l], dl[l]);
    }
    for (int i = 0; i < I; ++i) {
      f[i] = interface_coeffs(p[ip], i, lay[i], lay[i + 1]);
      interface_tangents(p[ip], i, lay[i], dl[i], lay[i + 1], dl[i + 1], t[i]);
    }
    std::vector<cd> sums(12 * I, mk(0.0, 0.0));
    for (int k = 0; k < nw; ++k) {
      const cd om = mk(w[2 * k], w[2 * k + 1]);
      RayStore s;
      s.st = st.data();
      s.robs = mk(R_obs[2 * ((size_t)ip * nw + k)], R_obs[2 * ((size_t)ip * nw + k) + 1]);
      s.fs = fs != 0;
      s.last = I - 1;
      s.coef = f.data();
      s.K = S3{mk(0.0, 0.0), mk(0.0, 0.0), mk(0.0, 0.0)};
      s.sums = &sums;
      adjoint_rays(L, om, fs != 0, checkpoint_spacing(I > 1 ? I - 1 : 1), f.data(),
                   PhaseDirect{om, lay.data()}, s);
      for (int l = 1; l <= I; ++l)
        hess_layer(l, I, om, s.seed, s.zeta, st[l - 1], st[l], f[l - 1], f[l], t[l - 1], t[l],
                   dl[l], pub[l], own[l]);
      for (int m = 1; m <= I; ++m) {
        for (int j = 0; j < 4; ++j)
          for (int kk = 0; kk <= j; ++kk) add(m, j, m, kk, own[m].s[j * (j + 1) / 2 + kk]);
        Ray g[4] = {own[m].gn[0], own[m].gn[1], own[m].gn[2], own[m].gn[3]};
        for (int l = m + 1; l <= I; ++l)
          for (int kk = 0; kk < 4; ++kk) {
            if (l > m + 2) g[kk] = hess_down(pub[l - 2].G, g[kk]);
            for (int j = 0; j < 4; ++j)
              add(l, j, m, kk, l == m + 1
                  ? hess_adjacent(pub[l].w[j], pub[l].dx[j], pub[l].A[j], own[m], kk)
                  : hess_far(pub[l].w[j], pub[l].A[j], g[kk], own[m].J[kk]));
          }
      }
    }
    for (int i = 0; i < I; ++i)
      for (int item = 0; item < kHessItems; ++item) {
        const double v = hess_curvature(tab, L, i, p[ip], lay.data(), dl.data(), d2.data() + i,
                                        sums.data() + 12 * i, item);
        if (item >= 21) {
          static const int ja[4] = {0, 3, 1, 3}, ka[4] = {0, 0, 1, 1};
          add(i + 1, ja[item - 21], i + 1, ka[item - 21], v);
          continue;
        }
        int a = 0;
        while ((a + 1) * (a + 2) / 2 <= item) ++a;
        const int b = item - a * (a + 1) / 2;
        const int la = a < 3 ? i : i + 1, lb = b < 3 ? i : i + 1;
        if (la == 0 || lb == 0) continue;  // the ocean is not a parameter
        add(la, a % 3, lb, b % 3, v);
      }
  }
}
