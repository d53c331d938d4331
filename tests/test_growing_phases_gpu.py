"""Jacobian, gradients and Hessian at frequencies whose phases grow with depth (negative real part,
thick attenuating layers; also a few such frequencies within an ordinary grid), against fourth-order
differences of the forward kernel.

Tolerance: steps of 1e-5 turn phases by up to 1e-3, 1e-2 near a turning point, whose fourth power
bounds the differences' error; the forward's rounding, 1e-13 over 1e-3, adds 1e-10.  1e-6 of the
largest entry."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [5, 9, 52, 70])
@pytest.mark.parametrize("grid", ["line", "off", "mixed"])
@pytest.mark.parametrize("fs", [False, True])
def test_derivatives_with_growing_phases(layers, grid, fs):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.batch import BatchItem, ModelBatch
    from seismicinversion_b200.earth_models import default_ocean_crust_model, random_layered_model
    from seismicinversion_b200.layer_model import LayerModel, pack_layers
    from seismicinversion_b200.taup_inversion import _Problem

    m = default_ocean_crust_model() if layers == 5 else random_layered_model(layers - 1, seed=3)
    th = m.thickness * (20.0 if layers < 50 else 4.0)
    m = LayerModel.from_arrays(m.alpha, m.beta, m.rho, th, m.Q_alpha, m.Q_beta)
    tab = torch.as_tensor(np.ascontiguousarray(pack_layers(m)), device="cuda")
    L = layers
    w = -np.arange(1, 34) * 0.098 + 0.05j
    if grid == "off":
        w = w * np.linspace(0.9, 1.0, 33) ** 2
    if grid == "mixed":
        w[5:] = np.abs(w[5:].real)
    p = torch.tensor([0.03, 0.2, 0.55], dtype=torch.float64, device="cuda")
    w = torch.as_tensor(w, device="cuda")
    gen = torch.Generator(device="cpu").manual_seed(layers)
    obs = 0.3 * torch.randn(3, 33, dtype=torch.complex128, generator=gen).cuda()
    R, J = D.jacobian(tab, p, w, fs)
    want = torch.zeros_like(J)
    for k in range(4):
        for l in range(L):
            d = 1e-5 * float(tab[k, l])
            if d == 0.0 or not d < 1e20:
                continue
            for o, c in ((2, -1.0), (1, 8.0), (-1, -8.0), (-2, 1.0)):
                t = tab.clone()
                t[k, l] += o * d
                want[:, k * L + l] += c / (12.0 * d) * D.reflectivity(t, p, w, fs)
    assert float((J - want).abs().max()) <= 1e-6 * float(want.abs().max())
    r = R - obs
    g = 2.0 * (r.conj().unsqueeze(1) * J).real.sum((0, 2))
    b = ModelBatch([BatchItem(m, p, w, gradient=True, R_obs=obs, free_surface=fs)])
    b.launch()
    for v in (D.misfit_gradient(tab, p, w, obs, fs)[0][:-1], D.vjp(tab, p, w, 2.0 * r, fs)[0],
              b.misfit_gradient(0)[1]):
        v = torch.as_tensor(v).to(g.device).reshape(-1)
        assert float((v - g).abs().max()) <= 1e-12 * float(g.abs().max())
    if layers <= 9:
        assert bool(torch.isnan(D.misfit_hessian(tab, p, w, obs, fs)).all())
        prob = _Problem(m.alpha, m.beta, m.rho, th, m.Q_alpha, m.Q_beta, p.cpu().numpy(), w,
                        obs.cpu().numpy(), free_surface=fs)
        par = np.concatenate([m.alpha[1:], m.beta[1:], m.rho[1:], th[1:-1]])
        H = prob.hessian_exact(par)
        fd = prob.hessian_fd(par, step=1e-5, stencil=4)
        assert np.abs(H - fd).max() <= 1e-6 * np.abs(fd).max()
