"""A misfit's adjoint made from the forward sweep's R, against the derivative sweep's own R.

Without the free surface R = exp(2 i omega eta_0 h_0) R_below, so the thickness derivative of
chi = sum |R - obs|^2 by the water layer is sum 2 Re(conj(R - obs) 2 i omega eta_0 R) with the
forward's R; kr_vjp forms the same sum with the R of its own sweep.  The part with |R|^2 cancels
only as far as the two agree.

Tolerance: where both sweeps round the phase of a frequency tile alike, a term differs by the
rounding of a few exponentials and products, below 5e-16 of its magnitude and independent from
frequency to frequency; 5e-16 of the sum of magnitudes bounds it.  (Phases rounded differently
are off by up to an ulp of omega eta_0 h_0 for a whole tile: several 1e-15.)
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sub,n_p,n_w", [(4, 63, 873), (8, 4, 717), (30, 5, 300)])
def test_water_thickness_gradient_from_the_forward_R(n_sub, n_p, n_w):
    from seismicinversion_b200.earth_models import random_layered_model
    from seismicinversion_b200.kennett_torch import kennett_reflectivity_torch, model_to_tensors

    m = random_layered_model(n_sub, seed=14)
    p = np.linspace(0.05, 0.6, n_p)
    w = np.arange(1, n_w + 1) * (2 * np.pi / 64)
    t = {k: v.cuda() for k, v in model_to_tensors(m).items()}
    h = t["thickness"].requires_grad_(True)
    R = kennett_reflectivity_torch(t["alpha"], t["beta"], t["rho"], h, t["Q_alpha"], t["Q_beta"],
                                   torch.as_tensor(p, device="cuda"),
                                   torch.as_tensor(w, device="cuda").to(torch.complex128))
    rng = np.random.default_rng(n_sub)
    obs = sum(a * np.exp(1j * w * tau) for a, tau in zip(rng.normal(0, 0.2, 6),
                                                         rng.uniform(1, 8, 6)))[None, :]
    r = R - torch.as_tensor(obs, device="cuda")
    g = torch.autograd.grad((r.real ** 2 + r.imag ** 2).sum(), h)[0][0].item()

    Rn = R.detach().cpu().numpy()
    q2 = 2.0 * m.Q_alpha[0]
    den = (1.0 + q2 * q2) * m.alpha[0]
    s = q2 * q2 / den + 1j * q2 / den
    eta = np.sqrt((s + p) * (s - p))
    eta = np.where(eta.imag <= 0, -eta, eta)[:, None]
    term = 2j * w[None, :] * eta * Rn
    ref = np.sum(2.0 * (np.conj(Rn - obs) * term).real)
    scale = np.sum(2.0 * np.abs((Rn - obs) * term))
    assert abs(g - ref) <= 5e-16 * scale, ((g - ref) / scale, g / scale)
