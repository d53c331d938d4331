"""A misfit's gradient as torch forms it, kr_vjp of 2 (R - obs) with the forward kernel's R, against
kr_misfit_gradient, which seeds the same sweep with the sweep's own R.

The difference is the sum of conj(2 dR) dR/dtheta over dR = R_forward - R_sweep: small only where
both round their phases alike, since a rounding that a whole frequency tile shares adds up over
the tile.  Geometric mean over six models of the largest difference relative to the largest gradient
component: 1e-15 or below for random models and 1.4e-15 for the 5-layer default model when alike;
2.5e-14 and more when one side's phases are rounded otherwise (exponentials of the sums of two
layer exponents at 5 layers: 3.3e-14; plain exponentials against a table at 49 to 66: 2.5e-14).  8e-15 lies between, by a factor of three and more each way.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [5, 12, 30, 31, 48, 49, 64, 66, 67])
def test_adjoint_of_the_forward_R(layers):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.earth_models import default_ocean_crust_model, random_layered_model
    from seismicinversion_b200.layer_model import pack_layers

    logs = []
    for s in range(6):
        m = default_ocean_crust_model() if layers == 5 else random_layered_model(layers - 1, s + layers)
        t = np.ascontiguousarray(pack_layers(m))
        rng = np.random.default_rng(s)
        t[:4, 1:] *= rng.uniform(0.9, 1.1, (4, layers))[:, 1:]
        tab = torch.as_tensor(t, device="cuda")
        n_p, n_w = ((26, 314), (4, 717), (63, 500), (9, 1024))[s % 4]
        p = torch.linspace(0.05, 0.6, n_p, dtype=torch.float64, device="cuda")
        w = np.arange(1, n_w + 1) * (2 * np.pi / 64)
        obs = sum(a * np.exp(1j * w * tau) for a, tau in zip(rng.normal(0, 0.2, 6),
                                                             rng.uniform(1, 8, 6)))
        obs = torch.as_tensor(obs, device="cuda")[None, :].expand(n_p, n_w).contiguous()
        w = torch.as_tensor(w, device="cuda").to(torch.complex128)
        R = D.reflectivity(tab, p, w, False)
        v = D.vjp(tab, p, w, 2.0 * (R - obs), False)[0]
        g = D.misfit_gradient(tab, p, w, obs, False)[0][:-1]
        logs.append(np.log(float((v - g).abs().max() / g.abs().max()) + 1e-18))
    assert np.exp(np.mean(logs)) <= 8e-15, np.exp(logs)
