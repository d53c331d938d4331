"""The ray sweep's frequency sums (matrix-instruction sums of the adjoints) at the edges of its
tiles: frequency counts around a warp (32) and a block (128), the fewest layers, and models
around the tape's 64 steps, single model and batch, against the Jacobian contraction."""

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [2, 3, 21, 31, 66, 67])
@pytest.mark.parametrize("n_w", [1, 31, 33, 128, 161])
def test_frequency_sums_match_the_jacobian(layers, n_w):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.batch import BatchItem, ModelBatch
    from seismicinversion_b200.earth_models import random_layered_model

    m = random_layered_model(layers - 1, seed=40 + layers)
    tab = D.layer_table(m)
    p = torch.linspace(0.03, 0.55, 3, dtype=torch.float64, device="cuda")
    w = torch.arange(1, n_w + 1, dtype=torch.float64, device="cuda") * (2 * np.pi / 64) + 0.05j
    gen = torch.Generator(device="cpu").manual_seed(n_w)
    obs = torch.randn(3, n_w, dtype=torch.complex128, generator=gen).cuda()
    for fs in (False, True):
        R, J = D.jacobian(tab, p, w, fs)
        r = R - obs
        want = 2.0 * (r.conj().unsqueeze(1) * J).real.sum((0, 2)).cpu().numpy()
        chi = float((r.real ** 2 + r.imag ** 2).sum())
        # 3 n_w terms of size <= max|r| max|J| a sum: rounding stays below 1e-12 of the largest
        out, _ = D.misfit_gradient(tab, p, w, obs, fs)
        assert rel_err(out[:-1].cpu().numpy(), want) < 1e-12
        assert abs(float(out[-1]) - chi) < 1e-12 * chi
        b = ModelBatch([BatchItem(m, p, w, gradient=True, R_obs=obs, free_surface=fs)])
        b.launch()
        assert rel_err(b.misfit_gradient(0)[1].cpu().numpy(), want) < 1e-12
        g, _ = D.vjp(tab, p, w, 2.0 * r, fs)
        assert rel_err(g.cpu().numpy(), want) < 1e-12
