"""Misfit gradient, vector-Jacobian product, batch and Hessian of the default model up to 1.2 s/km,
where the water layer is evanescent and its phase underflows gradually: finite, and the sums equal
to the contraction of the Jacobian.

Tolerance: a term is a product of ten coefficient adjoints with their tangents, which cancel by up
to ~1e3 near the interface poles above 0.67 s/km; 1e3 roundings are 2e-13 of a term's magnitude,
1e-12 of the largest parameter's sum of magnitudes bounds the difference of the two orders.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fs", [False, True])
def test_gradients_into_the_evanescent_range(fs):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.batch import BatchItem, ModelBatch
    from seismicinversion_b200.earth_models import default_ocean_crust_model

    m = default_ocean_crust_model()
    tab = D.layer_table(m)
    p = torch.linspace(0.05, 1.2, 64, dtype=torch.float64, device="cuda")
    w = torch.arange(1, 2048, dtype=torch.float64, device="cuda").to(torch.complex128)
    w = w * (2 * np.pi / 64)
    gen = torch.Generator(device="cpu").manual_seed(0)
    obs = torch.randn(64, 2047, dtype=torch.complex128, generator=gen).cuda()
    R, J = D.jacobian(tab, p, w, fs)
    r = R - obs
    want = 2.0 * (r.conj().unsqueeze(1) * J).real.sum((0, 2))
    scale = float((2.0 * r.abs().unsqueeze(1) * J.abs()).sum((0, 2)).max())
    assert bool(torch.isfinite(want).all())
    b = ModelBatch([BatchItem(m, p, w, gradient=True, R_obs=obs, free_surface=fs)])
    b.launch()
    for g in (D.misfit_gradient(tab, p, w, obs, fs)[0][:-1], D.vjp(tab, p, w, 2.0 * r, fs)[0],
              b.misfit_gradient(0)[1]):
        g = torch.as_tensor(g).to(want.device).reshape(-1)
        assert bool(torch.isfinite(g).all())
        assert float((g - want).abs().max()) <= 1e-12 * scale
    assert bool(torch.isfinite(D.misfit_hessian(tab, p, w, obs, fs)).all())
    # a cotangent that is subnormal itself
    tiny = torch.full_like(obs, 5e-324j)
    assert bool(torch.isfinite(D.vjp(tab, p, w, tiny, fs)[0]).all())
