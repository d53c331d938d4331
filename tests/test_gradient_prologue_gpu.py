"""The frequency-sum sweep with its own prologue (small grids) and with the prepared coefficients
(large ones): R bit for bit the same, gradients the same to the order of the additions.

A slowness's share of the gradient sums the same products in the same order within a block; only the
blocks' sum is ordered otherwise: 1e-13 of the sum of magnitudes over up to 8 x 24 blocks."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,n_p", [(2, 96), (3, 96), (21, 96), (23, 96), (24, 96), (31, 96), (48, 60)])
@pytest.mark.parametrize("fs", [False, True])
def test_own_and_prepared_coefficients_agree(layers, n_p, fs):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.earth_models import random_layered_model

    tab = D.layer_table(random_layered_model(layers - 1, seed=layers))
    p = torch.linspace(0.03, 0.58, n_p, dtype=torch.float64, device="cuda")
    w = (torch.arange(1, 1001, dtype=torch.float64, device="cuda") * 0.1).to(torch.complex128)
    gen = torch.Generator(device="cpu").manual_seed(layers)
    obs = torch.randn(n_p, 1000, dtype=torch.complex128, generator=gen).cuda()
    g, R = D.misfit_gradient(tab, p, w, obs, fs, want_R=True)  # 8 n_p blocks: prepared
    parts, mags = torch.zeros_like(g), torch.zeros_like(g)
    for a in range(0, n_p, 12):  # 96 blocks: own
        ga, Ra = D.misfit_gradient(tab, p[a:a + 12], w, obs[a:a + 12], fs, want_R=True)
        assert torch.equal(torch.view_as_real(Ra), torch.view_as_real(R[a:a + 12]))
        parts += ga
        mags += ga.abs()
    assert bool(((parts - g).abs() <= 1e-13 * mags.max()).all())
