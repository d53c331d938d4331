"""The pairwise Hessian kernels at the edges of their blocks: frequency counts around a chunk of 16
and a tile of 128, layer counts around a round of eight and the deepest that fits, slownesses
processed in several turns, against the tangent-of-adjoint kernel direction by direction."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [2, 3, 9, 10, 21, 50, 51])
@pytest.mark.parametrize("n_w", [1, 15, 17, 140])
def test_pairwise_hessian_vs_directions(layers, n_w):
    from seismicinversion_b200 import _lib
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.earth_models import random_layered_model

    m = random_layered_model(layers - 1, seed=80 + layers)
    tab = D.layer_table(m)
    p = torch.linspace(0.04, 0.5, 3, dtype=torch.float64, device="cuda")
    w = torch.arange(1, n_w + 1, dtype=torch.float64, device="cuda") * (2 * np.pi / 64) + 0.05j
    gen = torch.Generator(device="cpu").manual_seed(n_w)
    obs = torch.randn(3, n_w, dtype=torch.complex128, generator=gen).cuda()
    fits = _lib.lib().kr_misfit_hessian_workspace_bytes(layers, 3, n_w) > 0
    assert fits == (layers <= 50)
    n = 4 * (layers - 1) - 1
    idx = torch.as_tensor([k * layers + l for k in range(4) for l in range(1, layers)][:n],
                          device="cuda")
    V = torch.zeros((n, 4 * layers), dtype=torch.float64, device="cuda")
    V[torch.arange(n, device="cuda"), idx] = 1.0
    for fs in (False, True):
        H = D.misfit_hessian(tab, p, w, obs, fs)
        want = D.misfit_hvp(tab, p, w, obs, V, fs)[:, idx]
        assert H.shape == (n, n) and torch.equal(H, H.T)
        # two orders of differentiation: rounding of ~1e-13 per term, 1e-10 as for the oracle
        assert float((H - want).abs().max()) < 1e-10 * float(want.abs().max())
        assert torch.equal(H, D.misfit_hessian(tab, p, w, obs, fs))  # deterministic


def test_turns_of_slownesses():
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.earth_models import random_layered_model

    tab = D.layer_table(random_layered_model(20, seed=3))
    # 320 B per (p, omega, layer): 5000 frequencies make a turn 16 slownesses
    p = torch.linspace(0.05, 0.4, 37, dtype=torch.float64, device="cuda")
    w = torch.arange(1, 5001, dtype=torch.float64, device="cuda") * 0.01 + 0.05j
    obs = torch.zeros(37, 5000, dtype=torch.complex128, device="cuda")
    H = D.misfit_hessian(tab, p, w, obs)
    parts = sum(D.misfit_hessian(tab, p[a:a + 5], w, obs[a:a + 5]) for a in range(0, 37, 5))
    assert float((H - parts).abs().max()) < 1e-12 * float(H.abs().max())
