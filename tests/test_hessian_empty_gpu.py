"""The misfit Hessian over an empty grid is zero for every depth, beyond the 50 layers of the
pairwise kernels too."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [5, 50, 51, 120])
@pytest.mark.parametrize("n_p,n_w", [(0, 7), (3, 0), (0, 0)])
def test_empty_grids(layers, n_p, n_w):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.earth_models import random_layered_model

    tab = D.layer_table(random_layered_model(layers - 1, seed=1))
    H = D.misfit_hessian(tab, np.linspace(0.1, 0.2, n_p), np.arange(1, n_w + 1) + 0j,
                         torch.zeros((n_p, n_w), dtype=torch.complex128, device="cuda"))
    n = 4 * (layers - 1) - 1
    assert H.shape == (n, n) and not bool(H.any())
