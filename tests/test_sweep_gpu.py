"""The forward sweep at the edges of its dispatch: layer counts around the phase-table classes (30
and 66 layers), frequency counts around a warp's pass and a tile, slowness counts that leave a
block's group partly empty, and a tile off the grid's line, against the oracle (1e-10, the
library's accuracy) and, bit for bit, the batched kernel."""

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [2, 3, 5, 30, 31, 66, 67])
@pytest.mark.parametrize("n_p,n_w", [(1, 1), (3, 33), (17, 129), (50, 300)])
def test_sweep_edges(layers, n_p, n_w):
    from oracle import kennett_oracle as O
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.batch import BatchItem, ModelBatch
    from seismicinversion_b200.earth_models import random_layered_model

    m = random_layered_model(layers - 1, seed=layers)
    tab = D.layer_table(m)
    p = np.linspace(0.02, 0.6, n_p)
    w = np.arange(1, n_w + 1) * (2 * np.pi / 64) + 1j * np.pi / 64
    if n_w == 300:
        w[[130, 131]] = w[[131, 130]]  # tile 1 leaves the line
    fs = n_p % 2 == 1
    R = D.reflectivity(tab, p, w, fs)
    want = O.reflectivity(m.alpha, m.beta, m.rho, m.thickness, m.Q_alpha, m.Q_beta, p, w, fs)
    assert rel_err(R.cpu().numpy(), want) < 1e-10
    for schedule in ((32, 64), (64, 100), (128, 2048)):
        b = ModelBatch([BatchItem(m, p, w, free_surface=fs)], schedule=schedule)
        b.launch()
        assert torch.equal(b.reflectivity(0), R)
