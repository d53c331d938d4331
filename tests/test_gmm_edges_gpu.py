"""The global-matrix form of the sweep at the edges of its dispatch (layer counts around the phase
classes, partial passes and groups, a tile off the grid's line) against the oracle's pivoted 4x4
systems (1e-10, the library's accuracy)."""

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [2, 3, 4, 30, 31, 67])
@pytest.mark.parametrize("n_p,n_w", [(1, 1), (3, 33), (18, 300)])
def test_gmm_edges(layers, n_p, n_w):
    from oracle import gmm_oracle as G
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.earth_models import random_layered_model

    m = random_layered_model(layers - 1, seed=20 + layers)
    p = np.linspace(0.02, 0.6, n_p)
    w = np.arange(1, n_w + 1) * (2 * np.pi / 64) + 1j * np.pi / 64
    if n_w == 300:
        w[[130, 131]] = w[[131, 130]]
    for fs in (False, True):
        R = D.gmm_reflectivity(D.layer_table(m), p, w, fs).cpu().numpy()
        want = G.gmm_reflectivity(m.alpha, m.beta, m.rho, m.thickness, m.Q_alpha, m.Q_beta, p, w,
                                  fs)
        assert rel_err(R, want) < 1e-10
