"""Batches of tables under their default schedules: every shape's R is kr_reflectivity's bit for bit."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,n,n_p,n_w", [(3, 20, 5, 64), (8, 3, 4, 512), (12, 400, 12, 40), (21, 30, 12, 700),
                                              (31, 10, 8, 33), (48, 420, 12, 64), (66, 3, 3, 1030), (66, 9, 4, 1),
                                              (67, 30, 4, 300), (128, 5, 3, 50), (256, 2, 3, 200)])
def test_default_schedule_gives_the_same_bits(layers, n, n_p, n_w):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.batch import ModelBatch
    from seismicinversion_b200.earth_models import random_layered_model
    from seismicinversion_b200.layer_model import pack_layers

    models = [random_layered_model(layers - 1, seed=s) for s in range(min(n, 4))]
    p, w = np.linspace(0.0, 0.6, n_p), np.arange(1, n_w + 1) * 0.1 + 0.03j
    batch = ModelBatch.from_tables(np.stack([pack_layers(models[i % len(models)]) for i in range(n)]), p, w)
    batch.launch()
    for b in {0, 1, n // 2, n - 1}:
        ref = D.reflectivity(D.layer_table(models[b % len(models)]), p, w)
        assert torch.equal(torch.view_as_real(batch.reflectivity(b)).reshape(n_p, n_w, 2), torch.view_as_real(ref))
