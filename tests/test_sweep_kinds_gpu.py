"""The kernels that the forward sweep of a deep model chooses from by the size of the grid: each slowness's
R is the same bit for bit in a large call (few slownesses' data fit an SM: phases by lanes, four warps
a block), in a call of its own (phase table, eight warps), and in a batch."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grids():
    k = np.arange(1, 65)
    yield "line", k * 0.098 + 0.05j
    yield "single", k[:1] * 0.3 + 0j
    yield "pass", k[:33] * 0.2 + 0j
    yield "falling", k[::-1] * 0.05 + 0.02j
    yield "growing", -k * 0.03 + 0.01j  # phases that grow with depth, to beyond a table's entries
    yield "irregular", np.sort(np.random.default_rng(3).uniform(0.1, 6.0, 50)) + 0.05j
    yield "two tiles", np.arange(1, 131) * 0.098 + 0j


@pytest.mark.parametrize("layers", [31, 48, 66, 67, 120, 128, 200, 256])
@pytest.mark.parametrize("name", [n for n, _ in _grids()])
def test_every_kernel_gives_the_same_bits(layers, name):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.batch import BatchItem, ModelBatch
    from seismicinversion_b200.earth_models import random_layered_model

    w = dict(_grids())[name]
    model = random_layered_model(layers - 1, seed=layers)
    tab = D.layer_table(model)
    p = np.linspace(0.0, 0.6, 700)
    for f in (D.reflectivity, D.gmm_reflectivity):
        R = torch.view_as_real(f(tab, p, w))
        for j in (0, 1, 2, 350, 698, 699):
            assert torch.equal(torch.view_as_real(f(tab, p[j:j + 1], w))[0].nan_to_num(), R[j].nan_to_num())
    batch = ModelBatch([BatchItem(model, p, w)])
    batch.launch()
    ref = torch.view_as_real(D.reflectivity(tab, p, w))
    assert torch.equal(torch.view_as_real(batch.reflectivity(0)).reshape(ref.shape).nan_to_num(), ref.nan_to_num())
