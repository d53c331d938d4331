"""The global-matrix R of models with a fluid layer below the ocean at vertical incidence, where
that layer's S slowness is zero, against the acoustic recursion of the P amplitudes alone (P and S
decouple at p = 0).

Tolerance: the recursion is a product of bounded factors, both evaluations agree to a few hundred
roundings; 1e-13 absolute (|R| <= 1 without the free surface)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,fluid", [(3, 1), (5, 1), (5, 2), (12, 1), (12, 2), (12, 10), (40, 1),
                                          (70, 1)])
def test_fluid_layer_at_vertical_incidence(layers, fluid):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.earth_models import random_layered_model
    from seismicinversion_b200.layer_model import pack_layers

    t = np.ascontiguousarray(pack_layers(random_layered_model(layers - 1, seed=layers)))
    t[1, fluid] = 0.0
    w = np.arange(1, 150) * (2 * np.pi / 64) + 0.05j
    p = torch.tensor([0.0, 0.1], dtype=torch.float64, device="cuda")
    R = D.gmm_reflectivity(torch.as_tensor(t, device="cuda"), p, torch.as_tensor(w, device="cuda"))
    assert bool(torch.isfinite(R.real).all())
    q2 = 2.0 * t[4]
    eta = (q2 * q2 + 1j * q2) / ((1.0 + q2 * q2) * t[0])
    Z = t[2] / eta
    r = np.zeros(len(w), dtype=np.complex128)
    for i in range(layers - 2, -1, -1):
        c = (Z[i + 1] - Z[i]) / (Z[i + 1] + Z[i])
        m = r * np.exp(2j * w * eta[i + 1] * t[3, i + 1]) if i < layers - 2 else 0.0
        r = (c + m) / (1.0 + c * m)
    r = r * np.exp(2j * w * eta[0] * t[3, 0])
    assert np.abs(R[0].cpu().numpy() - r).max() <= 1e-13
