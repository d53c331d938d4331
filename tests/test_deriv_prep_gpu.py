"""The derivative sweeps' preparation over many slownesses at once: blocks of it hold parts of several
slownesses, or part of one, and each slowness's results are the same bit for bit as by itself."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [2, 3, 5, 19, 20, 21, 38, 64])
def test_slownesses_do_not_depend_on_their_neighbours(layers):
    from seismicinversion_b200 import device as D
    from seismicinversion_b200.earth_models import random_layered_model

    tab = D.layer_table(random_layered_model(layers - 1, seed=layers))
    p = torch.linspace(0.03, 0.58, 41, dtype=torch.float64, device="cuda")
    w = (torch.arange(1, 36, dtype=torch.float64, device="cuda") * 0.1 + 0.05j).to(torch.complex128)
    R, J = D.jacobian(tab, p, w)
    assert bool(torch.isfinite(torch.view_as_real(J)).all())
    for j in (0, 1, 7, 18, 19, 39, 40):
        Rj, Jj = D.jacobian(tab, p[j:j + 1], w)
        assert torch.equal(torch.view_as_real(Rj[0]), torch.view_as_real(R[j]))
        assert torch.equal(torch.view_as_real(Jj[0]), torch.view_as_real(J[j]))
