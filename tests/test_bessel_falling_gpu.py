"""The Bessel sum over falling slownesses, against a direct sum with SciPy's j0: tiles above x = 25 for
every frequency, tiles below, tiles that cross it and tiles that cross zero, full and short.

Tolerance per entry, relative to sum_j |f_j omega R_j|: below 1.5e-15 sqrt(2 |x| / pi) from the
roundings of the phase (|x| <= 5e3: 9e-14), 2e-14 from 32 rotation steps, 1e-15 from J0.  2e-13
covers the sum.
"""

import numpy as np
import pytest
import torch
from scipy.special import j0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_p", [1, 2, 31, 32, 33, 64, 65, 200])
@pytest.mark.parametrize("hi,lo", [(0.6, 0.01), (1.2, 0.0), (1.2, 0.7), (0.6, -0.6), (-0.1, -1.2)])
def test_falling_slownesses(n_p, hi, lo):
    from seismicinversion_b200 import device as D

    rng = np.random.default_rng(n_p)
    p = np.linspace(hi, lo, n_p)
    om = np.r_[0.0, np.arange(1, 40) * 0.7, np.linspace(60.0, 100.0, 9)]
    r = np.array([0.0, 0.05, 0.8, 11.0, 40.0])
    R = rng.standard_normal((n_p, len(om))) + 1j * rng.standard_normal((n_p, len(om)))
    pw = rng.uniform(-0.5, 1.0, n_p)
    f = (pw[:, None] * om[None, :]) * 1e-2 * R
    scale = np.sum(np.abs(f), axis=0)
    U = D.bessel_sum(torch.as_tensor(R, device="cuda"), p, pw, 1e-2, om, r).cpu().numpy()
    for k, rk in enumerate(r):
        ref = np.sum(j0((om[None, :] * p[:, None]) * rk) * f, axis=0)
        assert np.all(np.abs(U[k] - ref) <= 2e-13 * scale), rk
