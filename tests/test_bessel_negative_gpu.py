"""The Bessel sum over slownesses that rise through zero or lie below it, against a direct sum with
SciPy's j0: tiles that cross zero, tiles with every argument on one side of -25 and tiles that
cross it, beside tiles above.

Tolerance per entry, relative to sum_j |f_j omega R_j|: below 1.5e-15 sqrt(2 |x| / pi) from the
roundings of the phase (|x| <= 5e3: 9e-14), 2e-14 from 32 rotation steps, 1e-15 from J0.  2e-13
covers the sum.
"""

import numpy as np
import pytest
import torch
from scipy.special import j0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_p", [31, 32, 33, 64, 65, 200])
@pytest.mark.parametrize("lo,hi", [(-0.6, 0.6), (-1.2, -0.1), (-0.6, 0.0), (-1e-3, 1.2)])
def test_slownesses_through_and_below_zero(n_p, lo, hi):
    from seismicinversion_b200 import _lib
    from seismicinversion_b200 import device as D

    rng = np.random.default_rng(n_p)
    p = np.linspace(lo, hi, n_p)
    om = np.r_[0.0, np.arange(1, 40) * 0.7, np.linspace(60.0, 100.0, 9)]
    r = np.array([0.0, 0.05, 0.8, 11.0, 40.0])
    R = rng.standard_normal((n_p, len(om))) + 1j * rng.standard_normal((n_p, len(om)))
    pw = rng.uniform(-0.5, 1.0, n_p)
    f = (pw[:, None] * om[None, :]) * 1e-2 * R
    scale = np.sum(np.abs(f), axis=0)
    Rd = torch.as_tensor(R, device="cuda")
    U = D.bessel_sum(Rd, p, pw, 1e-2, om, r)
    V = torch.empty_like(U)
    dev = [torch.as_tensor(v, device="cuda") for v in (p, pw, om, r)]
    st = _lib.lib().kr_bessel_sum_noalloc(
        Rd.data_ptr(), dev[0].data_ptr(), dev[1].data_ptr(), n_p, 1e-2, dev[2].data_ptr(), len(om),
        dev[3].data_ptr(), len(r), V.data_ptr(), D.stream_handle(Rd.device))
    _lib.check(st, "kr_bessel_sum_noalloc")
    for out in (U.cpu().numpy(), V.cpu().numpy()):
        for k, rk in enumerate(r):
            ref = np.sum(j0((om[None, :] * p[:, None]) * rk) * f, axis=0)
            assert np.all(np.abs(out[k] - ref) <= 2e-13 * scale), rk
