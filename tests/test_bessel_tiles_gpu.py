"""The Bessel sum at the edges of its tiles and ways, against a direct sum with SciPy's j0.

Slowness counts around the tile of 32 and the slice of 64; progressions whose tiles stay below
x = 25, cross it and lie above; step angles up to and beyond half a turn (coarse grids, where the
rotation is by products instead of shears); frequency 0 and offset 0 beside ordinary ones;
slownesses off the progression.

Tolerance per entry, relative to sum_j |f_j omega R_j|: the phase x carries a few roundings in each
of the two orders of evaluation and the progression holds to 4.5 ulp, together below 1.5e-15 x,
which J0's amplitude turns into at most 1.5e-15 sqrt(2 x / pi) = 1.4e-13 at x = 1.4e4; 32
rotation steps of a few roundings each add 2e-14, J0 itself 1e-15.  2e-13 covers the sum.
"""

import numpy as np
import pytest
import torch
from scipy.special import j0

pytestmark = pytest.mark.gpu


def _check(p, om, r, dp, seed):
    from seismicinversion_b200 import device as D

    rng = np.random.default_rng(seed)
    R = rng.standard_normal((len(p), len(om))) + 1j * rng.standard_normal((len(p), len(om)))
    pw = p * rng.uniform(0.2, 1.0, len(p))
    U = D.bessel_sum(torch.as_tensor(R, device="cuda"), p, pw, dp, om, r).cpu().numpy()
    f = (pw[:, None] * om[None, :]) * dp * R
    scale = np.sum(np.abs(f), axis=0)
    for k, rk in enumerate(r):
        ref = np.sum(j0((om[None, :] * p[:, None]) * rk) * f, axis=0)
        assert np.all(np.abs(U[k] - ref) <= 2e-13 * scale), (len(p), len(om), rk)


@pytest.mark.parametrize("n_p", [1, 2, 31, 32, 33, 64, 65, 95, 200])
@pytest.mark.parametrize("first", [0, 1])
def test_tile_edges_on_a_progression(n_p, first):
    """Small n_p makes coarse steps: angles of many turns at the large offsets and frequencies."""
    dp = 1.2 / n_p
    p = np.arange(first, n_p + first) * dp
    om = np.r_[0.0, np.arange(1, 65) * (2 * np.pi / 64), np.linspace(150.0, 200.0, 7)]
    _check(p, om, np.array([0.0, 0.02, 0.5, 3.0, 11.0, 24.0, 37.0, 49.0, 50.0]), dp, n_p)


@pytest.mark.parametrize("d", [0.4, 0.5 * np.pi, 2.05, 2.12, 3.1, np.pi, 3.2, 4.5, 2 * np.pi])
def test_step_angles_across_the_choice_of_rotation(d):
    """omega r dp around 2 pi / 3 (shears up to there), pi and a full turn, lanes on both sides."""
    n_p, dp = 150, 0.008
    p = np.arange(1, n_p + 1) * dp
    om = np.linspace(0.9, 1.1, 33) * (d / (dp * 40.0))
    _check(p, om, np.array([40.0, 39.5]), dp, 5)


def test_off_the_progression_and_reversed():
    rng = np.random.default_rng(2)
    p = np.sort(rng.uniform(0.0, 1.2, 130))
    p[40:110] = 0.3 + np.arange(70) * 0.004  # tiles on a progression that is not the slice's
    om = np.arange(1, 34) * 5.9
    for q in (p, p[::-1].copy(), -np.arange(1, 70) * 0.01):
        _check(q, om, np.array([0.0, 0.7, 33.0]), 1e-3, 3)
