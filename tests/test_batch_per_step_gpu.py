"""KR_DERIV_SUMS=0 takes the per-step contraction for gradient items of every depth class: the
same gradients to rounding by other additions, so not the same bits.  One item per model (32
frequencies of one slowness), whose sums have a fixed order."""

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_RUN = """
import sys
import numpy as np
from seismicinversion_b200.batch import BatchItem, ModelBatch
from seismicinversion_b200.earth_models import random_layered_model

w = np.arange(1, 33) * 0.3 + 0.05j
rng = np.random.default_rng(0)
items = [BatchItem(random_layered_model(L - 1, seed=L), np.array([0.2]), w, gradient=True,
                   R_obs=rng.standard_normal((1, 32)) + 1j * rng.standard_normal((1, 32)))
         for L in (3, 5, 21, 30, 31, 49, 70)]
b = ModelBatch(items, schedule=(32, 128))
b.launch()
rows = [b.misfit_gradient(i)[1].cpu().numpy().reshape(-1) for i in range(len(items))]
np.save(sys.argv[1], np.stack([np.pad(r, (0, 280 - len(r))) for r in rows]))
"""


def test_the_switch_reaches_every_class(tmp_path):
    root = Path(__file__).resolve().parent.parent
    out = []
    for value in ("1", "1", "0"):
        f = tmp_path / f"{len(out)}.npy"
        subprocess.run([sys.executable, "-c", _RUN, str(f)], check=True, cwd=root,
                       env={**os.environ, "KR_DERIV_SUMS": value, "PYTHONPATH": str(root)})
        out.append(np.load(f))
    assert np.array_equal(out[0], out[1])
    for a, b in zip(out[0], out[2]):
        # 32 terms a sum in another order, after a 60-term contraction: 1e-12 of the largest
        assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()
        assert not np.array_equal(a, b)
