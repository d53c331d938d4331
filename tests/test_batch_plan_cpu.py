"""The batch plan's work lists (host only): every (pair, frequency range) once, by descending
cost and, at equal cost, in model order; tables are validated in one call with the same errors."""

import ctypes

import numpy as np
import pytest

from seismicinversion_b200 import _lib
from seismicinversion_b200 import device as D

HEADER = np.dtype([("n", "<i4", 4), ("cfg", "<i4", 4), ("off", "<i8", 5)])
ITEM = np.dtype([("pair", "<i4"), ("w0", "<i4"), ("nw", "<i4"), ("pad", "<i4")])


@pytest.mark.parametrize("tile_w", [32, 100, 128, 2048])
def test_work_lists(tile_w):
    rng = np.random.default_rng(tile_w)
    n = 37
    desc = np.zeros(n, dtype=_lib.MODEL_DESC_FIELDS)
    desc["n_layers"] = rng.integers(2, 70, n)
    desc["n_p"] = rng.integers(0, 6, n)
    desc["n_w"] = rng.choice([0, 1, 64, 100, 128, 129, 2048], n)
    desc["flags"] = np.where(np.arange(n) % 2, _lib.KR_BATCH_GRADIENT, 0)
    cfg = _lib.BatchConfig(128, tile_w, 0, 0)
    h = _lib.lib()
    size = h.kr_batch_plan_meta_bytes(desc.ctypes.data, n, ctypes.byref(cfg))
    img = np.zeros(size, np.uint8)
    assert h.kr_batch_plan_host(desc.ctypes.data, n, ctypes.byref(cfg), img.ctypes.data, size) == 0
    head = img[:HEADER.itemsize].view(HEADER)[0]
    n_pairs, n_fwd, n_grad = (int(x) for x in head["n"][1:])
    assert n_pairs == desc["n_p"].sum()
    model = np.repeat(np.arange(n), desc["n_p"])
    for grad, off, count in ((0, head["off"][2], n_fwd), (1, head["off"][3], n_grad)):
        it = img[off:off + count * ITEM.itemsize].view(ITEM)
        want = [(q, w0, min(tile_w, int(desc[m]["n_w"]) - w0))
                for q, m in enumerate(model) if m % 2 == grad
                for w0 in range(0, int(desc[m]["n_w"]), tile_w)]
        got = [(int(i["pair"]), int(i["w0"]), int(i["nw"])) for i in it]
        assert sorted(got) == sorted(want)
        deep = [int(desc[model[q]]["n_layers"]) for q, _, _ in got]
        cost = [(d - 1) * nw for d, (_, _, nw) in zip(deep, got)]
        for a in range(1, len(got)):
            if (deep[a] > 30) == (deep[a - 1] > 30):
                assert cost[a] <= cost[a - 1]
                if cost[a] == cost[a - 1]:
                    assert got[a] > got[a - 1]


def test_validate_tables_reports_the_first_invalid_one():
    tab = np.ones((5, 6, 4))
    tab[:, 1, 0] = 0.0
    D.validate_tables(tab)
    D.validate_tables(tab[:0])
    tab[3, 0, 2] = -1.0
    with pytest.raises(ValueError, match="layer 2: alpha"):
        D.validate_tables(tab)
