"""The Bessel sum reads its J0 table inside its bounds whatever the sign and order of the
slownesses (csrc/kr_bessel.cuh walked on the host, tile by tile)."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
N = 25  # intervals of the table


@pytest.fixture(scope="module")
def intervals(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    so = tmp_path_factory.mktemp("bessel") / "libkr_bessel_emulate.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so),
                    str(HERE / "cpu_emulation" / "kr_bessel_emulate.cpp")], check=True)
    f = ctypes.CDLL(str(so)).emu_bessel_intervals

    def call(p, om, r):
        out = np.zeros(3, dtype=np.int32)
        p = np.ascontiguousarray(p)
        f(ctypes.c_void_p(p.ctypes.data), len(p), ctypes.c_double(om), ctypes.c_double(r), N,
          ctypes.c_void_p(out.ctypes.data))
        return out

    return call


@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 200])
@pytest.mark.parametrize("lo,hi", [(-0.6, 0.6), (-1.2, -0.1), (-0.6, 0.0), (0.0, 0.6), (-1e-3, 1.2),
                                   (0.6, -0.6)])
@pytest.mark.parametrize("omr", [0.0, 0.3, 12.0, 41.0, 700.0, -12.0])
def test_table_index_in_bounds(intervals, n, lo, hi, omr):
    p = np.linspace(lo, hi, n)
    least, most, rising = intervals(p, abs(omr), float(np.sign(omr)))
    assert least >= 0 and most < N, (least, most)
    if lo >= 0.0 and hi > lo and omr >= 0.0:
        assert rising > 0  # ascending slownesses from zero up keep the fast ways
    if hi < 0.0 or hi < lo:
        assert rising == 0


def test_interval_and_offset(intervals):
    """Every x in [0, 25) falls on an interval whose centre is within half a unit (plus rounding)."""
    for x in np.r_[0.0, -0.0, 5e-324, np.arange(0, 25), np.nextafter(np.arange(1.0, 26.0), 0.0),
                   np.random.default_rng(0).uniform(0, 25, 500)]:
        least, most, _ = intervals(np.array([x]), 1.0, 1.0)
        assert least == most and 0 <= least < N
        assert abs(x - (least + 0.5)) <= 0.5
