"""The Bessel sum takes falling slownesses the fast ways, and reads its J0 table inside its bounds."""

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
    f = ctypes.CDLL(str(so)).emu_bessel_steady

    def call(p, om, r):
        out = np.zeros(3, dtype=np.int32)
        p = np.ascontiguousarray(p)
        f(ctypes.c_void_p(p.ctypes.data), len(p), ctypes.c_double(om), ctypes.c_double(r), N,
          ctypes.c_void_p(out.ctypes.data))
        return out

    return call


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 200])
@pytest.mark.parametrize("lo,hi", [(0.6, -0.6), (0.6, 0.0), (0.6, 0.01), (-0.1, -1.2), (-0.6, 0.6), (0.0, 0.6),
                                   (0.3, 0.3)])
@pytest.mark.parametrize("omr", [0.0, 0.3, 12.0, 41.0, 700.0, -12.0])
def test_table_index_in_bounds(intervals, n, lo, hi, omr):
    least, most, fast = intervals(np.linspace(lo, hi, n), abs(omr), float(np.sign(omr)))
    assert least >= 0 and most < N, (least, most)
    if max(lo, hi) < 0.0 or lo == hi:
        assert fast == 0


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 200])
def test_falling_progression_takes_the_fast_ways(intervals, n):
    """Slownesses that are multiples of 1/256, so that the progression has no roundings of its own."""
    p = np.arange(n, 0, -1) / 256.0
    assert intervals(p, 41.0, 1.0)[2] == n
    assert intervals(p[::-1], 41.0, 1.0)[2] == n
