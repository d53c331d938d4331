"""Derivatives at frequencies whose phases grow with depth (negative real part, thick attenuating
layers): the kernels' adjoint sweep under g++ against differences of their forward sweep.

Tolerance: steps of 1e-5 of a parameter turn phases by up to omega eta h 1e-5 ~ 1e-3, and by ten
times that near a turning point (0.55 s/km against 1.8 km/s), so fourth-order differences are off by
up to (1e-2)^4; the forward's rounding adds 1e-13 / 1e-3.  1e-6 of the largest entry covers both.  (The full-matrix form loses eight digits at
these phases even in 80 bits and is no reference here.)"""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    so = tmp_path_factory.mktemp("grow") / "libkr_emulate.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so),
                    str(HERE / "cpu_emulation" / "kr_emulate.cpp")], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("layers,fs", [(5, 0), (5, 1), (9, 0), (70, 0)])
def test_adjoint_at_negative_frequencies(emu, layers, fs):
    from seismicinversion_b200.earth_models import default_ocean_crust_model, random_layered_model
    from seismicinversion_b200.layer_model import pack_layers

    ptr = lambda x: ctypes.c_void_p(x.ctypes.data)  # noqa: E731
    m = default_ocean_crust_model() if layers == 5 else random_layered_model(layers - 1, seed=3)
    tab = np.ascontiguousarray(pack_layers(m))
    tab[3, :-1] *= 20.0 if layers < 70 else 4.0
    L = layers
    p = np.array([0.03, 0.2, 0.55])
    w = -np.arange(1, 34, 4) * 0.098 + 0.05j
    n, nw = len(p), len(w)
    R = np.zeros((n, nw), dtype=np.complex128)
    J = np.zeros((n, 4 * L, nw), dtype=np.complex128)
    emu.emu_jacobian(ptr(tab), L, ptr(p), n, ptr(w), nw, fs, ptr(R), ptr(J))

    def forward(t):
        t, out = np.ascontiguousarray(t), np.zeros((n, nw), dtype=np.complex128)
        emu.emu_reflectivity(ptr(t), L, ptr(p), n, ptr(w), nw, fs, ptr(out))
        return out

    want = np.zeros_like(J)
    for k in range(4):
        for l in range(L):
            d = 1e-5 * tab[k, l]
            if d == 0.0 or not d < 1e20:
                continue
            for o, c in ((2, -1.0), (1, 8.0), (-1, -8.0), (-2, 1.0)):
                t = tab.copy()
                t[k, l] += o * d
                want[:, k * L + l] += c / (12.0 * d) * forward(t)
    assert np.abs(J - want).max() <= 1e-6 * np.abs(want).max()
    rng = np.random.default_rng(1)
    gR = rng.standard_normal((n, nw)) + 1j * rng.standard_normal((n, nw))
    out = np.zeros(4 * L + 1)
    emu.emu_gradient_sums(ptr(tab), L, ptr(p), n, ptr(w), nw, fs, 1, ptr(gR), ptr(out))
    g = (np.conj(gR)[:, None, :] * J).real.sum((0, 2))
    assert np.abs(out[:-1] - g).max() <= 1e-12 * np.abs(g).max()
