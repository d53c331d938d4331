"""The pairwise Hessian's arithmetic (kr_hess.cuh, compiled with g++) against the tangent of the
adjoint (kr_hvp.cuh), direction by direction: the fewest layers, a half-space right below the
ocean, tapes of more than one segment, with and without the free surface."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("hess")
    made = []
    for name in ("kr_hess_emulate", "kr_emulate"):
        so = out / f"lib{name}.so"
        subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so),
                        str(HERE / "cpu_emulation" / f"{name}.cpp")], check=True)
        made.append(ctypes.CDLL(str(so)))
    return made


@pytest.mark.parametrize("n_sub", [1, 2, 3, 6, 20, 70])
@pytest.mark.parametrize("fs", [0, 1])
def test_pairwise_hessian_vs_tangent_of_adjoint(libs, n_sub, fs):
    from seismicinversion_b200.earth_models import random_layered_model
    from seismicinversion_b200.layer_model import pack_layers

    hess, emu = libs
    m = random_layered_model(n_sub, seed=60 + n_sub)
    L, I = n_sub + 1, n_sub
    tab = np.ascontiguousarray(pack_layers(m))
    p = np.array([0.07, 0.31, 0.52])
    w = (np.arange(1, 8) * 0.9 + 0.05j).astype(np.complex128)
    rng = np.random.default_rng(3)
    obs = (rng.normal(size=(3, 7)) + 1j * rng.normal(size=(3, 7))).astype(np.complex128)
    ptr = lambda x: ctypes.c_void_p(x.ctypes.data)  # noqa: E731
    H = np.zeros((4 * I, 4 * I))
    hess.emu_hessian(ptr(tab), L, ptr(p), 3, ptr(w), 7, fs, ptr(obs), ptr(H))
    want = np.zeros_like(H)
    cols = [k * L + l for k in range(4) for l in range(1, L)]
    hv, jd = np.zeros(4 * L), np.zeros(1, dtype=np.complex128)
    for c, full in enumerate(cols):
        v = np.zeros(4 * L)
        v[full] = 1.0
        emu.emu_hvp(ptr(tab), L, ptr(p), 3, ptr(w), 7, fs, ptr(v), 0, ptr(obs), ptr(hv), ptr(jd))
        want[:, c] = hv[cols]
    # the two orders of differentiation round alike per pair: 1e-11 of the largest entry
    assert np.abs(H - want).max() < 1e-11 * np.abs(want).max()
    assert np.array_equal(H, H.T)
