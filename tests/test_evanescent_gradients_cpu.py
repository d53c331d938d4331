"""Gradients where the water layer is evanescent and its phase underflows gradually: the complex
root at the ends of the range, and the frequency sums of the adjoint (kernel code under g++)."""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("root")

    def build(name):
        so = out / f"lib{name}.so"
        subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so),
                        str(HERE / "cpu_emulation" / f"{name}.cpp")], check=True)
        return ctypes.CDLL(str(so))

    return build


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def test_csqrt_over_the_whole_range(lib):
    tiny, huge = 5e-324, np.finfo(float).max
    parts = [0.0, tiny, 3 * tiny, 1e-310, 2.3e-308, 1e-290, 1e-160, 1.0, 1e160, 1e300, huge]
    z = np.array([complex(sx * x, sy * y) for x in parts for y in parts
                  for sx in (1, -1) for sy in (1, -1)])
    out = np.zeros_like(z)
    lib("kr_root_emulate").emu_csqrt_any(_ptr(z), len(z), _ptr(out))
    want = np.sqrt(z.astype(np.clongdouble))
    assert np.all(np.isfinite(out.real) & np.isfinite(out.imag))
    # a few roundings; the smaller part may itself be subnormal (an ulp of 4.9e-324)
    for a, b in ((out.real, want.real), (out.imag, want.imag)):
        assert np.all(np.abs(a - b) <= 1e-15 * np.abs(b) + 5e-324)
        nz = b != 0
        assert np.array_equal(np.signbit(a[nz]), np.signbit(b[nz]))


@pytest.mark.parametrize("fs", [0, 1])
@pytest.mark.parametrize("vjp", [0, 1])
def test_gradient_sums_are_finite(lib, fs, vjp):
    from seismicinversion_b200.earth_models import default_ocean_crust_model
    from seismicinversion_b200.layer_model import pack_layers

    emu = lib("kr_emulate")
    tab = np.ascontiguousarray(pack_layers(default_ocean_crust_model()))
    L, nw = tab.shape[1], 2047
    p = np.linspace(0.05, 1.2, 64)[58:]  # from 1.11 on: the water phase reaches the subnormals
    w = (np.arange(1, nw + 1) * (2 * np.pi / 64)).astype(np.complex128)
    rng = np.random.default_rng(0)
    obs = rng.standard_normal((len(p), nw)) + 1j * rng.standard_normal((len(p), nw))
    out = np.zeros(4 * L + 1)
    emu.emu_gradient_sums(_ptr(tab), L, _ptr(p), len(p), _ptr(w), nw, fs, vjp, _ptr(obs), _ptr(out))
    assert np.all(np.isfinite(out))
