"""Performance cases of the framework: what its users have it compute, at the sizes they use.

Every case goes through a public entry point, with inputs made from a seed alone.  The kinds,
and what each stands for:

``single``    ``kennett_reflectivity`` at one slowness: an interactive trace, a check of one model.
``grid``      ``kennett_reflectivity_batch``: the (slowness x frequency) grid of one model.
``gather``    ``compute_gather_gpu``: host model in, multi-offset traces out (grid, Bessel sum, FFT).
``gradient``  ``device.misfit_gradient``: one tau-p misfit and gradient, the step of a descent.
``autograd``  ``kennett_reflectivity_torch`` forward and ``backward`` of a loss written in torch.
``jacobian``  ``device.jacobian``: the sensitivities of a Gauss-Newton iteration.
``hessian``   ``taup_misfit_grad_hessian``: misfit, gradient and exact Hessian of an LM iteration.
``batch``     ``ModelBatch``: many models of uneven size, forward and forward + gradient mixed.
``training``  ``ModelBatch.from_tables``: a chunk of prior samples of one layer count, as the
              training-data generator evaluates it (new tables each time).
``gmm``       ``device.gmm_reflectivity``: the same grid by the global-matrix method.

Models are water over random crust (``earth_models``: 3 to 64 layers) or perturbations of the
5-layer default model.  Observed data are a few decaying arrivals.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from seismicinversion_b200 import device as kd
from seismicinversion_b200.batch import BatchItem, ModelBatch
from seismicinversion_b200.earth_models import default_ocean_crust_model, random_layered_model
from seismicinversion_b200.kennett_gather_gpu import compute_gather_gpu
from seismicinversion_b200.kennett_reflectivity import kennett_reflectivity
from seismicinversion_b200.kennett_reflectivity_gpu import kennett_reflectivity_batch
from seismicinversion_b200.kennett_torch import kennett_reflectivity_torch, model_to_tensors
from seismicinversion_b200.layer_model import LayerModel, pack_layers
from seismicinversion_b200.source import ricker_spectrum
from seismicinversion_b200.taup_inversion import taup_misfit_grad_hessian

_T = 64.0  # record length of every grid, s
_C, _F = torch.complex128, torch.float64


def listed() -> list[dict]:
    return [
        # the smallest call: one trace of the 6-layer model; launches and host latency count
        {"name": "single_trace", "kind": "single", "layers": 6, "np": 1, "nw": 2047, "fs": False},
        # the gather's grid of the 5-layer default model (layers 0: that model, perturbed)
        {"name": "grid_default", "kind": "grid", "layers": 0, "np": 4096, "nw": 2047,
         "p_max": 1.2, "damped": True, "fs": False},
        # a finely layered model on a ragged grid
        {"name": "grid_deep", "kind": "grid", "layers": 64, "np": 193, "nw": 1501,
         "p_max": 0.8, "damped": False, "fs": True},
        # the headline gather: 21 layers, 8192 slownesses, 100 offsets 0.5-50 km
        {"name": "gather_full", "kind": "gather", "layers": 21, "np": 8192, "nw": 2047,
         "offsets": 100, "r_max": 50.0, "fs": True},
        # a quick look: short grid, few offsets, default model
        {"name": "gather_small", "kind": "gather", "layers": 0, "np": 2048, "nw": 511,
         "offsets": 37, "r_max": 30.0, "fs": False},
        # one gradient of the 79-parameter tau-p inversion
        {"name": "gradient", "kind": "gradient", "layers": 21, "np": 64, "nw": 1024, "fs": False},
        # a torch training step on a ragged grid
        {"name": "autograd", "kind": "autograd", "layers": 12, "np": 201, "nw": 777, "fs": True},
        # Gauss-Newton sensitivities of the same inversion
        {"name": "jacobian", "kind": "jacobian", "layers": 21, "np": 64, "nw": 1024, "fs": False},
        # one exact-Hessian LM iterate of the same inversion
        {"name": "hessian", "kind": "hessian", "layers": 21, "np": 64, "nw": 1024},
        # uneven models in one launch, half of them with gradients
        {"name": "batch_uneven", "kind": "batch", "models": 96, "l_min": 3, "l_max": 64},
        # a chunk of amortised-inference training samples
        {"name": "training_chunk", "kind": "training", "layers": 0, "models": 4096, "np": 12,
         "nw": 64},
        # the independent global-matrix evaluation of a mid-sized grid
        {"name": "gmm_grid", "kind": "gmm", "layers": 21, "np": 1024, "nw": 1023, "p_max": 1.0,
         "fs": True},
    ]


def draw(rng) -> dict:
    def size(lo: int, hi: int) -> int:  # spread over the logarithm, any integer
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["single", "grid", "grid", "gather", "gather", "gradient", "gradient",
                       "autograd", "jacobian", "hessian", "batch", "training", "gmm"])
    c = {"kind": kind}
    if kind == "batch":
        return {**c, "models": size(4, 96), "l_min": 3, "l_max": rng.randint(8, 64)}
    if kind == "training":
        return {**c, "layers": rng.choice([0, rng.randint(4, 12)]), "models": size(64, 4096),
                "np": rng.randint(4, 12), "nw": rng.randint(32, 64)}
    deep = {"single": 64, "grid": 64, "gather": 30, "gradient": 48, "autograd": 32,
            "jacobian": 30, "hessian": 21, "gmm": 30}[kind]
    c["layers"] = rng.choice([0, rng.randint(3, deep), rng.randint(3, deep)])
    if kind != "hessian":
        c["fs"] = rng.random() < 0.5
    if kind == "single":
        return {**c, "np": 1, "nw": size(63, 4095)}
    if kind == "gather":
        return {**c, "np": size(512, 6000), "nw": size(255, 2047), "offsets": size(1, 100),
                "r_max": rng.uniform(5.0, 50.0)}
    if kind == "grid":
        return {**c, "np": size(16, 4096), "nw": size(63, 2047), "p_max": rng.uniform(0.4, 1.2),
                "damped": rng.random() < 0.5}
    if kind == "gmm":
        return {**c, "np": size(16, 1024), "nw": size(63, 1023), "p_max": rng.uniform(0.4, 1.0)}
    if kind == "hessian":
        return {**c, "np": size(4, 64), "nw": size(32, 1024)}
    return {**c, "np": size(4, 128), "nw": size(64, 1024)}


# -- inputs ------------------------------------------------------------------------------

def _model(layers: int, seed: int) -> LayerModel:
    if layers:
        return random_layered_model(layers - 1, seed=seed)
    m = default_ocean_crust_model()
    rng = np.random.default_rng(seed)
    f = rng.uniform(0.9, 1.1, (4, m.n_layers))
    f[:, 0] = 1.0  # the water stays as it is
    return LayerModel.from_arrays(m.alpha * f[0], m.beta * f[1], m.rho * f[2],
                                  m.thickness * f[3], m.Q_alpha, m.Q_beta)


def _grid(case: dict) -> tuple[np.ndarray, np.ndarray]:
    """Slownesses and frequencies (real or damped) of a case, in 64 bits."""
    n, nw = case["np"], case["nw"]
    omega = np.arange(1, nw + 1, dtype=np.float64) * (2.0 * np.pi / _T)
    if case["kind"] == "single":
        return np.array([0.2]), omega
    if case["kind"] == "gather":
        dp = 1.2 / n
        return np.arange(1, n + 1, dtype=np.float64) * dp, omega + 1j * np.pi / _T
    if case["kind"] in ("grid", "gmm"):
        p = np.arange(1, n + 1, dtype=np.float64) * (case["p_max"] / n)
        return p, omega + 1j * np.pi / _T if case.get("damped") else omega
    return np.linspace(0.05, 0.6, n), omega


def _observed(p, omega, seed: int) -> torch.Tensor:
    """Observed R(p, omega): six arrivals of random amplitude and hyperbolic delay (device)."""
    rng = np.random.default_rng(seed + 7)
    p = torch.as_tensor(p, device="cuda").to(_C).reshape(-1, 1)
    w = torch.as_tensor(omega, device="cuda").to(_C).reshape(1, -1)
    out = torch.zeros((p.shape[0], w.shape[1]), dtype=_C, device="cuda")
    for a, tau, v in zip(rng.normal(0.0, 0.2, 6), rng.uniform(1.0, 8.0, 6), rng.uniform(1.5, 3.0, 6)):
        out += a * torch.exp(1j * w * tau * torch.sqrt(1.0 - (p * v) ** 2 + 0.02j))
    return out


def _offsets(case: dict) -> np.ndarray:
    n = case["offsets"]
    return case["r_max"] * np.arange(1, n + 1, dtype=np.float64) / n


def _specs(case: dict, seed: int) -> list[tuple]:
    """(model, p, omega, gradient, free surface) of every model of a batch.  The shapes are the
    case's own, whatever the seed; the models' parameters come from the seed."""
    shapes = np.random.default_rng(1000 + case["models"])
    out = []
    for i in range(case["models"]):
        layers = int(shapes.integers(case["l_min"], case["l_max"] + 1))
        nw = int(shapes.choice([256, 512, 1024, 2048]))
        n = int(shapes.integers(16, 257))
        w = np.arange(1, nw + 1, dtype=np.float64) * (2.0 * np.pi / _T)
        p = np.arange(1, n + 1, dtype=np.float64) * (0.8 / n)
        out.append((_model(layers, seed * 1009 + i), p, w, i % 2 == 1, i % 4 < 2))
    return out


def _tables(case: dict, seed: int) -> np.ndarray:
    """Layer tables [n, 6, L]: prior samples around one model, the water and Q fixed."""
    base = pack_layers(_model(case["layers"], seed))
    rng = np.random.default_rng(seed)
    f = rng.uniform(0.8, 1.2, (case["models"], *base.shape))
    f[:, 2] = 1.0 + 0.75 * (f[:, 2] - 1.0)
    f[:, 4:] = 1.0
    f[:, :, 0] = 1.0
    return base[None] * f


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "batch":
        items = []
        for i, (m, p, w, grad, fs) in enumerate(_specs(case, seed)):
            obs = _observed(p, w, seed + i) if grad else None
            items.append(BatchItem(m, p, w, gradient=grad, R_obs=obs, free_surface=fs))
        st["batch"] = ModelBatch(items, schedule=(128, 2048))
        return st
    p, omega = _grid(case)
    if kind == "training":
        return {**st, "tables": _tables(case, seed), "p": p, "omega": omega}
    model = _model(case["layers"], seed)
    st["model"] = model
    if kind == "gather":
        return {**st, "offsets": _offsets(case)}
    st["p"] = torch.as_tensor(p, device="cuda")
    st["omega"] = torch.as_tensor(omega, device="cuda").to(_C)
    if kind in ("gradient", "jacobian", "gmm"):
        st["layers"] = kd.layer_table(model)
    if kind in ("gradient", "autograd", "hessian"):
        st["obs"] = _observed(p, omega, seed)
    if kind == "autograd":
        t = {k: v.cuda() for k, v in model_to_tensors(model).items()}
        st["theta"] = [t[k].requires_grad_(True) for k in ("alpha", "beta", "rho", "thickness")]
        st["q"] = [t["Q_alpha"], t["Q_beta"]]
    if kind == "hessian":
        st["tensors"] = model_to_tensors(model)
        st["p"] = p
        st["log"] = _log_params(pack_layers(model))
    return st


def _log_params(tab: np.ndarray) -> np.ndarray:
    return np.log(np.concatenate([tab[0, 1:], tab[1, 1:], tab[2, 1:], tab[3, 1:-1]]))


def run(st: dict):
    kind, case = st["kind"], st["case"]
    if kind == "single":
        return kennett_reflectivity(st["model"], 0.2, st["omega"], free_surface=case["fs"])
    if kind == "grid":
        return kennett_reflectivity_batch(st["model"], st["p"], st["omega"],
                                          free_surface=case["fs"])
    if kind == "gather":
        _, _, g = compute_gather_gpu(st["model"], st["offsets"], T=_T, nw=case["nw"] + 1,
                                     np_slow=case["np"], free_surface=case["fs"])
        return g
    if kind == "gradient":
        return kd.misfit_gradient(st["layers"], st["p"], st["omega"], st["obs"], case["fs"])[0]
    if kind == "autograd":
        R = kennett_reflectivity_torch(*st["theta"], *st["q"], st["p"], st["omega"],
                                       free_surface=case["fs"])
        r = R - st["obs"]
        loss = (r.real ** 2 + r.imag ** 2).sum()
        return {"R": R.detach(), "grad": torch.autograd.grad(loss, st["theta"])}
    if kind == "jacobian":
        R, J = kd.jacobian(st["layers"], st["p"], st["omega"], case["fs"])
        return {"R": R, "J": J}
    if kind == "hessian":
        t = st["tensors"]
        chi, g, H = taup_misfit_grad_hessian(
            st["log"], t["alpha"], t["beta"], t["rho"], t["thickness"], t["Q_alpha"],
            t["Q_beta"], st["p"], st["omega"], st["obs"])
        return {"chi": chi, "gradient": g, "hessian": H}
    if kind == "batch":
        st["batch"].launch()
        return {"R": st["batch"].R, "chi_grad": st["batch"].chi_grad}
    if kind == "training":
        b = ModelBatch.from_tables(st["tables"], st["p"], st["omega"])
        b.launch()
        return b.R
    return kd.gmm_reflectivity(st["layers"], st["p"], st["omega"], case["fs"])


# -- work --------------------------------------------------------------------------------
# Flops of one (omega, p, interface) update: the Kennett step in its shortest known real form
# (phases 24, one reciprocal 14, 2 x 2 symmetric algebra 162), its reverse step about twice
# that; a J0 term of the Bessel sum 6 (given the J0 value, which costs about 24).

_STEP, _REVERSE, _BESSEL = 200.0, 400.0, 30.0


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for m, p, w, grad, _ in _specs(case, 0):
            n = float(len(p) * len(w))
            b += 48.0 * m.n_layers + 8 * len(p) + 16 * len(w) + 16 * n
            f += n * (m.n_layers - 1) * (_STEP + (_REVERSE if grad else 0.0))
        return {"bytes": b, "flops": f}
    L = case["layers"] or 5
    n, grid = case["np"] * case["nw"], 8.0 * case["np"] + 16.0 * case["nw"]
    up = float(n) * (L - 1)
    if kind == "training":
        return {"bytes": case["models"] * (48.0 * L + 16.0 * n) + grid,
                "flops": case["models"] * up * _STEP}
    if kind == "gather":
        r = case["offsets"]
        return {"bytes": 48.0 * L + grid + 8.0 * r + 16.0 * r * (case["nw"] + 1),
                "flops": up * _STEP + _BESSEL * n * r}
    if kind in ("single", "grid", "gmm"):
        return {"bytes": 48.0 * L + grid + 16.0 * n, "flops": up * _STEP}
    if kind == "jacobian":
        return {"bytes": 48.0 * L + grid + 16.0 * n * (4 * L + 1),
                "flops": up * (_STEP + _REVERSE + 480.0)}
    if kind == "hessian":
        # per (omega, p): the gradient's sweeps and one 3-vector chain per pair of layers
        P = 4 * L - 5
        return {"bytes": 48.0 * L + grid + 16.0 * n + 8.0 * P * P,
                "flops": up * (_STEP + _REVERSE) + n * 0.5 * P * P * 24.0}
    out = 16.0 * n if kind == "autograd" else 0.0
    return {"bytes": 48.0 * L + grid + 16.0 * n + out + 32.0 * L,
            "flops": up * (_STEP + _REVERSE)}


# -- 64-bit values -----------------------------------------------------------------------

def _reflect(par, qa, qb, p, w, fs: bool):
    """R by the Kennett recursion in plain torch, complex128.  ``par`` is (alpha, beta, rho, h),
    each a list over layers of tensors that broadcast against p [np, 1] and w [nw]; the last
    layer is the half-space, layer 0 the water."""
    al, be, rh, h = par
    L = len(al)

    def slow(v, q):
        den = (1.0 + 4.0 * q * q) * v
        return torch.complex(4.0 * q * q / den, 2.0 * q / den)

    def vert(s):
        e = torch.sqrt((s + p) * (s - p))
        return torch.where(e.imag.detach() <= 0.0, -e, e)

    eta = [vert(slow(al[i], qa[i])) for i in range(L)]
    ss = [None] + [slow(be[i], qb[i]) for i in range(1, L)]
    neta = [None] + [vert(ss[i]) for i in range(1, L)]
    bc = [None] + [1.0 / ss[i] for i in range(1, L)]
    rho = [r.to(_C) for r in rh]
    q = p * p

    def coefficients(i):
        e1, e2, n2, r1, r2 = eta[i], eta[i + 1], neta[i + 1], rho[i], rho[i + 1]
        mu2 = r2 * bc[i + 1] * bc[i + 1]
        za1, za2, zb2 = torch.sqrt(e1) * torch.sqrt(r1), torch.sqrt(e2) * torch.sqrt(r2), \
            torch.sqrt(n2) * torch.sqrt(r2)
        if i == 0:
            d = 2.0 * mu2
            a, b, c = (r2 - r1) - q * d, r2 - q * d, r1 + q * d
            E, F, G, H = b * e1 + c * e2, b, a - d * e1 * n2, -d * e2
            D = E * F + G * H * q
            E, F, G, H = E / D, F / D, G / D, H / D
            t1, t2, t4 = (b * e1 - c * e2) * F, (a + d * e1 * n2) * H * q, b * E
            t5, t6 = d * e2 * G * q, b * d * e1 * p / D
            z = torch.zeros_like(t1)
            return (t1 - t2, z, z, -(t1 + t5),
                    -2j * torch.sqrt(e2) * torch.sqrt(n2) * t6, -(t2 + t4),
                    2.0 * za1 * za2 * F, z, -2j * za1 * zb2 * H * p, z)
        n1 = neta[i]
        zb1 = torch.sqrt(n1) * torch.sqrt(r1)
        d = 2.0 * (mu2 - r1 * bc[i] * bc[i])
        a, b, c = (r2 - r1) - q * d, r2 - q * d, r1 + q * d
        E, F = b * e1 + c * e2, b * n1 + c * n2
        G, H = a - d * e1 * n2, a - d * e2 * n1
        D = E * F + G * H * q
        E, F, G, H = E / D, F / D, G / D, H / D
        Qv, Rv = (b * e1 - c * e2) * F, (a + d * e1 * n2) * H * q
        Sv = (a * b + c * d * e2 * n2) * p / D
        Tv, Uv = (b * n1 - c * n2) * E, (a + d * e2 * n1) * G * q
        Vv = (a * c + b * d * e1 * n1) * p / D
        return (Qv - Rv, -2j * torch.sqrt(e1) * torch.sqrt(n1) * Sv, Tv - Uv, -(Qv + Uv),
                -2j * torch.sqrt(e2) * torch.sqrt(n2) * Vv, -(Tv + Rv),
                2.0 * za1 * za2 * F, -2j * zb1 * za2 * G * p, -2j * za1 * zb2 * H * p,
                2.0 * zb1 * zb2 * E)

    x11 = x12 = x22 = None
    for i in range(L - 2, -1, -1):
        d11, d12, d22, u11, u12, u22, t11, t12, t21, t22 = coefficients(i)
        if x11 is None:  # nothing comes back from the half-space
            one = torch.ones_like(w * p)
            x11, x12, x22 = d11 * one, d12 * one, d22 * one
            continue
        ea = torch.exp(1j * w * eta[i + 1] * h[i + 1])
        eb = torch.exp(1j * w * neta[i + 1] * h[i + 1])
        m11, m12, m22 = ea * ea * x11, ea * eb * x12, eb * eb * x22
        # Y = M (I - Ru M)^-1 = (M - det(M) adj(Ru)) / det: the 2 x 2 adjugate is linear
        dm = m11 * m22 - m12 * m12
        det = 1.0 - u11 * m11 - 2.0 * u12 * m12 - u22 * m22 + (u11 * u22 - u12 * u12) * dm
        y11, y12, y22 = (m11 - u22 * dm) / det, (m12 + u12 * dm) / det, (m22 - u11 * dm) / det
        x11 = d11 + t11 * t11 * y11 + 2.0 * t11 * t21 * y12 + t21 * t21 * y22
        x12 = d12 + t11 * t12 * y11 + (t11 * t22 + t21 * t12) * y12 + t21 * t22 * y22
        x22 = d22 + t12 * t12 * y11 + 2.0 * t12 * t22 * y12 + t22 * t22 * y22
    e0 = torch.exp(1j * w * eta[0] * h[0])
    y = e0 * e0 * x11
    return y / (1.0 + y) if fs else y


def _params(tab: np.ndarray):
    """(alpha, beta, rho, h) and (Q_alpha, Q_beta) as lists of 0-d tensors."""
    t = torch.as_tensor(tab, device="cuda")
    return [list(t[k].unbind(-1)) for k in range(4)], t[4].unbind(-1), t[5].unbind(-1)


def _plain(tab, p, w, fs: bool, rows: int = 512) -> torch.Tensor:
    par, qa, qb = _params(tab)
    return torch.cat([_reflect(par, qa, qb, p[a:a + rows], w, fs)
                      for a in range(0, p.shape[0], rows)])


def _chi_gradient(tab, p, w, obs, fs: bool):
    """chi, [4L] gradient (alpha, beta, rho, h) and R by torch's reverse mode."""
    par, qa, qb = _params(tab)
    free = [x.clone().requires_grad_(True) for k in range(4) for x in par[k]]
    L = len(qa)
    with torch.enable_grad():
        R = _reflect([free[k * L:(k + 1) * L] for k in range(4)], qa, qb, p, w, fs)
        r = R - obs
        chi = (r.real ** 2 + r.imag ** 2).sum()
        g = torch.autograd.grad(chi, free, allow_unused=True)
    g = torch.stack([torch.zeros((), dtype=_F, device="cuda") if x is None else x for x in g])
    return chi.detach(), g, R.detach()


def exact(case: dict, seed: int):
    kind, fs = case["kind"], case.get("fs", False)
    if kind == "batch":
        Rs, cg = [], []
        for i, (m, p, w, grad, fs) in enumerate(_specs(case, seed)):
            pt = torch.as_tensor(p, device="cuda").reshape(-1, 1)
            wt = torch.as_tensor(w, device="cuda").to(_C)
            if grad:
                chi, g, _ = _chi_gradient(pack_layers(m), pt, wt, _observed(p, w, seed + i), fs)
                cg += [g, chi.reshape(1)]
            else:
                Rs.append(_plain(pack_layers(m), pt, wt, fs).reshape(-1))
        return {"R": torch.cat(Rs) if Rs else None, "chi_grad": torch.cat(cg) if cg else None}
    p, omega = _grid(case)
    p = torch.as_tensor(p, device="cuda").reshape(-1, 1)
    w = torch.as_tensor(omega, device="cuda").to(_C)
    if kind == "training":
        t = torch.as_tensor(_tables(case, seed), device="cuda")
        col = [list(x[..., None, None] for x in t[:, k].unbind(-1)) for k in range(6)]
        return _reflect(col[:4], col[4], col[5], p, w, False).reshape(-1)
    tab = pack_layers(_model(case["layers"], seed))
    if kind == "single":
        return _plain(tab, p, w, fs)[0]
    if kind in ("grid", "gmm"):
        return _plain(tab, p, w, fs)
    if kind == "gather":
        return _plain_gather(case, tab, p, w, fs)
    if kind == "gradient":
        chi, g, _ = _chi_gradient(tab, p, w, _observed(p.cpu(), w, seed), fs)
        return torch.cat([g, chi.reshape(1)])
    if kind == "autograd":
        _, g, R = _chi_gradient(tab, p, w, _observed(p.cpu(), w, seed), fs)
        L = tab.shape[1]
        return {"R": R, "grad": tuple(g[k * L:(k + 1) * L] for k in range(4))}
    if kind == "jacobian":
        return _plain_jacobian(tab, p, w, fs)
    return _plain_hessian(tab, p, w, _observed(p.cpu(), w, seed))


def _j0(x):
    """J0(x), x >= 0, to a few 1e-16 (torch.special.bessel_j0 is only good to 4e-7): Bessel's
    integral by its midpoint rule below 25, Hankel's expansion from there on."""
    near = x < 25.0
    xn = x[near]
    lo = sum(torch.cos(xn * math.cos(math.pi * (k + 0.5) / 80)) for k in range(40)) / 40
    a = [1.0]
    for k in range(1, 20):
        a.append(-a[-1] * (2 * k - 1) ** 2 / (8 * k))
    y = 1.0 / x.clamp(min=25.0)
    P, Q = torch.zeros_like(x), torch.zeros_like(x)
    for m in range(9, -1, -1):
        P = P * y * y + (-1) ** m * a[2 * m]
        Q = Q * y * y + (-1) ** m * a[2 * m + 1]
    out = torch.sqrt(y / math.pi) * ((P + Q * y) * torch.cos(x) + (P - Q * y) * torch.sin(x))
    out[near] = lo
    return out


def _plain_gather(case: dict, tab, p, w, fs: bool) -> np.ndarray:
    n, nw = case["np"], case["nw"] + 1
    R = _plain(tab, p, w, fs)
    wr, dp = w.real, 1.2 / n
    taper = 0.5 * (1.0 + torch.cos(math.pi * p / 1.2))
    Rw = R * (taper * p * wr * dp)
    x = p * wr
    S = torch.as_tensor(ricker_spectrum(wr.cpu().numpy(), nw * 2.0 * np.pi / _T), device="cuda")
    time = torch.arange(2 * nw, dtype=_F, device="cuda") * (_T / (2 * nw))
    out = []
    for r in _offsets(case):
        Y = (Rw * _j0(x * float(r))).sum(0) * S
        z = torch.zeros(1, dtype=_C, device="cuda")
        spec = torch.cat([z, Y, z, Y.flip(0).conj()])
        out.append(torch.fft.fft(spec).real * torch.exp(-math.pi / _T * time))
    return torch.stack(out).cpu().numpy()


def _plain_jacobian(tab, p, w, fs: bool) -> dict:
    """Every (p, omega) gets its own copy of the parameters: two reverse passes (of Re R and
    Im R) give dR / d theta everywhere."""
    par, qa, qb = _params(tab)
    L, Rs, Js = len(qa), [], []
    for a in range(0, p.shape[0], 16):
        pc = p[a:a + 16]
        one = torch.ones((pc.shape[0], w.shape[0]), dtype=_F, device="cuda")
        free = [(x * one).requires_grad_(True) for k in range(4) for x in par[k]]
        with torch.enable_grad():
            R = _reflect([free[k * L:(k + 1) * L] for k in range(4)], qa, qb, pc, w, fs)
            gr = torch.autograd.grad(R.real.sum(), free, allow_unused=True, retain_graph=True)
            gi = torch.autograd.grad(R.imag.sum(), free, allow_unused=True)
        z = torch.zeros_like(one)
        Js.append(torch.stack([torch.complex(z if u is None else u, z if v is None else v)
                               for u, v in zip(gr, gi)], dim=1))
        Rs.append(R.detach())
    return {"R": torch.cat(Rs), "J": torch.cat(Js)}


def _plain_hessian(tab, p, w, obs) -> dict:
    """chi, gradient and Hessian over log parameters: forward over reverse, a few slownesses at
    a time."""
    L = tab.shape[1]
    t = torch.as_tensor(tab, device="cuda")
    x0 = torch.as_tensor(_log_params(tab), device="cuda")
    n = L - 1

    def chi(x, pc, oc):
        m = torch.exp(x)
        par = [[t[k, 0]] + list(m[k * n:(k + 1) * n].unbind(0)) for k in range(3)]
        par.append([t[3, 0]] + list(m[3 * n:].unbind(0)) + [t[3, -1]])
        r = _reflect(par, t[4].unbind(-1), t[5].unbind(-1), pc, w, False) - oc
        return (r.real ** 2 + r.imag ** 2).sum()

    step = max(1, 4096 // w.shape[0])
    c = torch.zeros((), dtype=_F, device="cuda")
    g, H = torch.zeros_like(x0), torch.zeros((x0.shape[0],) * 2, dtype=_F, device="cuda")
    with torch.enable_grad():
        for a in range(0, p.shape[0], step):
            pc, oc = p[a:a + step], obs[a:a + step]

            def grad_chi(x):
                gx, cx = torch.func.grad_and_value(chi)(x, pc, oc)
                return gx, (gx, cx)

            h, (gx, cx) = torch.func.jacfwd(grad_chi, has_aux=True)(x0)
            H, g, c = H + h.detach(), g + gx.detach(), c + cx.detach()
    return {"chi": float(c), "gradient": g.cpu().numpy(), "hessian": H.cpu().numpy()}
