"""Workloads of the transform and model-step path, for timing and comparing builds.

Each case is one thing a program does with this package on one GPU, through
its public entry points: transform pairs on device buffers (`ShtPlan.synth_dev`
+ `analys_dev`), round trips on host arrays (`ShtPlan.roundtrip_ptr`), model
steps (`GpuModel.step`) and the forward/backward pair (`GpuModel.forwardBackward`).
`listed` holds the fixed cases, `draw` more of the same ranges; `exact` gives
the outputs in 64-bit arithmetic from the transforms' definition.
"""
import math

import numpy as np
import torch

from turing_sphere_b200 import (GpuModel, ShtConfig, ShtPlan, defaultParams, gridForLmax,
                                mModelByKey, requestShtDevice)
from turing_sphere_b200.layout import gaussGrid
from turing_sphere_b200.registry import brusselatorSweep


def _pair(name, precision, lmax, batch, grid, mmax=None):
    return {"name": name, "kind": "pair", "precision": precision, "lmax": lmax,
            "mmax": lmax if mmax is None else mmax, "nlat": grid[0], "nphi": grid[1],
            "batch": batch}


def _step(name, precision, model, lmax, batch, steps, grid):
    return {"name": name, "kind": "step", "precision": precision, "model": model, "lmax": lmax,
            "mmax": lmax, "nlat": grid[0], "nphi": grid[1], "batch": batch, "steps": steps}


def listed():
    return [
        # one field on the solver's default grid: the transform benchmark's own
        # size and the smallest call a program makes
        _pair("pair_fp32_lmax63_b1", "fp32", 63, 1, (128, 256)),
        # a few fields at the default precision
        _pair("pair_fp32_lmax127_b16", "fp32", 127, 16, gaussGrid(127)),
        # a full batch at the default precision
        _pair("pair_fp32_lmax255_b256", "fp32", 255, 256, gaussGrid(255)),
        # one field on a tensor-core plan (a display field, a single read-back)
        _pair("pair_tf32x3_lmax255_b1", "tf32x3", 255, 1, gaussGrid(255)),
        # the benchmark's headline workload
        _pair("pair_tf32x3_lmax255_b256", "tf32x3", 255, 256, gaussGrid(255)),
        # sizes that fit no tile: odd latitudes, mmax < lmax, a ragged batch
        _pair("pair_tf32x3_lmax170_ragged", "tf32x3", 170, 37, (257, 512), mmax=150),
        # the highest resolution of the benchmark's transform sizes
        _pair("pair_tf32x3_lmax1023_b16", "tf32x3", 1023, 16, gaussGrid(1023)),
        # one interactive simulation at the defaults, 20 steps a frame
        _step("step_fp32_schnakenberg_lmax63_b1", "fp32", "schnakenberg", 63, 1, 20, (96, 192)),
        # a parameter sweep of many instances
        _step("step_tf32x3_brusselator_lmax127_b256", "tf32x3", "brusselator", 127, 256, 4,
              gaussGrid(127)),
        # the benchmark's batched time step
        _step("step_tf32x3_schnakenberg_lmax255_b128", "tf32x3", "schnakenberg", 255, 128, 2,
              gaussGrid(255)),
        # gradients of one simulation: forward, checkpoints, adjoint
        {"name": "adjoint_tf32x3_allencahn_lmax255_b1", "kind": "adjoint", "precision": "tf32x3",
         "model": "allencahn", "lmax": 255, "mmax": 255, "nlat": 384, "nphi": 768, "batch": 1,
         "steps": 16, "every": 8},
        # coefficients in page-locked host memory in, coefficients out
        {"name": "host_tf32x3_lmax255_b64", "kind": "host", "precision": "tf32x3", "lmax": 255,
         "mmax": 255, "nlat": 384, "nphi": 768, "batch": 64},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(["pair", "step", "adjoint", "host"], [6, 3, 1, 1])[0]
    precision = rng.choice(["fp32", "tf32x3"])
    model = None
    if kind in ("step", "adjoint"):
        model = rng.choice(["schnakenberg", "brusselator", "allencahn"])
    hi = {"pair": 1023 if precision == "tf32x3" else 511, "step": 511, "adjoint": 255,
          "host": 511}[kind]
    lmax = _log_int(rng, 31, hi)
    mmax = lmax
    if rng.random() < 0.5 or lmax > 511:  # the benchmark's 3/2 grids, at powers of two
        lmax = min(hi, 2 ** max(5, int(round(math.log2(lmax + 1)))) - 1)
        mmax = lmax
        nlat, nphi = gaussGrid(lmax)
    else:  # the solver's grid rule at any lmax, some with odd latitudes or a lower mmax
        nlat, nphi = gridForLmax(lmax, 3)
        if kind in ("pair", "host"):
            nlat += rng.randrange(2)
            mmax = lmax if rng.random() < 0.7 else rng.randint(lmax // 2, lmax)
    case = {"kind": kind, "precision": precision, "lmax": lmax, "mmax": mmax, "nlat": nlat,
            "nphi": nphi}
    if model:
        case["model"] = model
    if kind == "adjoint":
        case["batch"] = rng.choice([1, 1, 2, 3])
        case["steps"] = rng.choice([4, 8, 12])
        case["every"] = rng.choice([3, 4, 8])
        return case
    nfield = 1 if model in (None, "allencahn") else 2
    budget = 1.6e10 if precision == "fp32" else 3.2e10  # flops of the transforms in a pass
    case["batch"] = 1
    case["steps"] = 1
    most = int(budget / (nfield * _pair_flops(case)))
    case["batch"] = _log_int(rng, 1, max(1, min(256, most)))
    if kind == "step":
        case["steps"] = max(1, min(rng.choice([1, 2, 5, 10, 20]), most // case["batch"]))
    else:
        del case["steps"]
    return case


# ------------------------------------------------------------------- inputs


def _degrees(lmax, mmax):
    """(l, m) of every coefficient in storage order (m-major)."""
    ls = np.concatenate([np.arange(m, lmax + 1) for m in range(mmax + 1)])
    ms = np.concatenate([np.full(lmax + 1 - m, m) for m in range(mmax + 1)])
    return ls, ms


def _spectra(case, seed, count):
    """Seeded Gaussian coefficients scaled by 1/(l+1), (count, 2 nlm) float32
    on the GPU; the imaginary parts of m = 0 are zero."""
    ls, ms = _degrees(case["lmax"], case["mmax"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(count, ls.size, 2, generator=gen, device="cuda")
    q /= torch.from_numpy(ls + 1.0).to("cuda", torch.float32)[None, :, None]
    q[:, torch.from_numpy(ms == 0).cuda(), 1] = 0.0
    return q.reshape(count, -1)


def _params(case):
    """One parameter set per instance."""
    model = mModelByKey(case["model"])
    if case["model"] == "brusselator":
        return brusselatorSweep(case["batch"], seed=3)
    p = defaultParams(model)
    key = "D1" if "D1" in p else "eps2"
    return [dict(p, **{key: p[key] * (1 + 0.5 * k / case["batch"])}) for k in range(case["batch"])]


def _states(case, seed):
    """Initial spectral states, name -> (instances, 2 nlm): the homogeneous
    steady state of each instance plus a seeded perturbation."""
    root = math.sqrt(4 * math.pi)
    out = {}
    for i, name in enumerate(mModelByKey(case["model"]).state):
        u = 0.1 * _spectra(case, 2 * seed + i, case["batch"])
        for k, p in enumerate(_params(case)):
            if case["model"] == "schnakenberg":
                s = p["a"] + p["b"]
                u[k, 0] = root * (s, p["b"] / s ** 2)[i]
            elif case["model"] == "brusselator":
                u[k, 0] = root * (p["A"], p["B"] / p["A"])[i]
        out[name] = u
    return out


class _Buffer:
    """A device array of a model as torch sees foreign CUDA memory."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False),
                                         "version": 2}


def _view(gpu, ptr, n):
    t = torch.as_tensor(_Buffer(ptr, (gpu.batch, n)), device="cuda")
    t.owner = gpu  # the memory is the model's: it lives as long as the tensor
    return t


def prepare(case, seed):
    device = requestShtDevice(0)
    cfg = ShtConfig(case["lmax"], case["mmax"], case["nlat"], case["nphi"])
    plan = ShtPlan.create(device, cfg, {"precision": case["precision"]})
    state = {"kind": case["kind"], "plan": plan, "batch": case["batch"]}
    if case["kind"] == "pair":
        state["q"] = _spectra(case, seed, case["batch"])
        state["grid"] = torch.empty(case["batch"], cfg.nlat * cfg.nphi, device="cuda")
        state["back"] = torch.empty_like(state["q"])
    elif case["kind"] == "host":
        state["q"] = _spectra(case, seed, case["batch"]).cpu().pin_memory()
        state["back"] = torch.empty_like(state["q"]).pin_memory()
    else:
        model = mModelByKey(case["model"])
        gpu = GpuModel.create(device, plan, model.source, [p.key for p in model.params],
                              model.state, model.species, case["batch"])
        gpu.setParams(_params(case))
        for name, u in _states(case, seed).items():
            gpu.upload(name, u.cpu().numpy())
        state.update(gpu=gpu, steps=case["steps"], views={})
        if case["kind"] == "adjoint":
            state["every"] = case["every"]
            state["bar"] = {name: _spectra(case, 2 * seed + 1000003 + i, case["batch"]).cpu().numpy()
                            for i, name in enumerate(model.state)}
    torch.cuda.synchronize()
    return state


# --------------------------------------------------------------------- runs


def run(state):
    plan, batch = state["plan"], state["batch"]
    if state["kind"] == "pair":
        plan.synth_dev(state["q"].data_ptr(), state["grid"].data_ptr(), batch)
        plan.analys_dev(state["grid"].data_ptr(), state["back"].data_ptr(), batch)
        return [state["grid"], state["back"]]
    if state["kind"] == "host":
        plan.roundtrip_ptr(state["q"].data_ptr(), state["back"].data_ptr(), batch)
        return state["back"]
    gpu = state["gpu"]
    if state["kind"] == "adjoint":
        bar, grads = gpu.forwardBackward(state["steps"], state["every"], state["bar"])
        # the parameter gradients are sums of single-precision terms
        return {"states": bar, "params": grads.astype(np.float32)}
    gpu.step(state["steps"])
    out = {}
    for name in gpu.state:  # the states' two device buffers take turns
        ptr, n = gpu.valueBuffer(name)
        if ptr not in state["views"]:
            state["views"][ptr] = _view(gpu, ptr, n)
        out[name] = state["views"][ptr]
    return out


# --------------------------------------------------------------------- work


def _pair_flops(case):
    """Synthesis and analysis of one field: parity-folded Legendre sums and
    real FFTs of every latitude."""
    nlm = _degrees(case["lmax"], case["mmax"])[0].size
    return 2.0 * case["nlat"] * (2.0 * nlm + 2.5 * case["nphi"] * math.log2(case["nphi"]))


def work(case):
    nlm = _degrees(case["lmax"], case["mmax"])[0].size
    spec, grid = 8.0 * nlm, 4.0 * case["nlat"] * case["nphi"]
    fields, steps = case["batch"], case.get("steps", 1)
    if case["kind"] in ("step", "adjoint"):
        fields *= len(mModelByKey(case["model"]).state)
    flops = steps * fields * _pair_flops(case)
    if case["kind"] == "pair":  # two calls: the grid is an output and then an input
        return {"bytes": fields * 2 * (spec + grid), "flops": flops}
    if case["kind"] == "host":  # the grid is not asked for
        return {"bytes": fields * 2 * spec, "flops": flops}
    if case["kind"] == "step":  # the states, read and written by every step
        return {"bytes": steps * fields * 2 * spec, "flops": flops}
    # forward steps (with the states kept), then a transposed pair per step
    return {"bytes": steps * fields * 4 * spec, "flops": 2 * flops}


# -------------------------------------------------------------------- exact


class _Exact:
    """The transforms in 64 bits: Gauss nodes, orthonormal associated Legendre
    functions by their recurrence in l (every order at once), dense sums and
    torch's FFT."""

    def __init__(self, case):
        lmax, mmax, nlat = case["lmax"], case["mmax"], case["nlat"]
        self.nlat, self.nphi, self.mmax = nlat, case["nphi"], mmax
        x, w = np.polynomial.legendre.leggauss(nlat)
        x = torch.from_numpy(x[::-1].copy()).cuda()
        self.w = torch.from_numpy(w[::-1].copy()).cuda() * (2 * math.pi / self.nphi)
        m = torch.arange(mmax + 1, dtype=torch.float64, device="cuda")
        k = torch.arange(1, mmax + 1, dtype=torch.float64, device="cuda")
        log_ratio = torch.cat([m[:1] * 0, torch.cumsum(torch.log((2 * k - 1) / (2 * k)), 0)])
        sign = 1 - 2 * (m % 2)
        log_sin = 0.5 * torch.log1p(-x * x)
        diag = sign[:, None] * torch.exp(0.5 * (torch.log((2 * m + 1) / (4 * math.pi)) + log_ratio)[:, None]
                                         + m[:, None] * log_sin[None, :])
        # p[m, l, lat], zero for l < m
        self.p = torch.zeros(mmax + 1, lmax + 1, nlat, dtype=torch.float64, device="cuda")
        for l in range(lmax + 1):
            top = min(l, mmax + 1)  # orders m < l come from the recurrence
            if top:
                mm = m[:top]
                a = torch.sqrt((4.0 * l * l - 1) / (l * l - mm * mm))
                row = a[:, None] * x * self.p[:top, l - 1]
                if l > 1:
                    b = torch.sqrt(((l - 1.0) ** 2 - mm * mm).clamp(min=0) / (4 * (l - 1.0) ** 2 - 1))
                    row -= (a * b)[:, None] * self.p[:top, l - 2]
                self.p[:top, l] = row
            if l <= mmax:
                self.p[l, l] = diag[l]
        ls, ms = _degrees(lmax, mmax)
        self.at = torch.from_numpy(ms * (lmax + 1) + ls).cuda()
        self.ll = torch.from_numpy((ls * (ls + 1.0)).repeat(2)).cuda()

    def synth(self, q):  # (fields, 2 nlm) -> (fields, nlat, nphi)
        n = q.shape[0]
        full = torch.zeros(self.p.shape[0] * self.p.shape[1], n, 2, dtype=torch.float64, device="cuda")
        full = full.index_copy(0, self.at, q.reshape(n, -1, 2).transpose(0, 1))
        f = torch.bmm(self.p.transpose(1, 2), full.reshape(self.p.shape[0], self.p.shape[1], 2 * n))
        f = torch.view_as_complex(f.reshape(self.mmax + 1, self.nlat, n, 2)).permute(2, 1, 0)
        return torch.fft.irfft(f, n=self.nphi, dim=2) * self.nphi

    def analys(self, g):  # (fields, nlat, nphi) -> (fields, 2 nlm)
        n = g.shape[0]
        f = torch.fft.rfft(g, dim=2)[:, :, :self.mmax + 1] * self.w[None, :, None]
        f = torch.view_as_real(f.permute(2, 1, 0).contiguous()).reshape(self.mmax + 1, self.nlat, 2 * n)
        q = torch.bmm(self.p, f).reshape(-1, n, 2)
        return q.index_select(0, self.at).transpose(0, 1).reshape(n, -1)

    def step(self, model, s, p):  # one IMEX Euler step of every instance
        grid = {k: self.synth(v) for k, v in s.items()}
        dt = p["dt"][:, None]
        g = {k: v[:, None, None] for k, v in p.items()}
        u = grid["U"]
        if model == "allencahn":
            rate, d = {"U": u - u ** 3}, {"U": p["eps2"]}
        else:
            uuv = u * u * grid["V"]
            d = {"U": p["D1"], "V": p["D2"]}
            if model == "schnakenberg":
                rate = {"U": g["a"] - u + uuv, "V": g["b"] - uuv}
            else:
                rate = {"U": g["A"] - (g["B"] + 1) * u + uuv, "V": g["B"] * u - uuv}
        return {k: (s[k] + dt * self.analys(rate[k])) / (1 + dt * d[k][:, None] * self.ll) for k in s}


def exact(case, seed):
    if case["kind"] == "host":  # a round trip of band-limited fields is the identity
        return _spectra(case, seed, case["batch"]).double().cpu()
    t = _Exact(case)
    if case["kind"] == "pair":
        q = _spectra(case, seed, case["batch"]).double()
        return [t.synth(q).reshape(case["batch"], -1), q]
    model = mModelByKey(case["model"])
    names = [p.key for p in model.params]
    values = np.array([[p[k] for k in names] for p in _params(case)], dtype=np.float32)
    params = torch.from_numpy(values).cuda().double()
    states = {k: v.double() for k, v in _states(case, seed).items()}
    if case["kind"] == "step":
        for _ in range(case["steps"]):
            states = t.step(case["model"], states, dict(zip(names, params.unbind(1))))
        return states
    first = {k: v.requires_grad_() for k, v in states.items()}
    params.requires_grad_()
    s = first
    for _ in range(case["steps"]):
        s = t.step(case["model"], s, dict(zip(names, params.unbind(1))))
    loss = 0.0
    for i, name in enumerate(model.state):
        loss = loss + (s[name] * _spectra(case, 2 * seed + 1000003 + i, case["batch"]).double()).sum()
    loss.backward()
    return {"states": {k: v.grad for k, v in first.items()}, "params": params.grad}
