"""Timed cases of the framework: line-by-line spectra, Jacobians and the surrogate network.

``listed()`` names one case per kind of call that programs make, ``draw(rng)`` gives more of
the same ranges. ``prepare`` makes what a program holds before the call (line list, profile,
kept job or network), ``run`` is one call through the public entry points, ``work`` the bytes
and operations that call cannot do without, and ``exact`` the call's results in float64 by
plain torch (a restatement of the same formulas that shares no code with the engine).
"""

from __future__ import annotations

import math

import numpy as np
import torch

from pylblrtm_b200 import AtmosphericProfile, adjoint, compute_transmittance, engine, surrogate, synthetic

DEV = "cuda"


def listed():
    return [
        # one microwindow of a CO2 band, 20-layer standard atmosphere: the smallest spectrum a
        # program asks for; launches and host work count here
        dict(name="od_microwindow", kind="od", n_lines=2000, gases=1, list_lo=700.0, list_hi=750.0, lo=720.0,
             hi=725.0, step=0.001, layers=20, cutoff=25.0, tile=2.0, strength=1e-3, deterministic=False),
        # a 100 cm-1 band out of a whole three-gas line list, 60 layers: the ordinary call
        dict(name="od_band_of_list", kind="od", n_lines=200_000, gases=3, list_lo=600.0, list_hi=2500.0, lo=1000.0,
             hi=1100.0, step=0.001, layers=60, cutoff=25.0, tile=2.0, strength=1.0, deterministic=False),
        # sizes off every round number (grid, tile, layers, cut-off), bit-reproducible sums
        dict(name="od_ragged_reproducible", kind="od", n_lines=50_021, gases=3, list_lo=790.0, list_hi=1130.0,
             lo=811.3, hi=1103.77, step=0.0023, layers=37, cutoff=10.3, tile=1.05, strength=1e-2,
             deterministic=True),
        # the whole 600-2500 cm-1 spectrum on a kept job (inputs already on the device): the
        # benchmark's step, the largest single spectrum
        dict(name="od_full_resident", kind="job", n_lines=200_000, gases=3, list_lo=600.0, list_hi=2500.0, lo=600.0,
             hi=2500.0, step=0.001, layers=60, cutoff=25.0, tile=2.0, strength=1.0, deterministic=False),
        # float64 spectra (validation of retrievals, reference runs): a CO2 band piece ...
        dict(name="trans_fp64_co2", kind="trans64", n_lines=2000, gases=1, list_lo=700.0, list_hi=750.0, lo=715.0,
             hi=735.0, step=0.001, layers=20, cutoff=25.0, tile=2.0, strength=1e-3, deterministic=False),
        # ... and a window of the three-gas list at 60 layers
        dict(name="trans_fp64_three_gas", kind="trans64", n_lines=200_000, gases=3, list_lo=600.0, list_hi=2500.0,
             lo=1000.0, hi=1020.0, step=0.001, layers=60, cutoff=25.0, tile=2.0, strength=1e-5,
             deterministic=False),
        # channel-mean transmittances of a batch of 20-layer profiles: how training spectra and
        # the gate's fallback are made
        dict(name="channels_batch", kind="channels", n_lines=200_000, gases=3, list_lo=600.0, list_hi=2500.0,
             lo=650.0, hi=1150.0, step=0.001, layers=20, profiles=16, channel=0.25, cutoff=25.0, tile=2.0,
             strength=1e-4, deterministic=False),
        # layer Jacobians of one profile over 200 cm-1: one linearisation of a retrieval
        dict(name="jacobian_band", kind="jac", n_lines=200_000, gases=3, list_lo=600.0, list_hi=2500.0, lo=1000.0,
             hi=1200.0, step=0.001, layers=60, cutoff=25.0, tile=2.0, strength=1e-4, deterministic=False),
        # a gradient step of a small batch of profiles through torch autograd (forward and backward)
        dict(name="retrieval_gradient", kind="vjp", n_lines=20_000, gases=3, list_lo=690.0, list_hi=880.0, lo=720.0,
             hi=760.0, step=0.001, layers=20, profiles=4, cutoff=25.0, tile=2.0, strength=1e-4,
             deterministic=False),
        # optimiser steps of the surrogate network at its training batch (forward, backward, Adam)
        dict(name="surrogate_train", kind="train", batch=4096, samples=16_384, n_out=2000, hidden=1024, depth=4,
             steps=4),
        # the gated ensemble on a handful of profiles (a service's request) and on a large batch
        dict(name="ensemble_small", kind="gate", batch=200, members=4, n_out=2000, hidden=1024, depth=4),
        dict(name="ensemble_large", kind="gate", batch=20_000, members=4, n_out=2000, hidden=1024, depth=4),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["od", "od", "od", "job", "trans64", "trans64", "channels", "jac", "vjp", "train", "gate",
                       "gate"])
    if kind == "train":
        batch = 128 * max(2, round(_log_uniform(rng, 256, 4096) / 128))
        return dict(kind=kind, batch=batch, samples=2 * batch + rng.randrange(1, 4000),
                    n_out=rng.choice([400, 1000, 2000]), hidden=rng.choice([512, 768, 1024]),
                    depth=rng.choice([2, 3, 4]), steps=rng.choice([2, 4]))
    if kind == "gate":
        return dict(kind=kind, batch=round(_log_uniform(rng, 20, 20_000)), members=rng.choice([2, 4]),
                    n_out=rng.choice([400, 1000, 2000]), hidden=rng.choice([512, 1024]), depth=rng.choice([2, 4]))
    gases = rng.choice([1, 3])
    list_lo = round(rng.uniform(600.0, 1100.0), 2)
    list_hi = round(list_lo + _log_uniform(rng, 150.0, 1300.0), 2)
    # lines per cm-1 between the CO2 band's 40 and the three-gas list's 105
    n_lines = round((list_hi - list_lo) * rng.uniform(30.0, 110.0))
    widest = {"od": 300.0, "job": 1200.0, "trans64": 18.0, "channels": 200.0, "jac": 150.0, "vjp": 50.0}[kind]
    width = min(_log_uniform(rng, 2.0, widest), list_hi - list_lo)
    lo = round(rng.uniform(list_lo, list_hi - width), 2)
    c = dict(kind=kind, n_lines=n_lines, gases=gases, list_lo=list_lo, list_hi=list_hi, lo=lo,
             hi=round(lo + width, 2), step=rng.choice([0.001, 0.001, 0.0013, 0.002, 0.0047, 0.01]),
             layers=rng.choice([20, 20, 31, 45, 60]), cutoff=rng.choice([25.0, 25.0, 10.0, 5.5]),
             tile=rng.choice([2.0, 2.0, 1.0, 0.73]), strength=rng.choice([1e-5, 1e-4, 1e-3]),
             deterministic=kind in ("od", "job", "jac") and rng.random() < 0.3)
    if kind in ("channels", "vjp"):
        c.update(gases=3, layers=20, profiles=rng.choice([1, 2, 3, 5, 8]))
    if kind == "channels":
        c["channel"] = rng.choice([0.25, 0.5, 1.0])
    return c


# ---------------------------------------------------------------------------------- inputs

def _gases(case):
    return ("H2O", "CO2", "O3") if case["gases"] == 3 else ("CO2",)


def _lines(case, seed):
    if case["gases"] == 3:
        sd = synthetic.three_gas_lines(case["n_lines"], case["list_lo"], case["list_hi"], seed=seed)
    else:
        sd = synthetic.co2_band(case["n_lines"], case["list_lo"], case["list_hi"], seed=seed)
    return sd if case["strength"] == 1.0 else synthetic.scale_strengths(sd, case["strength"])


def _levels(case, seed, n_profiles=1):
    base = synthetic.ussa_levels() if case["layers"] == 20 else synthetic.logp_levels(case["layers"] + 1)
    return synthetic.perturbed_levels(base, n_profiles, seed + 1)


def _profiles(case, seed, n_profiles=1):
    lv = _levels(case, seed, n_profiles)
    return [AtmosphericProfile(lv["p"][i], lv["t"][i], {g: lv[g][i] for g in _gases(case)})
            for i in range(n_profiles)]


def _observations(case, seed, shape):
    g = torch.Generator(device=DEV).manual_seed(seed + 2)
    return torch.rand(shape, generator=g, device=DEV)


def _network_state(case, seed, step):
    """A network (and, for training, moments as they are some way into a run) as a state dict."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    pad = lambda n: (n + 127) // 128 * 128
    n_in, n_out, hidden, depth = 61, case["n_out"], case["hidden"], case["depth"]
    st = {"dims": (n_in, n_out, hidden, depth), "step": step, "lr": 1e-3, "betas": (0.9, 0.999), "eps": 1e-8,
          "w": [], "b": [], "mw": [], "vw": [], "mb": [], "vb": []}
    for i in range(depth + 1):
        k = n_in if i == 0 else hidden
        n = n_out if i == depth else hidden
        std = 0.1 * math.sqrt(1.0 / k) if i == depth else math.sqrt(2.0 / k)
        for name, shape, real in (("w", (pad(n), pad(k)), (n, k)), ("b", (pad(n),), (n,))):
            at = tuple(slice(0, r) for r in real)
            for key, scale in ((name, std if name == "w" else 0.05), ("m" + name, 1e-5), ("v" + name, 1e-5)):
                t = torch.zeros(shape, device=DEV)
                v = rnd(*real) * scale
                t[at] = v.square() + 1e-12 if key[0] == "v" else v
                st[key].append(t)
    st["mean"] = 0.1 * rnd(n_in)
    st["inv_std"] = 1.0 + 0.1 * torch.rand(n_in, generator=g, device=DEV)
    return st


def _train_data(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 7)
    x = torch.randn((case["samples"], 61), generator=g, device=DEV)
    a = torch.randn((61, case["n_out"]), generator=g, device=DEV) * 0.12
    return x, torch.sigmoid(x @ a)


def _train_config(case, seed):
    return surrogate.TrainConfig(batch=case["batch"], steps=20_000, seed=seed % 1000)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        net = surrogate.MLP(61, case["n_out"], hidden=case["hidden"], depth=case["depth"])
        net.load_state_dict(_network_state(case, seed, step=400))
        x, y = _train_data(case, seed)
        return {"case": case, "trainer": surrogate.Trainer(net, x, y, _train_config(case, seed))}
    if kind == "gate":
        nets = []
        for m in range(case["members"]):
            net = surrogate.MLP(61, case["n_out"], hidden=case["hidden"], depth=case["depth"])
            net.load_state_dict(_network_state(case, seed + 1000 * m, step=0))
            nets.append(net)
        g = torch.Generator(device=DEV).manual_seed(seed + 3)
        raw = torch.randn((case["batch"], 61), generator=g, device=DEV)
        return {"case": case, "gate": surrogate.GatedSurrogate(nets, gate=0.05), "raw": raw}
    s = {"case": case, "sd": _lines(case, seed)}
    s["grid"] = engine.make_grid(case["lo"], case["hi"], case["step"], case["tile"])
    if kind == "channels":
        s["profiles"] = surrogate.sample_profiles(case["profiles"], seed + 1)
        s["problem"] = surrogate.SurrogateProblem(case["lo"], case["hi"], case["step"], case["channel"],
                                                  case["cutoff"], case["tile"])
    elif kind == "vjp":
        profs = _profiles(case, seed, case["profiles"])
        s["state"] = adjoint.LayerState.from_profiles(s["sd"], profs, "H2O", case["lo"], case["hi"], case["step"],
                                                      case["cutoff"], case["tile"])
        lay = [p.build_layers() for p in profs]
        s["t"] = torch.tensor(np.stack([l.temperature_k for l in lay]), dtype=torch.float32, device=DEV)
        s["lnv"] = torch.tensor(np.log(np.stack([l.vmr["H2O"] for l in lay])), dtype=torch.float32, device=DEV)
        s["obs"] = _observations(case, seed, (case["profiles"], s["grid"].n_nu))
    else:
        s["profile"] = _profiles(case, seed)[0]
        if kind == "job":
            s["job"] = engine.Job(s["sd"], engine.layer_input_from_profile(s["profile"]), s["grid"], case["cutoff"])
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "od":
        res = engine.optical_depth(s["sd"], engine.layer_input_from_profile(s["profile"]), s["grid"], c["cutoff"],
                                   deterministic=c["deterministic"])
        return {"od": res.od}
    if kind == "job":
        return {"od": s["job"].run("fp32", deterministic=c["deterministic"]).od}
    if kind == "trans64":
        nu, trans = compute_transmittance(s["sd"], s["profile"], c["lo"], c["hi"], step_cm1=c["step"],
                                          line_cutoff_cm1=c["cutoff"], tile_width_cm1=c["tile"], mu_view=0.8,
                                          precision="fp64")
        return {"nu": nu, "trans": trans}
    if kind == "channels":
        return {"channels": surrogate.engine_channels(s["sd"], s["profiles"], s["problem"], as_numpy=False)}
    if kind == "jac":
        out = adjoint.layer_jacobians(s["sd"], s["profile"], c["lo"], c["hi"], step_cm1=c["step"],
                                      line_cutoff_cm1=c["cutoff"], tile_width_cm1=c["tile"], gas=_gases(c)[0],
                                      as_numpy=False, deterministic=c["deterministic"])
        return {k: out[k] for k in ("od", "dtau_dT", "dtau_dlnvmr")}
    if kind == "vjp":
        t, lnv = s["t"].clone().requires_grad_(True), s["lnv"].clone().requires_grad_(True)
        tau = adjoint.layer_optical_depth(t, lnv, s["state"])
        resid = torch.exp(-tau).float() - s["obs"]
        resid.square().sum().backward()
        return {"dT": t.grad, "dlnvmr": lnv.grad}
    if kind == "train":
        tr = s["trainer"]
        losses = tr.run(steps=c["steps"])
        net = tr.net
        return {"losses": losses[-c["steps"]:], "w": net.w, "b": net.b, "mw": net.mw, "vw": net.vw}
    mean, est, flag = s["gate"].ensemble(s["raw"])
    return {"mean": mean, "est": est, "flag": flag}


# ---------------------------------------------------------------------------------- work

def _grid_points(case):
    return int(np.ceil((case["hi"] - case["lo"]) / case["step"])) + 1


def _lines_per_point(case):
    """Lines that must be summed point by point: those within 128 points either side."""
    density = case["n_lines"] / (case["list_hi"] - case["list_lo"])
    return density * min(256 * case["step"], 2 * case["cutoff"])


def _window_evals(case):
    """Line evaluations of the tile-window rule (layer, point, line)."""
    density = case["n_lines"] / (case["list_hi"] - case["list_lo"])
    return case.get("profiles", 1) * case["layers"] * _grid_points(case) * density * (2 * case["cutoff"] + case["tile"])


def work(case):
    kind = case["kind"]
    if kind in ("train", "gate"):
        dims = [61] + [case["hidden"]] * case["depth"] + [case["n_out"]]
        n_w = sum(a * b for a, b in zip(dims[:-1], dims[1:]))
        if kind == "train":      # float32 weights and both moments read and written once a step
            return {"flops": 6.0 * n_w * case["batch"] * case["steps"],
                    "bytes": case["steps"] * (24.0 * n_w + 4.0 * case["batch"] * (61 + case["n_out"]))}
        return {"flops": 2.0 * n_w * case["batch"] * case["members"],
                "bytes": 2.0 * n_w * case["members"] + 4.0 * case["batch"] * (61 + case["n_out"] + 2)}
    n, rows = _grid_points(case), case["layers"] * case.get("profiles", 1)
    outs = {"od": 4.0 * rows * n, "job": 4.0 * rows * n, "trans64": 16.0 * n, "jac": 12.0 * rows * n,
            "vjp": 4.0 * n * case.get("profiles", 1),
            "channels": 4.0 * case.get("profiles", 1) * (n * case["step"] / case.get("channel", 1.0))}[kind]
    per_line = {"trans64": 60.0, "jac": 60.0, "vjp": 84.0}.get(kind, 24.0)
    return {"bytes": 60.0 * case["n_lines"] + outs, "flops": rows * n * (per_line * _lines_per_point(case) + 40.0)}


# ---------------------------------------------------------------------------------- float64 results

_T_REF, _C2, _SQRT_LN2 = 296.0, 1.4387752, math.sqrt(math.log(2.0))
_K = math.sqrt(math.log(2.0) / math.pi)


def _weideman(n=64):
    """Weideman's (1994) rational approximation: coefficients (highest power first) and L."""
    m2 = 4 * n
    k = np.arange(-m2 + 1, m2)
    scale = math.sqrt(n / math.sqrt(2.0))
    t = scale * np.tan(k * math.pi / m2 / 2)
    f = np.concatenate([[0.0], np.exp(-t * t) * (scale * scale + t * t)])
    a = np.real(np.fft.fft(np.fft.fftshift(f))) / (2 * m2)
    return np.flipud(a[1:n + 1]), scale


def _w_near(z):
    a, scale = _weideman()
    big = (scale + 1j * z) / (scale - 1j * z)
    p = torch.zeros_like(z)
    for c in a:
        p = p * big + float(c)
    return 2.0 * p / (scale - 1j * z) ** 2 + (1.0 / math.sqrt(math.pi)) / (scale - 1j * z)


def _w_far(z, terms):
    """(w, w') by the asymptotic series."""
    i2 = 1.0 / (z * z)
    c = [1.0]
    for k in range(1, terms):
        c.append(c[-1] * (2 * k - 1) / 2.0)
    s = torch.full_like(z, c[-1])
    d = torch.full_like(z, c[-1] * (2 * terms - 1))
    for k in range(terms - 2, -1, -1):
        s = s * i2 + c[k]
        d = d * i2 + c[k] * (2 * k + 1)
    f = 1j / math.sqrt(math.pi)
    return f * s / z, -f * d * i2


def _w_and_slope(z):
    """w and w' of any z with Im z >= 0."""
    z2 = z.real ** 2 + z.imag ** 2
    w, d = _w_far(z, 5)
    for sel, terms in (((z2 < 2500.0) & (z2 >= 100.0), 12), (z2 < 100.0, 0)):
        at = sel.nonzero(as_tuple=True)
        if at[0].numel():
            zs = z[at]
            if terms:
                w[at], d[at] = _w_far(zs, terms)
            else:
                ws = _w_near(zs)
                w[at], d[at] = ws, -2.0 * zs * ws + 2j / math.sqrt(math.pi)
    return w, d


def _re_w(x, y):
    """Re w by the real form of the same series (5 terms), else by _w_and_slope."""
    y2 = (y * y).expand_as(x)
    z2 = x * x + y2
    r = 1.0 / z2
    q = y2 * r
    s = (((1680.0 * q - 3780.0) * q + 2835.0) * q - 787.5) * q + 59.0625
    s = s * r + (((-120.0 * q + 210.0) * q - 105.0) * q + 13.125)
    s = s * r + ((12.0 * q - 15.0) * q + 3.75)
    s = s * r + (1.5 - 2.0 * q)
    u = (s * r + 1.0) * r * (y / math.sqrt(math.pi))
    at = (z2 < 2500.0).nonzero(as_tuple=True)
    if at[0].numel():
        u[at] = _w_and_slope(torch.complex(x[at], y.expand_as(x)[at]))[0].real
    return u


def _interp(t, xp, fp):
    """np.interp (clamped), differentiable in t."""
    i = torch.clamp(torch.searchsorted(xp, t.detach().contiguous(), right=True) - 1, 0, xp.numel() - 2)
    v = fp[i] + (fp[i + 1] - fp[i]) / (xp[i + 1] - xp[i]) * (t - xp[i])
    return torch.where(t >= xp[-1], fp[-1], torch.where(t < xp[0], fp[0], v))


def _exact_lines(case, sd, p_max):
    """Sorted in-band lines as float64 tensors, with their gas and tables."""
    nu0 = np.asarray(sd.lines["nu0"], np.float64)
    sb = np.abs(sd.lines["shift"]) * p_max
    n = _grid_points(case)
    last = case["lo"] + (n - 1) * case["step"]
    keep = np.flatnonzero((nu0 >= case["lo"] - case["cutoff"] - sb) & (nu0 <= last + case["cutoff"] + sb))
    keep = keep[np.argsort(nu0[keep], kind="stable")]
    L = {k: torch.tensor(np.asarray(sd.lines[k])[keep], device=DEV) for k in sd.lines}
    groups = []
    for key, (t, q) in sd.tips.items():
        gas = {1: "H2O", 2: "CO2", 3: "O3"}[key[0]]
        groups.append((gas, (L["mol_id"] == key[0]), torch.tensor(t, device=DEV), torch.tensor(q, device=DEV),
                       sd.molar_masses[key]))
    return L, groups, float(sb.max() if sb.size else 0.0)


def _line_params(L, groups, p, t, vmr, col):
    """(nuc, amp, sc, y) [rows, lines]: Voigt argument (nu - nuc) sc + i y, factor amp."""
    tc, pc = t[:, None], p[:, None]
    v, c, dop, q = (torch.zeros((t.shape[0], L["nu0"].numel()), dtype=torch.float64, device=DEV) for _ in range(4))
    for gas, sel, tt, qq, mass in groups:
        m = sel.double()[None, :]
        v = v + vmr[gas][:, None] * m
        c = c + col[gas][:, None] * m
        dop = dop + torch.sqrt(tc / mass) * m
        q = q + (_interp(torch.full_like(t, _T_REF), tt, qq) / _interp(t, tt, qq))[:, None] * m
    p_self = v * pc
    p_air = pc - p_self
    nuc = L["nu0"] + L["shift"] * p_air
    stim = -torch.expm1(-_C2 * L["nu0"] / tc) / -torch.expm1(-_C2 * L["nu0"] / _T_REF)
    strength = L["Sref"] * q * torch.exp(-_C2 * L["Elow"] * (1.0 / tc - 1.0 / _T_REF)) * stim * c
    strength = strength / (nuc * torch.tanh(0.5 * _C2 * nuc / tc))
    gamma = (_T_REF / tc) ** L["n_air"] * (L["g_air"] * p_air + L["g_self"] * p_self)
    alpha = L["nu0"] * 3.5810e-7 * dop
    return nuc, strength * _K / alpha, _SQRT_LN2 / alpha, _SQRT_LN2 * gamma / alpha


def _radiation(nu, t):
    return nu * torch.tanh(0.5 * _C2 * nu / t)


def _exact_spectrum(case, sd, p, t, vmr, col, gas=None):
    """od [rows, n_nu] and, for a gas, d od/dT and d od/dln VMR, one row per (profile, layer)."""
    L, groups, pad = _exact_lines(case, sd, float(p.max()))
    params = lambda tt, lv: _line_params(L, groups, p, tt,
                                         {g: vmr[g] * torch.exp(lv) if g == gas else vmr[g] for g in vmr},
                                         {g: col[g] * torch.exp(lv) if g == gas else col[g] for g in col})
    zero, one = torch.zeros_like(t), torch.ones_like(t)
    tangents = None
    if gas is None:
        nuc, amp, sc, y = params(t, zero)
    else:
        (nuc, amp, sc, y), d_t = torch.func.jvp(params, (t, zero), (one, zero))
        tangents = [d_t, torch.func.jvp(params, (t, zero), (zero, one))[1]]
    n = _grid_points(case)
    nu = case["lo"] + torch.arange(n, dtype=torch.float64, device=DEV) * case["step"]
    eff = float((nu[1] - nu[0]).item()) if n > 1 else 0.001
    tile = max(1, int(np.floor(case["tile"] / eff + 1e-8)))
    rows = t.numel()
    out = [torch.zeros((rows, n), dtype=torch.float64, device=DEV) for _ in range(1 if gas is None else 3)]
    nu0 = L["nu0"].cpu().numpy()
    most = 100_000_000 if gas is None else 40_000_000
    for t0 in range(0, n, tile):
        seg = nu[t0:t0 + tile]
        lo, hi = float(seg[0]) - case["cutoff"], float(seg[-1]) + case["cutoff"]
        a, b = np.searchsorted(nu0, lo - pad - 1e-6), np.searchsorted(nu0, hi + pad + 1e-6)
        if b <= a:
            continue
        per = max(1, most // (seg.numel() * int(b - a)))
        for r0 in range(0, rows, per):
            rs = slice(r0, min(rows, r0 + per))
            cut = lambda v: v[rs, a:b]
            inside = (cut(nuc) >= lo) & (cut(nuc) <= hi)
            x = (seg[None, :, None] - cut(nuc)[:, None, :]) * cut(sc)[:, None, :]
            yy = cut(y)[:, None, :]
            am = torch.where(inside, cut(amp), 0.0)
            mul = lambda u, f: torch.bmm(u, f[:, :, None])[:, :, 0]
            if gas is None:
                out[0][rs, t0:t0 + tile] = mul(_re_w(x, yy), am)
                continue
            w, d = _w_and_slope(torch.complex(x, yy.expand_as(x)))
            u, ux, uy = w.real.contiguous(), d.real.contiguous(), -d.imag
            out[0][rs, t0:t0 + tile] = mul(u, am)
            for o, (dn, da, ds, dy) in zip(out[1:], tangents):
                xux = x * ux
                o[rs, t0:t0 + tile] = (mul(u, torch.where(inside, cut(da), 0.0)) + mul(xux, am * cut(ds) / cut(sc))
                                       - mul(ux, am * cut(dn) * cut(sc)) + mul(uy.contiguous(), am * cut(dy)))
    rad, rad_t = torch.func.jvp(lambda tt: _radiation(nu[None, :], tt), (t[:, None],), (torch.ones_like(t)[:, None],))
    if gas is None:
        return out[0] * rad
    return out[0] * rad, rad_t * out[0] + rad * out[1], rad * out[2]


def _rows(case, profiles):
    """Layer quantities of level profiles, one row per (profile, layer)."""
    lay = [p.build_layers() for p in profiles]
    cat = lambda f: torch.tensor(np.concatenate([f(l) for l in lay]), dtype=torch.float64, device=DEV)
    gases = _gases(case)
    return (cat(lambda l: l.pressure_atm), cat(lambda l: l.temperature_k),
            {g: cat(lambda l: l.vmr[g]) for g in gases}, {g: cat(lambda l: l.column_cm2[g]) for g in gases})


def _mlp(st, x):
    """Hidden activations, pre-activations and logits in float64."""
    w, b = [v.double() for v in st["w"]], [v.double() for v in st["b"]]
    h = torch.zeros((x.shape[0], w[0].shape[1]), dtype=torch.float64, device=DEV)
    h[:, :61] = (x.double() - st["mean"].double()) * st["inv_std"].double()
    hs, zs = [h], []
    for i in range(len(w)):
        zs.append(hs[-1] @ w[i].T + b[i])
        if i + 1 < len(w):
            hs.append(0.5 * zs[-1] * (1.0 + torch.erf(zs[-1] / math.sqrt(2.0))))
    return w, b, hs, zs


def _exact_train(case, seed):
    st = _network_state(case, seed, step=400)
    x, target = _train_data(case, seed)
    cfg = _train_config(case, seed)
    n_out, batch = case["n_out"], case["batch"]
    state = {k: [v.double() for v in st[k]] for k in ("w", "b", "mw", "vw", "mb", "vb")}
    state["mean"], state["inv_std"] = st["mean"], st["inv_std"]
    step, cursor, epoch, losses, order = 400, 0, 0, [], None
    for _ in range(case["steps"]):
        if order is None or cursor + batch > case["samples"]:
            epoch += order is not None
            cursor = 0
            g = torch.Generator().manual_seed(cfg.seed * 1_000_003 + epoch)
            order = torch.randperm(case["samples"], generator=g).to(DEV)
        idx = order[cursor:cursor + batch]
        cursor += batch
        lr = cfg.lr_final + 0.5 * (cfg.lr - cfg.lr_final) * (
            1 + math.cos(math.pi * (step - cfg.warmup) / (cfg.steps - cfg.warmup)))
        w, b, hs, zs = _mlp(state, x[idx])
        p = torch.sigmoid(zs[-1][:, :n_out])
        e = p - target[idx].double()
        losses.append(float(e.square().sum()) / (batch * n_out))
        dz = torch.zeros_like(zs[-1])
        dz[:, :n_out] = 2.0 * e * p * (1.0 - p) / batch
        grads = []
        for i in range(len(w) - 1, -1, -1):
            grads.append((dz.T @ hs[i], dz.sum(0)))
            if i:
                z = zs[i - 1]
                slope = 0.5 * (1.0 + torch.erf(z / math.sqrt(2.0))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi)
                dz = (dz @ w[i]) * slope
        step += 1
        c1, c2 = 1.0 / (1.0 - 0.9 ** step), 1.0 / (1.0 - 0.999 ** step)
        for i, pair in enumerate(reversed(grads)):
            for name, g in zip("wb", pair):
                m = 0.9 * state["m" + name][i] + 0.1 * g
                v = 0.999 * state["v" + name][i] + 0.001 * g * g
                state["m" + name][i], state["v" + name][i] = m, v
                state[name][i] = state[name][i] - lr * m * c1 / (torch.sqrt(v * c2) + 1e-8)
    return {"losses": losses, **{k: state[k] for k in ("w", "b", "mw", "vw")}}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "gate":
        g = torch.Generator(device=DEV).manual_seed(seed + 3)
        raw = torch.randn((case["batch"], 61), generator=g, device=DEV)
        pred = []
        for m in range(case["members"]):
            zs = _mlp(_network_state(case, seed + 1000 * m, step=0), raw)[3]
            pred.append(torch.sigmoid(zs[-1][:, :case["n_out"]]))
        pred = torch.stack(pred)
        return {"mean": pred.mean(0), "est": pred.std(0, unbiased=False).max(1).values, "flag": None}
    # the derivatives cost about four times an optical depth; beyond this the sums take too long
    if _window_evals(case) * (4 if kind in ("jac", "vjp") else 1) > 1.2e11:
        return None
    sd = _lines(case, seed)
    if kind == "channels":
        pb = surrogate.sample_profiles(case["profiles"], seed + 1)
        t64 = lambda a: torch.tensor(a.reshape(-1), dtype=torch.float64, device=DEV)
        vmr = {g: t64(pb.vmr[:, i]) for i, g in enumerate(_gases(case))}
        air = t64(pb.air_col)
        od = _exact_spectrum(case, sd, t64(pb.p_atm), t64(pb.t), vmr, {g: v * air for g, v in vmr.items()})
        tau = od.reshape(case["profiles"], case["layers"], -1).sum(1)
        width = int(round(case["channel"] / case["step"]))
        n_ch = tau.shape[1] // width
        trans = torch.exp(-tau / torch.tensor(pb.mu, device=DEV)[:, None])
        return {"channels": trans[:, :n_ch * width].reshape(case["profiles"], n_ch, width).mean(2)}
    profs = _profiles(case, seed, case.get("profiles", 1))
    p, t, vmr, col = _rows(case, profs)
    if kind in ("od", "job"):
        return {"od": _exact_spectrum(case, sd, p, t, vmr, col)[None]}
    if kind == "trans64":
        od = _exact_spectrum(case, sd, p, t, vmr, col)
        nu = case["lo"] + np.arange(_grid_points(case)) * case["step"]
        return {"nu": nu, "trans": torch.exp(-od.sum(0) / 0.8)}
    if kind == "jac":
        od, d_t, d_v = _exact_spectrum(case, sd, p, t, vmr, col, gas=_gases(case)[0])
        return {"od": od, "dtau_dT": d_t, "dtau_dlnvmr": d_v}
    n_prof, n_lay = case["profiles"], case["layers"]
    # the call's own inputs are float32 layer temperatures and ln VMR
    air = col["CO2"] / vmr["CO2"]
    t = t.float().double()
    vmr["H2O"] = torch.exp(torch.log(vmr["H2O"]).float().double())
    col["H2O"] = vmr["H2O"] * air
    od, d_t, d_v = _exact_spectrum(case, sd, p, t, vmr, col, gas="H2O")
    shape = (n_prof, n_lay, -1)
    trans = torch.exp(-od.reshape(shape).sum(1))
    obs = _observations(case, seed, (n_prof, od.shape[1])).double()
    g = -2.0 * (trans - obs) * trans
    return {"dT": (d_t.reshape(shape) * g[:, None]).sum(2), "dlnvmr": (d_v.reshape(shape) * g[:, None]).sum(2)}
