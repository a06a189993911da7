"""Performance cases of the public entry points: what a program that uses this package has it do.

A case is a dict of plain values.  ``listed()`` names the fixed ones, ``draw(rng)`` gives more of
the same ranges, ``prepare`` makes what a program holds before the call (inputs on the GPU, the
plan or the resident batch), ``run`` is one pass through the public API, ``work`` the bytes and
operations that a pass cannot do without, and ``exact`` what ``run`` returns in 64 bits, by plain
torch and numpy.

Kinds of case:

* ``frame``     a firing simulated with a plan in hand and demodulated: simus_compute, rf2iq
* ``call``      the same from nothing but the scatterers: simus (plan included), rf2iq
* ``spectrum``  the selected-band spectrum of a firing: simus_gb300
* ``field``     the RMS pressure map of a firing: pfield_compute.  The package computes it in
                32 bits and widens it; the program keeps the map in 32 bits
* ``batch``     many firings on several phantoms: BatchedSimus.run ('fp32' and 'tc' backends)
* ``image``     delay-and-sum of many firings: rf2iq, das
* ``validate``  the transmit-field network against the exact field on fresh samples:
                TxFieldSurrogate.predict and .exact
* ``gradients`` one training step's gradients of that network: TxFieldSurrogate.gradients
"""

from __future__ import annotations

import math

import numpy as np
import torch

import fastsimus_gb300 as F
from fastsimus_gb300 import workloads as W
from fastsimus_gb300.batched import BatchedSimus
from fastsimus_gb300.beamform import DasParam, das, rf2iq
from fastsimus_gb300.surrogate import TxFieldSurrogate, cfg5_box

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")

# probe name -> (constructor, scatterer / grid box: x half-width, z range in m)
PROBES = {
    "lin64": (W.cfg1_probe, 10e-3, (5e-3, 30e-3)),
    "lin128": (W.cfg2_probe, 19e-3, (5e-3, 50e-3)),
    "P4-2v": (F.P4_2v, 20e-3, (8e-3, 60e-3)),
    "L11-5v": (F.L11_5v, 19e-3, (5e-3, 35e-3)),
    "L12-3v": (F.L12_3v, 19e-3, (5e-3, 35e-3)),
    "C5-2v": (F.C5_2v, 30e-3, (15e-3, 80e-3)),
}


def listed():
    return [
        # the smallest call: the 64-element probe's plain configuration, 2,000 scatterers
        {"name": "frame_2k", "kind": "frame", "probe": "lin64", "n_scat": 2000, "wave": "plane", "angle": 0.0,
         "apod": False, "atten": 0.0, "ffd": False},
        # the benchmark's frame: 128 elements, 200,000 scatterers, an attenuating medium
        {"name": "frame_200k", "kind": "frame", "probe": "lin128", "n_scat": 200_000, "wave": "plane", "angle": 0.0,
         "apod": False, "atten": 0.5, "ffd": False},
        # one call of the plain API on a 192-element linear array: focused, apodized firing, ragged count
        {"name": "call_192", "kind": "call", "probe": "L12-3v", "n_scat": 20_011, "wave": "focused", "angle": 6.0,
         "apod": True, "atten": 0.5, "ffd": False},
        # convex array with full-frequency directivity: the spectrum hook of a program with its own epilogue
        {"name": "spectrum_convex", "kind": "spectrum", "probe": "C5-2v", "n_scat": 15_001, "wave": "focused",
         "angle": 0.0, "apod": False, "atten": 0.5, "ffd": True},
        # the benchmark's pressure map, 256 x 512 points
        {"name": "field_map", "kind": "field", "probe": "lin128", "nx": 256, "nz": 512, "wave": "plane", "angle": 0.0,
         "apod": False, "atten": 0.5, "ffd": False},
        # a quick look at a focused beam of the phased array, odd grid
        {"name": "field_small", "kind": "field", "probe": "P4-2v", "nx": 81, "nz": 101, "wave": "focused",
         "angle": 10.0, "apod": True, "atten": 0.0, "ffd": False},
        # 75 plane waves on two phantoms in FP32
        {"name": "batch_fp32_75", "kind": "batch", "backend": "fp32", "n_tx": 75, "n_phantoms": 2, "n_scat": 30_000,
         "span": 16.0},
        # 31 plane waves, 262,144 scatterers, tensor cores
        {"name": "batch_tc_31", "kind": "batch", "backend": "tc", "n_tx": 31, "n_phantoms": 1, "n_scat": 262_144,
         "span": 12.0},
        # 75 plane waves on three uneven phantoms, tensor cores
        {"name": "batch_tc_75", "kind": "batch", "backend": "tc", "n_tx": 75, "n_phantoms": 3, "n_scat": 60_000,
         "span": 16.0},
        # the image of a 75-firing acquisition: demodulation and compounded delay-and-sum
        {"name": "image_75", "kind": "image", "probe": "lin64", "n_tx": 75, "n_samples": 1080, "nx": 256, "nz": 512,
         "span": 16.0, "method": "linear"},
        # validation of the transmit-field network on fresh samples
        {"name": "validate_1M", "kind": "validate", "n": 1 << 20},
        # a training step's gradients, 152 tiles of 128 rows
        {"name": "gradients_152", "kind": "gradients", "n_data": 200_000, "n_tiles": 152},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shot(rng):
    return {"wave": rng.choice(["plane", "plane", "focused"]), "angle": round(rng.uniform(-14.0, 14.0), 2),
            "apod": rng.random() < 0.3, "atten": rng.choice([0.0, 0.5]), "ffd": rng.random() < 0.15}


def draw(rng):
    kind = rng.choice(["frame", "frame", "call", "spectrum", "field", "field", "fp32", "tc", "tc", "image", "validate",
                       "gradients"])
    if kind in ("frame", "call", "spectrum"):
        probe = rng.choice(list(PROBES))
        top = 40_000 if probe in ("L11-5v", "L12-3v", "C5-2v") else 100_000
        return {"kind": kind, "probe": probe, "n_scat": _log(rng, 500, top), **_shot(rng)}
    if kind == "field":
        return {"kind": kind, "probe": rng.choice(list(PROBES)), "nx": _log(rng, 40, 256), "nz": _log(rng, 40, 400),
                **_shot(rng)}
    if kind == "fp32":
        return {"kind": "batch", "backend": "fp32", "n_tx": rng.randint(2, 75), "n_phantoms": rng.randint(1, 4),
                "n_scat": _log(rng, 1000, 20_000), "span": 16.0}
    if kind == "tc":
        return {"kind": "batch", "backend": "tc", "n_tx": rng.randint(2, 96), "n_phantoms": rng.randint(1, 4),
                "n_scat": _log(rng, 2000, 40_000), "span": 14.0}
    if kind == "image":
        return {"kind": kind, "probe": rng.choice(["lin64", "lin128", "L11-5v"]), "n_tx": _log(rng, 1, 75),
                "n_samples": rng.randint(700, 1800), "nx": _log(rng, 60, 256), "nz": _log(rng, 60, 512), "span": 14.0,
                "method": rng.choice(["linear", "linear", "nearest"])}
    if kind == "validate":
        return {"kind": kind, "n": _log(rng, 4000, 1_000_000)}
    return {"kind": kind, "n_data": _log(rng, 20_000, 200_000), "n_tiles": _log(rng, 8, 152)}


# ---- inputs -------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _probe(case):
    make, half, z = PROBES[case["probe"]]
    return make(), half, z


def _medium(case):
    return F.MediumParams(speed_of_sound=1540.0, attenuation=float(case.get("atten", 0.0)))


def _scatterers(n, half, z, seed):
    """n scatterers uniform over the box, four of them in its corners (so that the plan is the
    box's), reflectivity N(0, 1), zero inside one 2 mm cyst."""
    g = _gen(seed)
    r = torch.rand(n, 2, generator=g, dtype=torch.float64, device=DEV)
    lo = torch.tensor([-half, z[0]], dtype=torch.float64, device=DEV)
    hi = torch.tensor([half, z[1]], dtype=torch.float64, device=DEV)
    s = lo + r * (hi - lo)
    s[:4] = _corners(half, z)
    rc = torch.randn(n, generator=g, dtype=torch.float64, device=DEV)
    rc[(s[:, 0] ** 2 + (s[:, 1] - 0.5 * (z[0] + z[1])) ** 2) < 4e-6] = 0.0
    return s.contiguous(), rc.contiguous()


def _shot_law(case):
    """Delays (n_elements,) and apodization (n_elements,) or None of a firing, host FP64."""
    p, _, z = _probe(case)
    xe, te, apex = _elements(p)
    c, a = 1540.0, math.radians(case["angle"])
    if case["wave"] == "plane" and math.isinf(p.radius):
        d = xe[:, 0] * math.sin(a) / c
    else:
        zf = 0.6 * z[1]
        focus = np.array([zf * math.sin(a), zf * math.cos(a)])
        d = -np.sqrt(((xe - focus) ** 2).sum(-1)) / c
    apod = np.hanning(p.n_elements + 2)[1:-1] if case["apod"] else None
    return d - d.min(), apod


def _dev(a):
    return None if a is None else torch.as_tensor(np.ascontiguousarray(a), device=DEV)


def _grid(case):
    _, half, z = _probe(case)
    x, zz = np.meshgrid(np.linspace(-half, half, case["nx"]), np.linspace(z[0], z[1], case["nz"]))
    return x, zz


def _batch_inputs(case, seed):
    counts = [int(case["n_scat"] / (1.0 + 0.7 * i)) + 13 * i for i in range(case["n_phantoms"])]
    phantoms = [_scatterers(n, 10e-3, (5e-3, 30e-3), 1000 * seed + i) for i, n in enumerate(counts)]
    return phantoms, _plane_waves(W.cfg1_probe(), case["n_tx"], case["span"])


def _plane_waves(p, n_tx, span):
    xe, _, _ = _elements(p)
    a = np.radians(np.linspace(-span, span, n_tx))
    d = xe[None, :, 0] * np.sin(a)[:, None] / 1540.0
    return d - d.min(axis=1, keepdims=True)


def _echoes(case, seed):
    """RF (n_tx, n_samples, n_elements) float32 of 24 point targets, Gaussian-windowed pulses."""
    p, half, z = _probe(case)
    g = _gen(seed)
    xe = torch.as_tensor(_elements(p)[0][:, 0], device=DEV)
    txd = torch.as_tensor(_plane_waves(p, case["n_tx"], case["span"]), device=DEV)
    fs, ns = 4.0 * p.freq_center, case["n_samples"]
    t = torch.arange(ns, dtype=torch.float32, device=DEV) / fs
    rf = torch.zeros(case["n_tx"], ns, p.n_elements, device=DEV)
    r = torch.rand(24, 2, generator=g, dtype=torch.float64, device=DEV)
    amp = torch.randn(24, generator=g, dtype=torch.float64, device=DEV)
    for k in range(24):
        x, zz = (2 * r[k, 0] - 1) * half, z[0] + r[k, 1] * (z[1] - z[0])
        d = torch.sqrt((x - xe) ** 2 + zz * zz)
        arrive = ((txd * 1540.0 + d).amin(1)[:, None] + d) / 1540.0  # (n_tx, E)
        u = (t[None, :, None] - arrive.float()[:, None, :]) * p.freq_center
        rf += float(amp[k]) * torch.exp(-u * u) * torch.cos(2 * math.pi * u)
    return rf


def _samples(n, seed):
    """(n, 4) samples x, z, f, theta uniform over the network's box."""
    b = cfg5_box(W.cfg1_probe())
    r = torch.rand(n, 4, generator=_gen(seed), dtype=torch.float64, device=DEV)
    lo = torch.tensor([b.x[0], b.z[0], b.f[0], -b.max_angle], dtype=torch.float64, device=DEV)
    hi = torch.tensor([b.x[1], b.z[1], b.f[1], b.max_angle], dtype=torch.float64, device=DEV)
    return lo + r * (hi - lo)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("frame", "call", "spectrum"):
        p, half, z = _probe(case)
        m = _medium(case)
        s, rc = _scatterers(case["n_scat"], half, z, seed)
        d, a = _shot_law(case)
        st |= {"p": p, "m": m, "s": s, "rc": rc, "d": _dev(d), "a": _dev(a), "fs": 4.0 * p.freq_center}
        if kind != "call":
            st["plan"] = F.simus_precompute(s, rc, d, p, m)
    elif kind == "field":
        p, _, _ = _probe(case)
        m = _medium(case)
        x, z = _grid(case)
        # grids of the same shape, moved sideways by up to half a wavelength
        shift = float(torch.rand(1, generator=_gen(seed), device=DEV, dtype=torch.float64)) * 1e-4
        pos = _dev(np.stack([x + shift, z], axis=-1))
        d, a = _shot_law(case)
        st |= {"p": p, "m": m, "pos": pos, "d": _dev(d), "a": _dev(a), "plan": F.pfield_precompute(pos, d, p, m)}
    elif kind == "batch":
        phantoms, delays = _batch_inputs(case, seed)
        st["b"] = BatchedSimus(phantoms, delays, W.cfg1_probe(), W.cfg1_medium(), backend=case["backend"])
    elif kind == "image":
        p, _, _ = _probe(case)
        x, z = _grid(case)
        st |= {"p": p, "rf": _echoes(case, seed), "x": x, "z": z, "fs": 4.0 * p.freq_center,
               "txd": _plane_waves(p, case["n_tx"], case["span"]), "param": DasParam.from_params(p, W.cfg1_medium())}
    elif kind == "validate":
        p = W.cfg1_probe()
        st |= {"sur": TxFieldSurrogate(p, W.cfg1_medium(), cfg5_box(p), seed=seed), "q": _samples(case["n"], seed)}
    else:
        p = W.cfg1_probe()
        sur = TxFieldSurrogate(p, W.cfg1_medium(), cfg5_box(p), seed=seed)
        q = _samples(case["n_data"], seed)
        field = sur.exact(q)
        sur.scale = float(torch.sqrt((field.abs().double() ** 2).mean()))
        u, aux = sur.inputs(q, field)
        st |= {"sur": sur, "u": u, "aux": aux, "seed": seed}
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "frame":
        r = F.simus_compute(st["s"], st["rc"], st["d"], st["plan"], st["p"], st["m"], tx_apodization=st["a"],
                            full_frequency_directivity=case["ffd"])
        return rf2iq(r.rf, st["fs"], st["p"].freq_center)
    if kind == "call":
        r = F.simus(st["s"], st["rc"], st["d"], st["p"], st["m"], tx_apodization=st["a"],
                    full_frequency_directivity=case["ffd"])
        return rf2iq(r.rf, st["fs"], st["p"].freq_center)
    if kind == "spectrum":
        return F.simus_gb300(st["s"], st["rc"], st["p"], st["plan"], st["m"], st["d"], st["a"],
                             full_frequency_directivity=case["ffd"])
    if kind == "field":
        return F.pfield_compute(st["pos"], st["d"], st["plan"], st["p"], st["m"], tx_apodization=st["a"],
                                full_frequency_directivity=case["ffd"]).float()
    if kind == "batch":
        return [[r.rf, r.spectrum] for r in st["b"].run()]
    if kind == "image":
        iq = rf2iq(st["rf"], st["fs"], st["p"].freq_center)
        return das(iq, st["x"], st["z"], st["txd"], st["param"], method=case["method"])
    if kind == "validate":
        return {"predicted": st["sur"].predict(st["q"]), "exact": st["sur"].exact(st["q"])}
    gw, gb, rows = st["sur"].gradients(st["u"], st["aux"], n_tiles=case["n_tiles"], n_split=15, seed=st["seed"])
    return {"w": gw, "b": gb, "rows": rows}


# ---- work ---------------------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("frame", "call", "spectrum"):
        p, half, z = _probe(case)
        plan = _simus_plan(_corners(half, z), _shot_law(case)[0], p)
        E, n = p.n_elements, case["n_scat"]
        terms = float(n) * plan["f"].size * E
        return {"bytes": 24.0 * n + 8.0 * E * plan["n_fft"] / 2, "flops": terms * (8 * plan["U"] + 16)}
    if kind == "field":
        p, half, z = _probe(case)
        plan = _field_plan(_corners(half, z), _shot_law(case)[0], p)
        n = case["nx"] * case["nz"]
        return {"bytes": 24.0 * n, "flops": 8.0 * n * plan["f"].size * p.n_elements * plan["U"]}
    if kind == "batch":
        p = W.cfg1_probe()
        plan = _simus_plan(_corners(10e-3, (5e-3, 30e-3)), _plane_waves(p, case["n_tx"], case["span"])[0], p)
        n = sum(int(case["n_scat"] / (1.0 + 0.7 * i)) + 13 * i for i in range(case["n_phantoms"]))
        out = 64.0 * case["n_tx"] * case["n_phantoms"] * (8 * plan["n_full"] + 4 * plan["n_fft"] / 2)
        return {"bytes": 24.0 * n + out, "flops": float(n) * plan["f"].size * 64 * (8 * plan["U"] + 16 * case["n_tx"])}
    if kind == "image":
        p, _, _ = _probe(case)
        rf = case["n_tx"] * case["n_samples"] * p.n_elements
        pix = case["nx"] * case["nz"]
        return {"bytes": 4.0 * rf + 24.0 * pix, "flops": 120.0 * rf + 20.0 * pix * case["n_tx"] * p.n_elements}
    if kind == "validate":
        return {"bytes": 48.0 * case["n"], "flops": case["n"] * (463_872.0 + 128 * 40)}
    return {"bytes": 48.0 * 128 * case["n_tiles"], "flops": 3 * 463_872.0 * 128 * case["n_tiles"]}


# ---- 64-bit reference, plain torch and numpy ------------------------------------------------------


def _corners(half, z):
    return torch.tensor([[-half, z[0]], [half, z[0]], [-half, z[1]], [half, z[1]]], dtype=torch.float64, device=DEV)


def _elements(p):
    """Element centres (E, 2), angles (E,), apex offset.  Linear x positions are float32 products."""
    n = p.n_elements
    if math.isinf(p.radius):
        x = (np.arange(n, dtype=np.float32) - np.float32((n - 1) / 2)) * np.float32(p.pitch)
        return np.stack([x.astype(np.float64), np.zeros(n)], -1), np.zeros(n), 0.0
    half = math.asin(p.pitch / 2 / p.radius)
    chord = 2 * p.radius * math.sin(half * (n - 1))
    apex = math.sqrt(p.radius**2 - (chord / 2) ** 2)
    th = np.linspace(math.atan2(-chord / 2, apex), math.atan2(chord / 2, apex), n)
    return np.stack([p.radius * np.sin(th), p.radius * np.cos(th) - apex], -1), th, apex


def _n_sub(p):
    return math.ceil(p.element_width / (1540.0 / (p.freq_center * (1.0 + p.bandwidth / 2.0))))


def _sources(p):
    U = _n_sub(p)
    xe, th, _ = _elements(p)
    seg = p.element_width / U
    off = np.array([-p.element_width / 2 + seg / 2 + i * seg for i in range(U)])
    d = np.stack([off * np.cos(th)[:, None], -off * np.sin(th)[:, None]], -1)
    return (xe[:, None, :] + d).reshape(-1, 2)


def _pulse(f, p):
    w, wc, dur = 2 * np.pi * f, 2 * np.pi * p.freq_center, 1.0 / p.freq_center
    return 1j * (np.sinc(dur * (w - wc) / 2 / np.pi) - np.sinc(dur * (w + wc) / 2 / np.pi))


def _response(f, p):
    w, wc = 2 * np.pi * f, 2 * np.pi * p.freq_center
    shape = math.log(126) / math.log(2 / p.bandwidth)
    sigma = p.bandwidth * wc / 2 / math.log(2) ** (1 / shape)
    return np.sqrt(np.exp(-((np.abs(w - wc) / sigma) ** shape)))


def _band(p, df):
    n = int(2 * math.ceil(p.freq_center / df) + 1)
    f = np.linspace(0, 2 * p.freq_center, n)
    mag = np.abs(_pulse(f, p) * _response(f, p))
    keep = np.nonzero(20 * np.log10(1e-200 + mag / mag.max()) > -60.0)[0]
    f = f[keep[0]:keep[-1] + 1]
    return {"f": f, "pulse": _pulse(f, p), "resp": _response(f, p), "df": 2 * p.freq_center / (n - 1), "n_full": n,
            "k0": int(keep[0]), "U": _n_sub(p)}


def _farthest(points, targets):
    t, best = torch.as_tensor(targets, device=points.device), 0.0
    for q in points.split(1 << 16):
        best = max(best, float(torch.sqrt((q[:, None, 0] - t[:, 0]) ** 2 + (q[:, None, 1] - t[:, 1]) ** 2).max()))
    return best


def _simus_plan(points, delays, p):
    fc, dt = p.freq_center, 1e-9
    n_fft = 2 ** math.ceil(math.log2(1 / dt / 2 / (fc / 32)))
    f = np.linspace(0, 1 / dt / 2, n_fft)
    two = np.fft.fftshift(np.fft.irfft(_pulse(f, p) * _response(f, p) ** 2))
    above = np.nonzero(two / np.abs(two).max() > 1 / 1023)[0]
    trim = min(above[0] + 1, 2 * n_fft - 1 - above[-1] - 1)
    far = _farthest(points, _elements(p)[0]) + len(two[-trim:trim - 2:-1]) * dt * 1540.0
    plan = _band(p, 0.5 / (2 * far / 1540.0 + float(np.max(delays))))
    return plan | {"n_fft": math.ceil(4 * fc / 2 / fc * (plan["n_full"] - 1))}


def _field_plan(points, delays, p):
    far = max(_farthest(points, _sources(p)), 1540.0 / p.freq_center / 2)
    return _band(p, 1.0 / (far / 1540.0 + float(np.max(delays))))


def _green(points, p, f0, df, atten, ffd, U):
    """First term and per-step factor (n, E, U) complex128, sin(theta), in-field mask."""
    xe, th, apex = _elements(p)
    src = torch.as_tensor(_sources(p), device=DEV).reshape(p.n_elements, U, 2)
    te = torch.as_tensor(th, device=DEV)[:, None]
    dx, dz = points[:, None, None, 0] - src[..., 0], points[:, None, None, 1] - src[..., 1]
    r = torch.sqrt(dx * dx + dz * dz)
    theta = torch.asin((dx + 1e-16) / (r + 1e-16)) - te
    r = torch.clamp(r, min=1540.0 / p.freq_center / 2)
    ob = torch.where(theta.abs() >= math.pi / 2, torch.full_like(theta, 1e-16), torch.cos(theta))
    neper = atten / (20 / math.log(10)) / 1e6 * 1e2
    st = torch.sin(theta)
    amp = ob / torch.sqrt(r) / U
    if not ffd:
        amp = amp * torch.sinc(p.freq_center / 1540.0 * p.element_width / U * st)
    g = torch.polar(amp * torch.exp(-neper * f0 * r), 2 * math.pi * f0 / 1540.0 * r)
    step = torch.polar(torch.exp(-neper * df * r), 2 * math.pi * df / 1540.0 * r)
    out = points[:, 1] < 0
    if not math.isinf(p.radius):
        out |= points[:, 0] ** 2 + (points[:, 1] + apex) ** 2 <= p.radius**2
    return g, step, st, ~out


def _weighted(g, st, f, p, U, ffd):
    """Sub-element sums (n, E) at frequency f."""
    return (g * torch.sinc(f / 1540.0 * p.element_width / U * st)).sum(-1) if ffd else g.sum(-1)


def _sweep(s, rc, delays, apod, p, plan, atten, ffd, chunk=50_000):
    """Spectra (F, E, n_tx) of a phantom, before the correction factor."""
    f, U, E = plan["f"], plan["U"], p.n_elements
    df = float(f[1] - f[0])
    ftau = torch.as_tensor(f, device=DEV)[:, None, None] * torch.as_tensor(delays, device=DEV)  # (F, n_tx, E)
    law = torch.polar(torch.ones_like(ftau), 2 * math.pi * (ftau - torch.floor(ftau)))
    if apod is not None:
        law = law * torch.as_tensor(apod, device=DEV)
    out = torch.zeros(f.size, E, law.shape[1], dtype=torch.complex128, device=DEV)
    for i in range(0, s.shape[0], chunk):
        g, step, st, ok = _green(s[i:i + chunk], p, float(f[0]), df, atten, ffd, U)
        w = torch.where(ok, rc[i:i + chunk], torch.zeros_like(rc[i:i + chunk])).to(torch.complex128)
        for k in range(f.size):
            m = _weighted(g, st, float(f[k]), p, U, ffd)
            pr = (m @ law[k].T) * w[:, None]
            out[k] += m.T @ pr
            g = g * step
    scale = plan["pulse"] * plan["resp"] * plan["resp"]
    return out * torch.as_tensor(scale, device=DEV)[:, None, None]


def _rf(sel, plan, p):
    """RF (n_samples, E, n_tx) and full spectrum of selected-band spectra (F, E, n_tx)."""
    full = torch.zeros(plan["n_full"], *sel.shape[1:], dtype=torch.complex128, device=DEV)
    full[plan["k0"]:plan["k0"] + sel.shape[0]] = sel * (plan["df"] * p.element_width)
    n = plan["n_fft"]
    rf = torch.fft.irfft(full.conj().resolve_conj(), n=n, dim=0)[: (n + 1) // 2]
    rel = rf.abs() / (rf.abs().amax(dim=(0, 1), keepdim=True) + 1e-30)
    return rf * (0.5 * (1 + torch.tanh((rel - 1e-5) / 1e-6))), full


def _lowpass(wn, order=5):
    """Second-order sections (b0, b1, b2, a1, a2) of the Butterworth low-pass, bilinear transform."""
    k = 4 * math.tan(math.pi * wn / 2)
    poles = [k * complex(math.cos(t), math.sin(t)) for t in
             (math.pi * (2 * i + order + 1) / (2 * order) for i in range((order + 1) // 2))]
    sos = []
    for s in poles:
        z = (4 + s) / (4 - s)
        if abs(s.imag) < 1e-9 * abs(s):
            g = (1 - z.real) / 2
            sos.append((g, g, 0.0, -z.real, 0.0))
        else:
            g = abs(1 - z) ** 2 / 4
            sos.append((g, 2 * g, g, -2 * z.real, abs(z) ** 2))
    return sos


def _filter(x, sos):
    """The cascade along the first axis, started in its steady state for the first sample."""
    y = np.array(x)
    for b0, b1, b2, a1, a2 in sos:
        gain = (b0 + b1 + b2) / (1 + a1 + a2)
        z1, z2 = (gain - b0) * y[0], (b2 - a2 * gain) * y[0]
        for n in range(y.shape[0]):
            v = y[n]
            o = b0 * v + z1
            z1, z2 = b1 * v - a1 * o + z2, b2 * v - a2 * o
            y[n] = o
    return y


def _iq(rf, fs, fc):
    """I/Q (n_samples, ...) complex128 of RF, forward and backward, odd padding of 18 samples."""
    n, pad = rf.shape[0], 18
    t = (np.arange(n) / fs).reshape((n,) + (1,) * (rf.ndim - 1))
    x = rf * np.exp(-2j * np.pi * fc * t)
    x = np.concatenate([2 * x[0] - x[pad:0:-1], x, 2 * x[-1] - x[-2:-pad - 2:-1]])
    sos = _lowpass(min(2 * fc / fs, 0.5))
    return 2 * _filter(_filter(x, sos)[::-1], sos)[::-1][pad:pad + n]


def _fnumber(p):
    lam, lo, hi = 1540.0 / p.freq_center, 0.0, math.pi / 2
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        inside = np.sinc(p.element_width / lam * math.sin(mid)) * math.cos(mid) > 1 / math.sqrt(2)
        lo, hi = (mid, hi) if inside else (lo, mid)
    return 1 / (2 * math.tan(0.5 * (lo + hi)))


def _image(case, iq):
    """Compounded delay-and-sum (nz, nx) complex128 of iq (n_tx, n_samples, E)."""
    p, _, _ = _probe(case)
    fs, fc, ns = 4.0 * p.freq_center, p.freq_center, case["n_samples"]
    x, z = _grid(case)
    px, pz = (torch.as_tensor(a.reshape(-1), device=DEV)[:, None] for a in (x, z))
    xe = torch.as_tensor((np.arange(p.n_elements) - 0.5 * (p.n_elements - 1)) * p.pitch, device=DEV)
    d = torch.sqrt((px - xe) ** 2 + pz**2)
    inside = (px - xe).abs() <= pz / (2 * _fnumber(p))
    txd = torch.as_tensor(_plane_waves(p, case["n_tx"], case["span"]), device=DEV)
    img = torch.zeros(px.shape[0], dtype=torch.complex128, device=DEV)
    col = torch.arange(p.n_elements, device=DEV)[None, :] * ns
    for k in range(case["n_tx"]):
        sig = torch.as_tensor(np.ascontiguousarray(iq[k].T), device=DEV).reshape(-1)
        t = ((1540.0 * txd[k] + d).amin(1, keepdim=True) + d) / 1540.0
        s = t * fs
        i = torch.floor(s if case["method"] == "linear" else s + 0.5)
        last = ns - 1 if case["method"] == "linear" else ns
        ok = inside & (i >= 0) & (i < last)
        j = torch.where(ok, i, torch.zeros_like(i)).long() + col
        v = sig[j]
        if case["method"] == "linear":
            w = s - i
            v = v + w * (sig[torch.where(ok, j + 1, j)] - v)
        cyc = fc * t
        img += torch.where(ok, v * torch.polar(torch.ones_like(cyc), 2 * math.pi * (cyc - torch.floor(cyc))),
                           torch.zeros_like(v)).sum(1)
    return img.reshape(x.shape)


def _network(seed, n_carriers=5):
    """The surrogate's initial parameters: Fourier matrix, weights (hidden ones in bf16), biases."""
    g = torch.Generator().manual_seed(seed)
    bmat = torch.randn(64, 4, generator=g) * 0.5
    ws, bs = [], []
    for o, i in [(256, 128)] + [(256, 256)] * 3 + [(2 * n_carriers, 256)]:
        ws.append((torch.rand(o, i, generator=g) * 2 - 1) / math.sqrt(i))
        bs.append((torch.rand(o, generator=g) * 2 - 1) / math.sqrt(i))
    ws = [w.bfloat16() if k < 4 else w for k, w in enumerate(ws)]
    return bmat.double().to(DEV), [w.double().to(DEV) for w in ws], [b.double().to(DEV) for b in bs]


def _units(q):
    b = cfg5_box(W.cfg1_probe())
    lo = torch.tensor([b.x[0], b.z[0], b.f[0], -b.max_angle], dtype=torch.float64, device=DEV)
    hi = torch.tensor([b.x[1], b.z[1], b.f[1], b.max_angle], dtype=torch.float64, device=DEV)
    return ((2 * q - (lo + hi)) / (hi - lo)).float().double()


def _forward(u, net):
    bmat, ws, bs = net
    t = 2 * math.pi * (u @ bmat.T)
    a = torch.cat([torch.sin(t), torch.cos(t)], 1)
    for w, b in zip(ws[:-1], bs[:-1]):
        a = torch.nn.functional.silu(a @ w.T + b)
    return a @ ws[-1].T + bs[-1]


def _waves(q, p):
    """The five analytic carriers (n, 5) complex128."""
    x, z, f, th = q.unbind(1)
    st, x0 = torch.sin(th), -0.5 * (p.n_elements - 1) * p.pitch
    first = torch.minimum(x0 * st, -x0 * st)
    paths = [x * st + z * torch.cos(th)]
    paths += [torch.sqrt((x - xe) ** 2 + z * z) + xe * st for xe in (x0 - p.pitch / 2, -x0 + p.pitch / 2)]
    on = [torch.ones_like(x)] * 3
    for m in (-1, 1):
        sm = st + m * 1540.0 / f / p.pitch
        paths.append(x * sm + z * torch.sqrt(torch.clamp(1 - sm * sm, min=0)))
        on.append((sm.abs() < 1).double())
    cyc = torch.stack([f / 1540.0 * (a - first) for a in paths], 1)
    return torch.polar(torch.stack(on, 1), 2 * math.pi * (cyc - torch.floor(cyc)))


def _transmit(q, p):
    """The exact transmit pressure (n,) complex128 at samples (x, z, f, theta), unit apodization."""
    U = _n_sub(p)
    xe = torch.as_tensor(_elements(p)[0][:, 0], device=DEV)
    out = []
    for c in q.split(32_768):
        f, st = c[:, 2], torch.sin(c[:, 3])
        tau = xe[None, :] * st[:, None]
        tau = (tau - tau.amin(1, keepdim=True)) / 1540.0
        g, _, _, _ = _green(c[:, :2], p, 0.0, 0.0, 0.0, False, U)  # amplitudes
        src = torch.as_tensor(_sources(p), device=DEV)
        r = torch.sqrt((c[:, None, 0] - src[:, 0]) ** 2 + (c[:, None, 1] - src[:, 1]) ** 2)
        r = torch.clamp(r, min=1540.0 / p.freq_center / 2).reshape(g.shape)
        cyc = f[:, None, None] * (r / 1540.0 + tau[:, :, None])
        s = torch.polar(g.real, 2 * math.pi * (cyc - torch.floor(cyc))).sum((1, 2))
        fn = f.cpu().numpy()
        out.append(s * torch.as_tensor(_pulse(fn, p) * _response(fn, p), device=DEV))
    return torch.cat(out)


def _rows(seed, n_tiles, n_data):
    """The data rows a training step draws: splitmix64 of the seed and the row's number."""
    with np.errstate(over="ignore"):
        h = np.uint64(seed) ^ np.arange(128 * n_tiles, dtype=np.uint64)
        h = h + np.uint64(0x9E3779B97F4A7C15)
        h = (h ^ (h >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        h = (h ^ (h >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return torch.as_tensor(((h ^ (h >> np.uint64(31))) % np.uint64(n_data)).astype(np.int64), device=DEV)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("frame", "call", "spectrum"):
        p, half, z = _probe(case)
        s, rc = _scatterers(case["n_scat"], half, z, seed)
        d, a = _shot_law(case)
        plan = _simus_plan(s, d, p)
        sel = _sweep(s, rc, d[None], a, p, plan, float(case["atten"]), case["ffd"])
        if kind == "spectrum":
            return sel[..., 0]
        return _iq(_rf(sel, plan, p)[0][..., 0].cpu().numpy(), 4.0 * p.freq_center, p.freq_center)
    if kind == "field":
        p, _, _ = _probe(case)
        x, z = _grid(case)
        shift = float(torch.rand(1, generator=_gen(seed), device=DEV, dtype=torch.float64)) * 1e-4
        pos = _dev(np.stack([x + shift, z], axis=-1).reshape(-1, 2))
        d, a = _shot_law(case)
        plan = _field_plan(pos, d, p)
        f = plan["f"]
        w = np.ones(p.n_elements) if a is None else a
        out = []
        for c in pos.split(16_384):
            g, step, st, ok = _green(c, p, float(f[0]), float(f[1] - f[0]), float(case["atten"]), case["ffd"],
                                     plan["U"])
            acc = torch.zeros(c.shape[0], dtype=torch.float64, device=DEV)
            for k in range(f.size):
                law = _dev(w * np.exp(2j * np.pi * f[k] * d))
                v = (_weighted(g, st, float(f[k]), p, plan["U"], case["ffd"]) @ law)
                acc += (v.abs() * abs(plan["pulse"][k] * plan["resp"][k])) ** 2
                g = g * step
            out.append(torch.where(ok, torch.sqrt(acc * plan["df"] * p.element_width), torch.zeros_like(acc)))
        return torch.cat(out).reshape(x.shape)
    if kind == "batch":
        p = W.cfg1_probe()
        phantoms, delays = _batch_inputs(case, seed)
        out = []
        for s, rc in phantoms:
            plan = _simus_plan(s, delays[int(np.argmax(np.ptp(delays, axis=1)))], p)
            out.append(list(_rf(_sweep(s, rc, delays, None, p, plan, 0.0, False), plan, p)))
        return out
    if kind == "image":
        p, _, _ = _probe(case)
        rf = _echoes(case, seed).double().permute(1, 0, 2).cpu().numpy()
        return _image(case, _iq(rf, 4.0 * p.freq_center, p.freq_center).transpose(1, 0, 2))
    p = W.cfg1_probe()
    net = _network(seed)
    if kind == "validate":
        q = _samples(case["n"], seed)
        pred = [(torch.view_as_complex(_forward(_units(c), net).reshape(-1, 5, 2)) * _waves(c, p)).sum(1)
                for c in q.split(131_072)]
        return {"predicted": torch.cat(pred), "exact": _transmit(q, p)}
    q = _samples(case["n_data"], seed)
    field = _transmit(q, p)
    scale = float(torch.sqrt((field.abs() ** 2).mean()))
    rows = _rows(seed, case["n_tiles"], case["n_data"])
    for t in net[1] + net[2]:
        t.requires_grad_(True)
    amp = torch.view_as_complex(_forward(_units(q[rows]), net).reshape(-1, 5, 2))
    err = (amp * _waves(q[rows], p)).sum(1) - field[rows] / scale
    (err.abs() ** 2).mean().backward()
    return {"w": [t.grad for t in net[1]], "b": [t.grad for t in net[2]], "rows": None}
