"""What this library is measured on: spectra, gradients, distributions, histograms and
inverse-Compton emission through the entry points that a program calls, over the sizes
that post-processing of particle simulations and spectral fits use.

``listed()`` are the fixed cases and ``draw(rng)`` makes more of the same ranges;
``prepare`` makes a case's inputs on the GPU from a seed, ``run`` is one pass through the
library, ``work`` the bytes and operations a pass cannot do without, and ``exact`` the
result in 64 bits by plain torch.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

DEV = "cuda:0"


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------

def listed():
    return [
        # A few thousand tracked particles, spectrum and energy histogram through the drop-in
        # module: a call is launches, allocations and copies.
        {"name": "species_10k", "kind": "species", "n": 10007, "nbins": 100, "nhist": 100, "index": -2.0,
         "umax": 100.0, "gcut": 0.0, "b": "z", "weights": False},
        # One species of the small benchmark configuration (1e6 particles x 200 bins, and the
        # 200-bin energy distribution of the same particles), drop-in module.
        {"name": "species_1m", "kind": "species", "n": 1000000, "nbins": 200, "nhist": 200, "index": -2.0,
         "umax": 100.0, "gcut": 0.0, "b": "z", "weights": False},
        # A Tristan-v2 dump: three species of 3.3e7 particles x 512 bins, the pairs as one
        # batched run and the protons as another (the benchmark's step).
        {"name": "dump_3x33m", "kind": "dump", "n": 33000000, "nbins": 512},
        # Particles in electric and magnetic fields, an odd count that leaves streams of no
        # round size, the reference's table through the torch extension.
        {"name": "fields_4m", "kind": "fields", "n": 4300001, "nbins": 300, "index": -2.2, "umax": 1e4, "weights": True},
        # Spectra of 256 uneven subvolumes in one batched run.
        {"name": "segments_256", "kind": "segments", "nseg": 256, "lo": 1e4, "hi": 1e6, "nbins": 200},
        # The differentiable spectrum of 1e7 particles x 512 bins and the gradients of weights
        # and four-velocities under a loss of the program's own (its derivative given).
        {"name": "gradient_10m", "kind": "gradient", "n": 10000000, "nbins": 512, "b": "z", "index": -2.0, "umax": 100.0,
         "log_loss": False},
        # A training step of a small fit, with the library's log-space loss: an odd handful of
        # particles, where launches count.
        {"name": "gradient_20k", "kind": "gradient", "n": 20011, "nbins": 128, "b": "iso", "index": -2.3, "umax": 1e3,
         "log_loss": True},
        # 4096 tabulated distributions mapped to 1024 photon bins (the tensor-core product).
        {"name": "fromdist_4096", "kind": "fromdist", "ndist": 4096, "ng": 1024, "nbins": 1024, "gmax": 1e6},
        # A fit step of 1024 distributions x 512 gamma bins x 512 photon bins: spectra, loss and
        # the gradient with respect to the distributions (both directions of the product).
        {"name": "fit_1024", "kind": "fit", "ndist": 1024, "ng": 512, "nbins": 512, "gmax": 1e5},
        # One tabulated distribution through the drop-in module, as its scripts call it.
        {"name": "one_dist", "kind": "onedist", "ng": 1000, "nbins": 512, "gmax": 1e6},
        # Energy distribution of one dump species, drop-in module: bytes read once.
        {"name": "histogram_33m", "kind": "histogram", "n": 33000000, "nhist": 200, "log": True, "fourvel": True},
        # Inverse-Compton spectrum of a tabulated distribution on tabulated soft photons.
        {"name": "ic_1024", "kind": "ic", "ng": 1024, "ns": 1024, "ne": 1024, "delta": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["species", "dump", "fields", "segments", "gradient", "fromdist", "fit", "onedist",
                       "histogram", "ic"])
    if kind == "species":
        return {"kind": kind, "n": _log_int(rng, 1000, 4e6), "nbins": _log_int(rng, 24, 700),
                "nhist": _log_int(rng, 16, 700), "index": rng.uniform(-3.0, -1.5),
                "umax": math.exp(rng.uniform(math.log(20.0), math.log(1e4))), "gcut": 0.0,
                "b": rng.choice(["z", "iso"]), "weights": rng.random() < 0.5}
    if kind == "dump":
        return {"kind": kind, "n": _log_int(rng, 1e6, 3.3e7), "nbins": _log_int(rng, 128, 512)}
    if kind == "fields":
        return {"kind": kind, "n": _log_int(rng, 3e3, 1.2e7), "nbins": _log_int(rng, 32, 600),
                "index": rng.uniform(-3.0, -1.5), "umax": math.exp(rng.uniform(math.log(50.0), math.log(1e4))),
                "weights": rng.random() < 0.5}
    if kind == "segments":
        hi = math.exp(rng.uniform(math.log(2e3), math.log(1e6)))
        return {"kind": kind, "nseg": _log_int(rng, 2, 256), "lo": max(100.0, 1e-2 * hi), "hi": hi,
                "nbins": _log_int(rng, 32, 300)}
    if kind == "gradient":
        return {"kind": kind, "n": _log_int(rng, 3e3, 1e7), "nbins": _log_int(rng, 32, 512),
                "b": rng.choice(["z", "iso"]), "index": rng.uniform(-3.0, -1.5),
                "umax": math.exp(rng.uniform(math.log(50.0), math.log(3e3))), "log_loss": rng.random() < 0.5}
    if kind in ("fromdist", "fit"):
        return {"kind": kind, "ndist": _log_int(rng, 8, 4096 if kind == "fromdist" else 2048),
                "ng": _log_int(rng, 100, 1024), "nbins": _log_int(rng, 100, 1024 if kind == "fromdist" else 700),
                "gmax": math.exp(rng.uniform(math.log(1e4), math.log(1e6)))}
    if kind == "onedist":
        return {"kind": kind, "ng": _log_int(rng, 50, 8000), "nbins": _log_int(rng, 32, 1024),
                "gmax": math.exp(rng.uniform(math.log(1e4), math.log(1e6)))}
    if kind == "histogram":
        return {"kind": kind, "n": _log_int(rng, 1e4, 3.3e7), "nhist": _log_int(rng, 16, 2000),
                "log": rng.random() < 0.75, "fourvel": rng.random() < 0.75}
    return {"kind": kind, "ng": _log_int(rng, 64, 1024), "ns": _log_int(rng, 32, 1024), "ne": _log_int(rng, 32, 1024),
            "delta": rng.random() < 0.25}


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(n, gen):
    return torch.rand(n, device=DEV, generator=gen, dtype=torch.float64)


def _powerlaw(n, gen, index, lo, hi, gcut):
    """|u| ~ |u|^index on [lo, hi], times exp(-gamma / gcut) when gcut > 0 (by rejection)."""
    q = index + 1.0
    out = torch.empty(0, device=DEV)
    while out.numel() < n:
        m = n if gcut <= 0.0 else int((n - out.numel()) * 1.2) + 1024
        r = _rand(m, gen)
        u = lo * (hi / lo) ** r if abs(q) < 1e-9 else ((hi**q - lo**q) * r + lo**q) ** (1.0 / q)
        if gcut > 0.0:
            u = u[_rand(m, gen) < torch.exp(-torch.sqrt(1.0 + u * u) / gcut)]
        out = torch.cat([out, u.float()])
    return out[:n].contiguous()


def _isotropic(mag, gen):
    n = mag.numel()
    mu = (2.0 * _rand(n, gen) - 1.0).float()
    ph = (2.0 * math.pi * _rand(n, gen)).float()
    s = torch.sqrt(torch.clamp(1.0 - mu * mu, min=0.0))
    return [mag * s * torch.cos(ph), mag * s * torch.sin(ph), mag * mu]


def _bfield(n, gen, kind):
    if kind == "z":
        zero = torch.zeros(n, device=DEV)
        return [zero, zero.clone(), torch.ones(n, device=DEV)]
    return _isotropic(torch.exp(0.5 * torch.randn(n, device=DEV, generator=gen)), gen)


def _particles(case, seed, n=None, index=None, gcut=None):
    """(u, b, e or None, w or None) of a case with one population."""
    gen = _gen(seed)
    n = n or case["n"]
    u = _isotropic(_powerlaw(n, gen, case["index"] if index is None else index, 1.0, case["umax"],
                             case.get("gcut", 0.0) if gcut is None else gcut), gen)
    b = _bfield(n, gen, case.get("b", "iso"))
    e = _isotropic(0.3 * _rand(n, gen).float(), gen) if case["kind"] == "fields" else None
    w = (_rand(n, gen) + 0.5).float() if case.get("weights") else None
    return u, b, e, w


SPECIES_EPS = (1.0, 1.0, 1.0 / 1836.0)  # e-, e+ and protons: e_syn_at_g_syn


def _dump_particles(case, seed):
    """Seven streams holding the three species back to back."""
    n = case["n"]
    comps = [torch.empty(3 * n, device=DEV) for _ in range(7)]
    for s in range(3):
        gen = _gen(int(seed) * 11 + s)
        u = _isotropic(_powerlaw(n, gen, -2.2, 1.0, 1e4, 3e3), gen)
        b = _isotropic(torch.exp(0.5 * torch.randn(n, device=DEV, generator=gen)), gen)
        w = (_rand(n, gen) + 0.5).float()
        for k, v in enumerate(u + b + [w]):
            comps[k][s * n:(s + 1) * n] = v
    return comps


def _segment_inputs(case, seed):
    """Uneven segments (log-uniform counts), each with a power-law index of its own."""
    r = np.random.default_rng(int(seed))
    counts = np.floor(np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["nseg"]))).astype(np.int64)
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    n = int(offs[-1])
    gen = _gen(seed)
    q = torch.from_numpy(1.0 + r.uniform(-3.0, -1.5, case["nseg"])).to(DEV)
    qp = torch.repeat_interleave(q, torch.from_numpy(counts).to(DEV))
    qp = torch.where(qp.abs() < 1e-6, torch.full_like(qp, 1e-6), qp)
    mag = (((100.0**qp - 1.0) * _rand(n, gen) + 1.0) ** (1.0 / qp)).float()
    u = _isotropic(mag, gen)
    return offs, u, torch.ones(n, device=DEV)


def _logbins(lo, hi, n):
    """Log-spaced bins as a program makes them with numpy."""
    return np.logspace(math.log10(lo), math.log10(hi), n).astype(np.float32)


def _species_bins(case):
    return _logbins(1e-2, 1e7 if case["umax"] <= 200.0 else 1e9, case["nbins"])


def _distributions(case, seed):
    """Power laws with random indices, breaks and cutoffs on log gamma bins."""
    gen = _gen(seed)
    g = _logbins(1.0, case["gmax"], case["ng"])
    gt = torch.from_numpy(g).to(DEV).double()[None, :]
    d = case.get("ndist", 1)
    p1 = (-3.0 + 1.5 * _rand(d, gen))[:, None]
    p2 = (-3.5 + 2.3 * _rand(d, gen))[:, None]
    lg = math.log(case["gmax"])
    gb = torch.exp(0.2 * lg + 0.5 * lg * _rand(d, gen))[:, None]
    gc = torch.exp(0.5 * lg + 0.5 * lg * _rand(d, gen))[:, None]
    f = torch.where(gt < gb, gt**p1, gb ** (p1 - p2) * gt**p2) * torch.exp(-gt / gc)
    return g, torch.clamp(f, min=1e-30).float().contiguous()


def _dist_bins(case):
    return _logbins(1e-2, 10.0 * case["gmax"] ** 2, case["nbins"])


def _ic_inputs(case, seed):
    gen = _gen(seed)
    g = _logbins(1e1, 1e6, case["ng"])
    gt = torch.from_numpy(g).to(DEV).double()
    f = (gt ** (-2.8 + 1.2 * float(_rand(1, gen))) * torch.exp(-gt / 3e5)).float()
    es = _logbins(1e-9, 1e-3, case["ns"])
    et = torch.from_numpy(es).to(DEV).double()
    if case["delta"]:  # photons of a narrow line
        fs = torch.exp(-0.5 * ((et.log() - math.log(1e-6 * (1.0 + float(_rand(1, gen))))) / 0.3) ** 2)
        fs = torch.where(fs > 1e-6, fs, torch.zeros_like(fs))
    else:
        fs = et ** -1.0 * (0.5 + _rand(case["ns"], gen))
    return g, f.contiguous(), es, fs.float().contiguous(), _logbins(1e-3, 1e6, case["ne"])


# ---------------------------------------------------------------------------------------
# states and passes
# ---------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _modules():
    import ragnar_gb300 as rg
    from ragnar_gb300 import capi
    from ragnar_gb300 import torch_ext as rt

    rg.Initialize()
    rg.SetVerbose(False)
    return rg, capi, rt


def _rg_bins(rg, a, log=True, unit=None):
    b = rg.Bins(a, unit if unit is not None else rg.EnergyUnits.mec2)
    b.log_spaced = log
    return b


def _rg_dist(rg, bins, f):
    return rg.TabulatedDistribution(bins, rg.Array1D_f(f.cpu().numpy()))


def _target(case, seed):
    """Spectra to fit, by plain torch: particles of another index and cutoff (a sample
    scaled to the case's count), or other distributions."""
    if case["kind"] == "gradient":
        m = min(case["n"], 1 << 17)
        u, b, _, _ = _particles(case, seed + 7919, n=m, index=-2.5, gcut=300.0)
        S = _spectrum64(_species_bins(case), u, b, None, None, 1.0, _aligned_table(case["nbins"], case["umax"] <= 200.0))
        return (S * (case["n"] / m)).float()
    g, f = _distributions(case, seed + 7919)
    return _fromdist64(g, f, _dist_bins(case), _smooth_table()).float()


def _cotangent(case, seed):
    """dL/dS of a relative misfit to the target, with the sign of the misfit at random."""
    St = _target(case, seed)
    r = 2.0 * _rand(case["nbins"], _gen(seed + 2)).float() - 1.0
    return r / torch.clamp(St, min=1e-6 * float(St.max())) / case["nbins"]


def prepare(case, seed):
    rg, capi, rt = _modules()
    k = case["kind"]
    if k in ("species", "histogram"):
        if k == "species":
            u, b, _, w = _particles(case, seed)
        else:
            gen = _gen(seed)
            u, b, w = _isotropic(_powerlaw(case["n"], gen, -2.2, 1.0, 1e4, 3e3), gen), None, None
        arrays = {"U%d" % (d + 1): u[d].cpu().numpy() for d in range(3)}
        if b is not None:
            arrays.update({"B%d" % (d + 1): b[d].cpu().numpy() for d in range(3)
                           if case.get("b") != "z" or d == 2})
        if w is not None:
            arrays["W"] = w.cpu().numpy()
        p = rg.Particles_3D("e-")
        p.fromArrays(arrays)
        hist = _rg_bins(rg, _hist_bins(case), log=case.get("log", True))
        if k == "histogram":
            return {"rg": rg, "k": k, "p": p, "hist": hist, "fourvel": case["fourvel"]}
        return {"rg": rg, "k": k, "p": p, "hist": hist, "bins": _rg_bins(rg, _species_bins(case))}
    if k == "dump":
        c, n = _dump_particles(case, seed), case["n"]
        bins = _logbins(1e-4, 1e9, case["nbins"])
        pairs = capi.particles([x[:2 * n] for x in c[0:3]], b=[x[:2 * n] for x in c[3:6]], w=c[6][:2 * n], n=2 * n)
        prot = capi.particles([x[2 * n:] for x in c[0:3]], b=[x[2 * n:] for x in c[3:6]], w=c[6][2 * n:], n=n)
        plan_e = capi.SpectrumPlan(bins, 1.0, 1.0, SPECIES_EPS[0])
        plan_e.reserve(2)
        return {"k": k, "c": c, "pairs": pairs, "prot": prot, "plan_e": plan_e,
                "plan_p": capi.SpectrumPlan(bins, 1.0, 1.0, SPECIES_EPS[2]),
                "offs": torch.tensor([0, n, 2 * n], device=DEV, dtype=torch.int64),
                "out": torch.empty((3, case["nbins"]), device=DEV)}
    if k == "fields":
        u, b, e, w = _particles(case, seed)
        plan = rt.spectrum_plan(_species_bins(case), 1.0, 1.0, 1.0, smooth=False)
        return {"rt": rt, "k": k, "plan": plan, "args": [w] + u + b + e}
    if k == "segments":
        offs, u, bz = _segment_inputs(case, seed)
        plan = capi.SpectrumPlan(_logbins(1e-2, 1e7, case["nbins"]), 1.0, 1.0, 1.0)
        plan.reserve(case["nseg"])
        return {"k": k, "plan": plan, "p": capi.particles(u, b=[None, None, bz], n=int(offs[-1])), "nseg": case["nseg"],
                "offs": torch.from_numpy(offs).to(DEV), "out": torch.empty((case["nseg"], case["nbins"]), device=DEV)}
    if k == "gradient":
        u, b, _, _ = _particles(case, seed)
        w = (_rand(case["n"], _gen(int(seed) + 1)) + 0.5).float()
        return {"rt": rt, "k": k, "plan": rt.spectrum_plan(_species_bins(case)), "b": b, "log_loss": case["log_loss"],
                "target": _target(case, int(seed)) if case["log_loss"] else _cotangent(case, int(seed)),
                "leaves": [t.requires_grad_(True) for t in [w] + u]}
    if k in ("fromdist", "fit"):
        g, f = _distributions(case, seed)
        plan = rt.fromdist_plan(g, _dist_bins(case), max_dist=case["ndist"])
        s = {"rt": rt, "k": k, "plan": plan, "f": f}
        if k == "fit":
            s["target"] = _target(case, int(seed))
            f.requires_grad_(True)
        return s
    if k == "onedist":
        g, f = _distributions(case, seed)
        return {"rg": rg, "k": k, "dist": _rg_dist(rg, _rg_bins(rg, g, unit=""), f[0]), "bins": _rg_bins(rg, _dist_bins(case))}
    g, f, es, fs, eic = _ic_inputs(case, seed)
    return {"rg": rg, "k": k, "dist": _rg_dist(rg, _rg_bins(rg, g, unit=""), f), "soft": _rg_dist(rg, _rg_bins(rg, es), fs),
            "bins": _rg_bins(rg, eic)}


def run(s):
    k = s["k"]
    if k == "species":
        rg = s["rg"]
        return {"spectrum": rg.SynchrotronSpectrum_3D(s["p"], s["bins"], 1.0, 1.0, 1.0).as_array(),
                "hist": s["p"].energyDistribution(s["hist"]).F().as_array()}
    if k == "dump":
        stream = torch.cuda.current_stream().cuda_stream
        s["plan_e"].run_batched(s["pairs"], s["offs"], 2, s["out"], stream)
        s["plan_p"].run(s["prot"], s["out"][2], stream)
        return s["out"]
    if k == "fields":
        with torch.no_grad():
            return s["rt"].synchrotron_spectrum(s["plan"], *s["args"])
    if k == "segments":
        s["plan"].run_batched(s["p"], s["offs"], s["nseg"], s["out"], torch.cuda.current_stream().cuda_stream)
        return s["out"]
    if k == "gradient":
        rt = s["rt"]
        S = rt.synchrotron_spectrum(s["plan"], *s["leaves"], *s["b"])
        if not s["log_loss"]:
            gw, gx, gy, gz = torch.autograd.grad(S, s["leaves"], s["target"])
            return {"spectrum": S.detach(), "gw": gw, "gux": gx, "guy": gy, "guz": gz}
        loss = rt.log_mse(S, s["target"])
        gw, gx, gy, gz = torch.autograd.grad(loss, s["leaves"])
        return {"spectrum": S.detach(), "loss": loss.detach(), "gw": gw, "gux": gx, "guy": gy, "guz": gz}
    if k == "fromdist":
        with torch.no_grad():
            return s["rt"].synchrotron_from_dist_batched(s["plan"], s["f"])
    if k == "fit":
        rt = s["rt"]
        S = rt.synchrotron_from_dist_batched(s["plan"], s["f"])
        loss = rt.log_mse(S, s["target"])
        (gf,) = torch.autograd.grad(loss, (s["f"],))
        return {"spectra": S.detach(), "loss": loss.detach(), "gf": gf}
    if k == "onedist":
        return s["rg"].SynchrotronSpectrumFromDist(s["dist"], s["bins"], 1.0, 1.0).as_array()
    if k == "histogram":
        return s["p"].energyDistribution(s["hist"], s["fourvel"]).F().as_array()
    return s["rg"].ICSpectrum(s["dist"], s["soft"], s["bins"]).as_array()


# ---------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------

KINEMATICS = 60  # operations of one particle: gamma, |gamma E + u x B|, its logarithm, its deposit


def work(case):
    """Inputs read once, outputs written once; the operations of the particle stage, the
    product or the (gamma, photon, photon) sum."""
    k = case["kind"]
    if k == "species":
        streams = 3 + (1 if case["b"] == "z" else 3) + int(case["weights"])
        return {"bytes": 4 * (streams + 3) * case["n"] + 4 * (case["nbins"] + case["nhist"]),
                "flops": (KINEMATICS + 10) * case["n"]}
    if k == "dump":
        return {"bytes": 4 * 7 * 3 * case["n"] + 12 * case["nbins"], "flops": KINEMATICS * 3 * case["n"]}
    if k == "fields":
        return {"bytes": 4 * (9 + int(case["weights"])) * case["n"] + 4 * case["nbins"], "flops": 90 * case["n"]}
    if k == "segments":
        n = case["nseg"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": 16.0 * n + 4 * case["nseg"] * case["nbins"], "flops": KINEMATICS * n}
    if k == "gradient":  # forward reads u, B, w; the backward reads them again and writes four gradients
        return {"bytes": 4 * (7 + 7 + 4) * case["n"], "flops": 2 * KINEMATICS * case["n"]}
    if k in ("fromdist", "fit"):
        d, g, e = case["ndist"], case["ng"], case["nbins"]
        b, f = 4.0 * (d * g + g * e + d * e), 2.0 * d * g * e
        return {"bytes": 2 * b, "flops": 2 * f} if k == "fit" else {"bytes": b, "flops": f}
    if k == "onedist":
        return {"bytes": 8 * case["ng"] + 8 * case["nbins"], "flops": 6.0 * case["ng"] * case["nbins"]}
    if k == "histogram":
        return {"bytes": 12 * case["n"] + 4 * case["nhist"], "flops": 10 * case["n"]}
    return {"bytes": 8 * (case["ng"] + case["ns"] + case["ne"]), "flops": 10.0 * case["ng"] * case["ns"] * case["ne"]}


# ---------------------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------------------

def _cosh_quad(x, p):
    """int_0^inf exp(-x cosh s) cosh(5 s / 3) / cosh(s)^p ds by the trapezoidal rule."""
    h = torch.clamp(0.5 / torch.sqrt(x), max=0.125)
    t = torch.zeros_like(x)
    for k in range(0, 400):
        s = k * h
        sh = torch.sinh(0.5 * s)
        v = torch.exp(-2.0 * x * sh * sh + 5.0 * s / 3.0) * 0.5 * (1.0 + torch.exp(-10.0 * s / 3.0))
        if p:
            v = v / torch.cosh(s)
        t = t + (0.5 * v if k == 0 else v)
    return torch.exp(-x) * t * h


def _logspace32(a, b, n):
    """The reference's grid: a float exponent, then a double power, rounded to float."""
    f = np.float32
    la, lr = f(math.log10(f(a))), f(math.log10(f(f(b) / f(a))))
    return np.array([f(10.0 ** float(f(la + f(f(i) * lr) / f(n - 1)))) for i in range(n)], np.float32)


@functools.lru_cache(maxsize=None)
def _reference_table():
    """(ln x0, dln, c0, c1): the 200-node table's segments, linear in log x, from float
    nodes and float values (a 100-point trapezoid of K_{5/3} in float steps)."""
    n = 200
    xs = _logspace32(1e-6, 100.0, n)
    grids = np.ones((n, 100), np.float32)
    for i, x in enumerate(xs):
        if 1e-5 <= float(x) and not x > 20.0:
            grids[i] = _logspace32(x, 20.0, 100)
    K = _cosh_quad(torch.from_numpy(grids.reshape(-1)).to(DEV).double(), 0).cpu().numpy().astype(np.float32)
    K = K.reshape(n, 100)
    ys = np.zeros(n, np.float32)
    for i, x in enumerate(xs):
        if float(x) < 1e-6 or x > 20.0:
            continue
        if float(x) < 1e-5:
            ys[i] = 4.0 * math.pi / (math.sqrt(3.0) * math.gamma(1.0 / 3.0)) * (0.5 * float(x)) ** (1.0 / 3.0)
            continue
        t = np.float32(0.0)
        for j in range(99):
            d = 0.5 * float(np.float32(K[i, j] + K[i, j + 1])) * float(np.float32(grids[i, j + 1] - grids[i, j]))
            t = np.float32(float(t) + d)
        ys[i] = np.float32(x * t)
    ln0 = math.log(float(xs[0]))
    dln = math.log(float(xs[-1]) / float(xs[0])) / (n - 1)
    x64, y64 = xs.astype(np.float64), ys.astype(np.float64)
    beta = (y64[1:] - y64[:-1]) / np.log(x64[1:] / x64[:-1])
    c0 = y64[:-1] + beta * (ln0 + np.arange(n - 1) * dln - np.log(x64[:-1]))
    t = torch.tensor(np.stack([c0, beta * dln]), device=DEV)
    return ln0, dln, t[0].contiguous(), t[1].contiguous()


def _hermite(ln0, dln, nseg):
    """(ln x0, dln, four coefficients): exact F at the nodes, slopes F - x^2 K_{5/3}."""
    x = torch.exp(ln0 + dln * torch.arange(nseg + 1, device=DEV, dtype=torch.float64))
    F = x * _cosh_quad(x, 1)
    D = F - x * x * _cosh_quad(x, 0)
    F0, F1, D0, D1 = F[:-1], F[1:], D[:-1], D[1:]
    return ln0, dln, F0.contiguous(), (D0 * dln).contiguous(), 3.0 * (F1 - F0) - dln * (2.0 * D0 + D1), \
        2.0 * (F0 - F1) + dln * (D0 + D1)


@functools.lru_cache(maxsize=None)
def _smooth_table():
    return _hermite(math.log(1e-6), math.log(1e8) / 2048, 2048)


@functools.lru_cache(maxsize=64)
def _aligned_table(nbins, narrow):
    """The smooth table of a plan over log-uniform bins: nodes on the bins' grid, a whole
    number of segments between bins, covering [1e-6, 100] (K0 = 1 here)."""
    le = np.log(_logbins(1e-2, 1e7 if narrow else 1e9, nbins).astype(np.float64))
    step = (le[-1] - le[0]) / (nbins - 1)
    dln = step / math.ceil(step / 0.0089954)
    ln0 = le[0] - math.ceil((le[0] - math.log(1e-6)) / dln) * dln
    return _hermite(ln0, dln, int(math.ceil((math.log(100.0) - ln0) / dln)))


def _evaluate(table, t, derivative=False):
    """F (and dF / dln x) at table coordinates t; zero outside the table."""
    c = table[2:]
    inside = (t >= 0) & (t < c[0].numel())
    s = torch.where(inside, t, torch.zeros_like(t))
    j = s.to(torch.int32).long()
    tau = s - j
    F = c[-1][j]
    for k in range(len(c) - 2, -1, -1):
        F = F * tau + c[k][j]
    F = F * inside
    if not derivative:
        return F
    return F, (c[1][j] + tau * (2.0 * c[2][j] + 3.0 * tau * c[3][j])) * inside / table[1]


def _kinematics64(u, b, e):
    """ln e_peak (K0 = 1) and chi_R (B0 = 1)."""
    x, y, z = (t.double() for t in u)
    bx, by, bz = (t.double() for t in b)
    G = 1.0 + x * x + y * y + z * z
    vx, vy, vz = y * bz - z * by, z * bx - x * bz, x * by - y * bx
    if e is None:
        W = vx * vx + vy * vy + vz * vz
    else:
        ex, ey, ez = (t.double() for t in e)
        g = torch.sqrt(G)
        vx, vy, vz = vx + g * ex, vy + g * ey, vz + g * ez
        W = vx * vx + vy * vy + vz * vz - (x * ex + y * ey + z * ez) ** 2
    live = W > 0
    W = torch.where(live, W, torch.ones_like(W))
    return 0.5 * (torch.log(G) + torch.log(W)), torch.sqrt(W / G) * live


def _chunks(n, nbins):
    m = max(1, (1 << 26) // max(nbins, 1))
    return [(a, min(n, a + m)) for a in range(0, n, m)]


def _spectrum64(bins, u, b, e, w, eps, table):
    le = torch.log(torch.from_numpy(bins).to(DEV).double())
    S = torch.zeros(len(bins), device=DEV, dtype=torch.float64)
    for i, j in _chunks(u[0].numel(), len(bins)):
        lp, A = _kinematics64([t[i:j] for t in u], [t[i:j] for t in b], None if e is None else [t[i:j] for t in e])
        if w is not None:
            A = A * w[i:j].double()
        t = (le[None, :] - (lp + math.log(eps))[:, None] - table[0]) / table[1]
        S += torch.mv(_evaluate(table, t).T, A)
    return S * torch.exp(le)


def _fromdist64(g, f, bins, table):
    le = torch.log(torch.from_numpy(bins).to(DEV).double())
    gt = torch.from_numpy(g).to(DEV).double()
    K = _evaluate(table, (le[:, None] - 2.0 * torch.log(gt)[None, :] - table[0]) / table[1]) * gt[None, :]
    K = K * torch.exp(le)[:, None]
    return f.double() @ K.T


def _log_mse64(S, St):
    """The loss and its derivative with respect to S."""
    m = (S > 1e-12 * S.max()) & (St > 1e-12 * St.max())
    d = torch.where(m, torch.log(torch.where(m, S, torch.ones_like(S)) / torch.where(m, St, torch.ones_like(St))),
                    torch.zeros_like(S))
    c = m.sum().clamp(min=1)
    return (d * d).sum() / c, 2.0 * d / torch.where(m, S, torch.ones_like(S)) / c


def _hist_bins(case):
    if not case.get("log", True):
        return np.linspace(1.0, 1e3, case["nhist"]).astype(np.float32)
    return _logbins(1e-2, 1e3, case["nhist"])


def _histogram64(case, u):
    bins = _hist_bins(case)
    n = len(bins)
    lo, hi = float(bins.min()), float(bins.max())
    S = (u[0] * u[0] + u[1] * u[1]) + u[2] * u[2]
    E = torch.sqrt(S).double() if case.get("fourvel", True) else torch.sqrt(1.0 + S.double())
    i = (float(np.float32(n - 1)) * torch.log10(E / lo).abs() / float(np.log10(np.float32(np.float32(hi) / np.float32(lo))))).long()
    i = torch.where(E < lo, torch.zeros_like(i), torch.where(E >= hi, torch.full_like(i, n - 1), i.clamp(max=n - 1)))
    return torch.bincount(i, weights=(1.0 / E) if case.get("log", True) else None, minlength=n).double()


def _gradient64(case, seed):
    u, b, _, _ = _particles(case, seed)
    w = (_rand(case["n"], _gen(int(seed) + 1)) + 0.5).float()
    bins = _species_bins(case)
    table = _aligned_table(case["nbins"], case["umax"] <= 200.0)
    S = _spectrum64(bins, u, b, None, w, 1.0, table)
    loss = None
    if case["log_loss"]:
        loss, G = _log_mse64(S, _target(case, int(seed)).double())
    else:
        G = _cotangent(case, int(seed)).double()
    le = torch.log(torch.from_numpy(bins).to(DEV).double())
    Ge = G * torch.exp(le)
    out = [torch.empty(case["n"], device=DEV, dtype=torch.float64) for _ in range(4)]
    for i, j in _chunks(case["n"], 2 * len(bins)):
        uc = [t[i:j].double().requires_grad_(True) for t in u]
        lp, chi = _kinematics64(uc, [t[i:j] for t in b], None)
        F, D = _evaluate(table, (le[None, :] - lp.detach()[:, None] - table[0]) / table[1], True)
        R1, R2 = torch.mv(F, Ge), torch.mv(D, Ge)
        A = w[i:j].double()
        out[0][i:j] = chi.detach() * R1
        # dL/du = w (R1 dchi/du - chi R2 dln e_peak/du)
        s = (A * R1 * chi).sum() - ((A * chi * R2).detach() * lp).sum()
        for d, gd in enumerate(torch.autograd.grad(s, uc)):
            out[1 + d][i:j] = gd
    r = {"spectrum": S, "gw": out[0], "gux": out[1], "guy": out[2], "guz": out[3]}
    return r if loss is None else dict(r, loss=loss)


def _ic64(case, seed):
    g, f, es, fs, eic = _ic_inputs(case, seed)
    to = lambda a: torch.from_numpy(a).to(DEV).double()  # noqa: E731
    gt, st, et = to(g), to(es), to(eic)
    out = torch.zeros(len(eic), device=DEV, dtype=torch.float64)
    ws = fs.double() / st
    for i in range(0, len(g), 32):
        G = gt[i:i + 32][:, None, None]
        Gam = 4.0 * G * st[None, :, None]
        d = G - et[None, None, :]
        ok = d > 0
        t = et[None, None, :] / torch.where(ok, d, torch.ones_like(d))  # Gamma q
        q = t / Gam
        ok = ok & (et[None, None, :] <= G * Gam / (1.0 + Gam))
        kn = 2.0 * q * torch.log(q) + (1.0 - q) * (1.0 + 2.0 * q + t * t / (2.0 * (1.0 + t)))
        kn = torch.where(ok, kn, torch.zeros_like(kn))
        out += torch.einsum("gse,s,g->e", kn, ws, f[i:i + 32].double() / gt[i:i + 32])
    return out * et * et


def exact(case, seed):
    k = case["kind"]
    if k == "species":
        u, b, _, w = _particles(case, seed)
        return {"spectrum": _spectrum64(_species_bins(case), u, b, None, w, 1.0, _reference_table()),
                "hist": _histogram64(case, u)}
    if k == "dump":
        c, n = _dump_particles(case, seed), case["n"]
        bins = _logbins(1e-4, 1e9, case["nbins"])
        return torch.stack([_spectrum64(bins, [x[s * n:(s + 1) * n] for x in c[0:3]], [x[s * n:(s + 1) * n] for x in c[3:6]],
                                        None, c[6][s * n:(s + 1) * n], SPECIES_EPS[s], _reference_table()) for s in range(3)])
    if k == "fields":
        u, b, e, w = _particles(case, seed)
        return _spectrum64(_species_bins(case), u, b, e, w, 1.0, _reference_table())
    if k == "segments":
        offs, u, bz = _segment_inputs(case, seed)
        bins = _logbins(1e-2, 1e7, case["nbins"])
        zero = torch.zeros_like(bz)
        return torch.stack([_spectrum64(bins, [t[a:z] for t in u], [zero[a:z], zero[a:z], bz[a:z]], None, None, 1.0,
                                        _reference_table()) for a, z in zip(offs[:-1].tolist(), offs[1:].tolist())])
    if k == "gradient":
        return _gradient64(case, seed)
    if k == "fromdist":
        g, f = _distributions(case, seed)
        return _fromdist64(g, f, _dist_bins(case), _smooth_table())
    if k == "fit":
        g, f = _distributions(case, seed)
        f64 = f.double().requires_grad_(True)
        S = _fromdist64(g, f64, _dist_bins(case), _smooth_table())
        loss, G = _log_mse64(S.detach(), _target(case, int(seed)).double())
        (gf,) = torch.autograd.grad(S, (f64,), G)
        return {"spectra": S.detach(), "loss": loss, "gf": gf}
    if k == "onedist":
        g, f = _distributions(case, seed)
        return _fromdist64(g, f, _dist_bins(case), _reference_table())[0]
    if k == "histogram":
        gen = _gen(seed)
        return _histogram64(case, _isotropic(_powerlaw(case["n"], gen, -2.2, 1.0, 1e4, 3e3), gen))
    return _ic64(case, seed)
