"""The interval-moment spectrum (moments.cu) against the fused kernel and the oracle.

Both sum the reference's sync::Kernel (synchrotron.hpp:145-172) over particles
and bins with the same fixed-point table coordinate; interval moments sum the
piecewise-linear F exactly in FP64 per (table cell, bin interval) instead of
evaluating every (particle, bin) pair in FP32.  Checked here: which plans and
runs take the path, agreement with the fused kernel and the FP64 oracle on
bin sets whose low parts tie or crowd one bucket, 256 uneven segments with
empty ones, and the fallback above 1024 segments.
"""

from __future__ import annotations

import numpy as np
import pytest

from helpers import SPECTRUM_RTOL, max_rel, particles

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
capi = pytest.importorskip("ragnar_gb300.capi")


def _device(P, dev):
    T = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in P.items()}
    prt = capi.particles([T["ux"], T["uy"], T["uz"]], b=[T["bx"], T["by"], T["bz"]],
                         e=[T["ex"], T["ey"], T["ez"]] if "ex" in T else None, w=T.get("w"), n=len(P["ux"]))
    return T, prt


@pytest.fixture(scope="module")
def table(oracle_lib):
    return oracle_lib.tabulate_ffunc()


def test_algorithm_selection(gpu, oracle_lib):
    bins = oracle_lib.logspace(0.01, 1e7, 200)
    ref = capi.SpectrumPlan(bins, 1.0, 1.0, 1.0)
    assert ref.algorithm(1) == capi.RG_ALGO_MOMENTS
    assert ref.algorithm(1024) == capi.RG_ALGO_MOMENTS
    assert ref.algorithm(1025) == capi.RG_ALGO_DIRECT  # more segments than the deposit stages
    ref.set_algorithm(capi.RG_ALGO_DIRECT)
    assert ref.algorithm(1) == capi.RG_ALGO_DIRECT
    with pytest.raises(capi.RgError):
        ref.set_algorithm(7)
    # smooth table: moments over log-uniform bins (the plan's bin-aligned table) only
    assert capi.SpectrumPlan(bins, 1.0, 1.0, 1.0, capi.RG_TABLE_SMOOTH).algorithm(1) == capi.RG_ALGO_MOMENTS
    uneven = np.sort(np.concatenate([bins[:100], bins[100:] * 1.01])).astype(np.float32)
    smooth = capi.SpectrumPlan(uneven, 1.0, 1.0, 1.0, capi.RG_TABLE_SMOOTH)
    assert smooth.algorithm(1) == capi.RG_ALGO_DIRECT
    smooth.set_algorithm(capi.RG_ALGO_MOMENTS)
    P = particles(100, seed=1)
    T, prt = _device(P, gpu)
    out = torch.empty(200, device=gpu)
    with pytest.raises(capi.RgError) as e:
        smooth.run(prt, out)
    assert e.value.status == capi.RG_ERR_UNSUPPORTED


@pytest.mark.parametrize("kind", ["log512", "ties", "one_bucket", "linear", "sparse"])
def test_moments_vs_fused_and_oracle(gpu, oracle_lib, table, kind):
    P = particles(40000, seed=["log512", "ties", "one_bucket", "linear", "sparse"].index(kind) + 70, bfield="iso", weights=True, efield=kind == "linear",
                  umax=1e4, index=-2.2)
    if kind == "log512":
        bins = oracle_lib.logspace(1e-4, 1e9, 512)
    elif kind == "ties":  # repeated bins: equal low parts
        bins = np.repeat(oracle_lib.logspace(1e-2, 1e6, 50), 4).astype(np.float32)
    elif kind == "one_bucket":  # bins a whole number of table segments apart: low parts crowd one bucket
        xs, _ = table
        r = float(xs[1]) / float(xs[0])
        bins = (0.5 * r ** np.arange(0, 300, 3)).astype(np.float32)
    elif kind == "linear":
        bins = oracle_lib.linspace(-10.0, 5000.0, 333)
    else:  # few bins far apart, some outside every particle's reach
        bins = np.array([1e-12, 1e-3, 7.0, 3e4, 2e9, 1e15], np.float32)
    T, prt = _device(P, gpu)
    res = {}
    for algo in (capi.RG_ALGO_DIRECT, capi.RG_ALGO_MOMENTS):
        plan = capi.SpectrumPlan(bins, 1.0, 1.0, 1.0)
        plan.set_algorithm(algo)
        out = torch.full((len(bins),), -1.0, device=gpu)
        plan.run(prt, out)
        plan.check()
        res[algo] = out.cpu().numpy()
        plan.close()
    truth = oracle_lib.sync_spectrum_f64(P, bins, 1.0, 1.0, 1.0, table)
    got = res[capi.RG_ALGO_MOMENTS]
    assert max_rel(got, truth) <= SPECTRUM_RTOL
    assert np.array_equal(got == 0, truth == 0)
    assert max_rel(got, res[capi.RG_ALGO_DIRECT]) <= SPECTRUM_RTOL


def test_moments_256_uneven_segments(gpu, oracle_lib, table):
    rng = np.random.default_rng(256)
    counts = np.floor(10.0 ** rng.uniform(0.0, 3.5, 256)).astype(np.int64)
    counts[[3, 100, 101, 255]] = 0
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    n = int(offs[-1])
    P = particles(n, seed=257, bfield="iso", weights=True)
    bins = oracle_lib.logspace(0.01, 1e7, 200)
    T, prt = _device(P, gpu)
    plan = capi.SpectrumPlan(bins, 1.0, 1.0, 1.0)
    plan.reserve(256)
    assert plan.algorithm(256) == capi.RG_ALGO_MOMENTS
    out = torch.empty((256, 200), device=gpu)
    plan.run_batched(prt, torch.from_numpy(offs).to(gpu), 256, out)
    plan.check()
    got = out.cpu().numpy()
    truth = oracle_lib.sync_spectrum_batched_f64(P, offs, bins, 1.0, 1.0, 1.0, table)
    for s in range(256):
        if counts[s] == 0:
            assert np.all(got[s] == 0)
        else:
            assert max_rel(got[s], truth[s]) <= SPECTRUM_RTOL, s


def test_more_segments_than_staged_fall_back_to_fused(gpu, oracle_lib, table):
    nseg = 1100
    offs = np.arange(0, 5 * nseg + 1, 5, dtype=np.int64)
    P = particles(int(offs[-1]), seed=1100, bfield="iso")
    bins = oracle_lib.logspace(0.01, 1e7, 64)
    T, prt = _device(P, gpu)
    plan = capi.SpectrumPlan(bins, 1.0, 1.0, 1.0)
    plan.reserve(nseg)
    assert plan.algorithm(nseg) == capi.RG_ALGO_DIRECT
    out = torch.empty((nseg, 64), device=gpu)
    plan.run_batched(prt, torch.from_numpy(offs).to(gpu), nseg, out)
    plan.check()
    truth = oracle_lib.sync_spectrum_batched_f64(P, offs, bins, 1.0, 1.0, 1.0, table)
    got = out.cpu().numpy()
    for s in (0, 1, 517, nseg - 1):
        assert max_rel(got[s], truth[s]) <= SPECTRUM_RTOL


@pytest.mark.parametrize("B0,eps,negw", [(1.0, 1.0, True), (-2.0, -1.5, False)])
def test_negative_amplitudes(gpu, oracle_lib, table, B0, eps, negw):
    """Negative weights, or B0 and e_syn_at_g_syn both negative (K0 > 0, amplitude
    1/B0 < 0): every particle still adds its (signed) term, as in the reference's sum."""
    P = particles(30000, seed=88, bfield="iso", weights=True)
    if negw:
        P["w"][::3] *= -1.0
    bins = oracle_lib.logspace(0.01, 1e7, 200)
    T, prt = _device(P, gpu)
    res = {}
    for algo in (capi.RG_ALGO_DIRECT, capi.RG_ALGO_MOMENTS):
        plan = capi.SpectrumPlan(bins, B0, 1.0, eps)
        plan.set_algorithm(algo)
        out = torch.empty(200, device=gpu)
        plan.run(prt, out)
        plan.check()
        res[algo] = out.cpu().numpy().astype(np.float64)
    truth = oracle_lib.sync_spectrum_f64(P, bins, B0, 1.0, eps, table)
    scale = np.abs(truth).max()
    for algo, got in res.items():
        # signed sums can cancel: compare against the largest magnitude
        assert np.max(np.abs(got - truth)) <= SPECTRUM_RTOL * scale, algo


@pytest.mark.parametrize("n,nbins", [(1, 1), (255, 31), (257, 32), (512, 63), (513, 200), (1023, 512), (1025, 513),
                                     (3001, 700)])
@pytest.mark.parametrize("wscale", [1.0, 1e-33, 1e31])
def test_moments_edges_of_steps_and_rows(gpu, oracle_lib, table, n, nbins, wscale):
    """Particle counts around the deposit's 512-particle steps, bin counts around the finish's
    32-entry lanes and 512-bin slices, streams that start off a 16-byte boundary, and weights
    near both ends of the float range, against FP64."""
    P = particles(n + 1, seed=n + nbins, bfield="iso", weights=True, umax=1e3)
    P = {k: v[1:] for k, v in P.items()}
    P["w"] = (P["w"] * np.float32(wscale)).astype(np.float32)
    bins = oracle_lib.logspace(1e-2, 1e6, nbins) if nbins > 1 else np.array([3.0], np.float32)
    full = {k: torch.zeros(n + 1, device=gpu) for k in P}
    for k, v in P.items():
        full[k][1:] = torch.from_numpy(np.ascontiguousarray(v)).to(gpu)
    T = {k: v[1:] for k, v in full.items()}
    prt = capi.particles([T["ux"], T["uy"], T["uz"]], b=[T["bx"], T["by"], T["bz"]], w=T["w"], n=n)
    plan = capi.SpectrumPlan(bins, 1.0, 1.0, 1.0)
    out = torch.full((nbins,), -1.0, device=gpu)
    for _ in range(2):  # the tables are clear again after a run
        plan.run(prt, out)
    plan.check()
    truth = oracle_lib.sync_spectrum_f64(P, bins, 1.0, 1.0, 1.0, table)
    assert max_rel(out.cpu().numpy(), truth) <= SPECTRUM_RTOL


@pytest.mark.parametrize("mode", ["reference", "smooth"])
@pytest.mark.parametrize("efield", [False, True])
@pytest.mark.parametrize("tilt", [2.0**-8, 2.0**-20])
def test_moments_nearly_cancelling_force(gpu, oracle_lib, table, mode, efield, tilt):
    """Fields almost parallel to the momentum, or an electric field that almost cancels u x B: the
    force is the small difference of products, whose remainders decide it (a sum that took an
    unrounded product instead would be off by the product's whole rounding error)."""
    n   = 4001
    P   = particles(n, seed=5, bfield="iso", weights=True, umax=1e3)
    rng = np.random.default_rng(6)
    u   = np.stack([P[k] for k in ("ux", "uy", "uz")]).astype(np.float64)
    b   = np.stack([P[k] for k in ("bx", "by", "bz")]).astype(np.float64)
    off = 1.0 + tilt * rng.uniform(-1.0, 1.0, (3, n))
    if efield:
        e = -np.cross(u.T, b.T).T / np.sqrt(1.0 + np.sum(u * u, axis=0)) * off
        P.update({k: e[d].astype(np.float32) for d, k in enumerate(("ex", "ey", "ez"))})
    else:
        b = u / np.sqrt(np.sum(u * u, axis=0)) * off
        P.update({k: b[d].astype(np.float32) for d, k in enumerate(("bx", "by", "bz"))})
    bins = oracle_lib.logspace(1e-8, 1e6, 300)
    T, prt = _device(P, gpu)
    out = torch.full((300,), -1.0, device=gpu)
    plan = capi.SpectrumPlan(bins, 1.0, 1.0, 1.0,
                             capi.RG_TABLE_SMOOTH if mode == "smooth" else capi.RG_TABLE_REFERENCE)
    plan.run(prt, out)
    plan.check()
    if mode == "reference":
        truth = oracle_lib.sync_spectrum_f64(P, bins, 1.0, 1.0, 1.0, table)
    else:
        coef, lnx, dln = plan.smooth_table()
        xmin, xmax = float(np.exp(lnx)), float(np.exp(lnx + coef.shape[0] * dln))
        truth = oracle_lib.sync_smooth_f64(P, bins, 1.0, 1.0, 1.0, coef, xmin, xmax)
    assert max_rel(out.cpu().numpy(), truth) <= SPECTRUM_RTOL


@pytest.mark.parametrize("mode", ["reference", "smooth"])
@pytest.mark.parametrize("nseg,spread", [(1, "near"), (1, "far"), (300, "near"), (300, "far")])
def test_moments_of_very_unequal_weights(gpu, oracle_lib, table, mode, nseg, spread):
    """One particle outweighs the others by 1e39, in their own cell and the next ones or over decades of
    energies; bins below the heavy one's table range see only the light ones, whose sums the FP64
    moments hold exactly whatever else their cell or its neighbours hold."""
    heavy = 1e4
    k  = np.arange(1, 61)
    ep = heavy / np.concatenate([[1.0], 1.0 + 4e-3 * k if spread == "near" else 1.2**k])
    a  = np.sqrt((np.sqrt(1.0 + 4.0 * ep * ep) - 1.0) / 2.0)  # e_peak = u sqrt(1 + u^2) for u across a unit B
    z  = np.zeros(len(a), np.float32)
    P  = {"ux": a.astype(np.float32), "uy": z, "uz": z, "bx": z, "by": z, "bz": z + np.float32(1.0),
          "w": np.concatenate([[1e30], np.resize([1e-9, 3e-9, 2e-9], 60)]).astype(np.float32)}
    bins = oracle_lib.logspace(1e-6 * ep.min() * 1.001, 1e-6 * heavy * 1.01, 24 if spread == "near" else 200)
    plan = capi.SpectrumPlan(bins, 1.0, 1.0, 1.0,
                             capi.RG_TABLE_SMOOTH if mode == "smooth" else capi.RG_TABLE_REFERENCE)
    assert plan.algorithm(nseg) == capi.RG_ALGO_MOMENTS
    xmin = 1e-6
    if mode == "reference":
        truth = oracle_lib.sync_spectrum_f64(P, bins, 1.0, 1.0, 1.0, table)
    else:
        coef, lnx, dln = plan.smooth_table()
        xmin, xmax = float(np.exp(lnx)), float(np.exp(lnx + coef.shape[0] * dln))
        truth = oracle_lib.sync_smooth_f64(P, bins, 1.0, 1.0, 1.0, coef, xmin, xmax)
    # bins next to the low end of a particle's table range count it or not by rounding
    keep = np.all(np.abs(bins[:, None].astype(np.float64) / (xmin * ep[None, :]) - 1.0) > 1e-4, axis=1)
    assert keep.sum() >= 20 and np.all(truth[keep] > 0.0) and truth[keep].max() > 1e36 * truth[keep].min()
    T, prt = _device({k: np.tile(v, nseg) for k, v in P.items()}, gpu)
    out = torch.full((nseg, len(bins)), -1.0, device=gpu)
    if nseg == 1:
        plan.run(prt, out)
    else:
        offs = torch.arange(nseg + 1, device=gpu, dtype=torch.int64) * len(a)
        plan.run_batched(prt, offs, nseg, out)
    plan.check()
    got = out.cpu().numpy().astype(np.float64)[:, keep]
    assert np.max(np.abs(got - truth[keep]) / truth[keep]) <= SPECTRUM_RTOL


@pytest.mark.parametrize("mode", ["reference", "smooth"])
def test_runs_that_overlapped_leave_nothing_behind(gpu, oracle_lib, table, mode):
    """Runs of one plan on two streams at once are outside its contract and may give wrong spectra, but
    the next ordered run is right again; so is one without particles."""
    P    = particles(200000, seed=40, bfield="iso", weights=True)
    bins = oracle_lib.logspace(1e-2, 1e7, 512)
    plan = capi.SpectrumPlan(bins, 1.0, 1.0, 1.0,
                             capi.RG_TABLE_SMOOTH if mode == "smooth" else capi.RG_TABLE_REFERENCE)
    T, prt = _device(P, gpu)
    want, out, junk = (torch.empty(512, device=gpu) for _ in range(3))
    plan.run(prt, want)
    offs = torch.tensor([0, 50000, 200000], device=gpu, dtype=torch.int64)
    two  = torch.empty((2, 512), device=gpu)
    plan.reserve(2)
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(gpu), torch.cuda.Stream(gpu)
    for _ in range(50):
        plan.run(prt, junk, a.cuda_stream)
        plan.run_batched(prt, offs, 2, two, b.cuda_stream)
    torch.cuda.synchronize()
    plan.check()
    none = capi.particles([T["ux"], T["uy"], T["uz"]], b=[T["bx"], T["by"], T["bz"]], w=T["w"], n=0)
    plan.run(none, out)
    assert torch.all(out == 0.0)
    for _ in range(2):
        plan.run(prt, out)
        plan.check()
        assert torch.allclose(out, want, rtol=1e-6, atol=0.0)
