"""Performance cases: what a user of the framework has it do, through its public entry points.

A user holds a grid of model spectra (an interpolator), a dispersion and a continuum fitter for each
observed spectrum, and calls one of: a model at given labels, chi2 at given labels, a swarm fit of one star,
a batch of fits, or the fit server.  The listed cases take each of these over the sizes of the three
workloads this repository is built for:

* ``small``: 9 x 11 x 5 models of 20,000 pixels (one star, a 40-particle swarm, 5 chunks of degree 8);
* ``survey``: 60 x 21 x 11 models of 80,000 pixels, 2.2 GB (many stars of 10k-60k pixels, 64-particle swarms,
  8 chunks of degree 5; variable resolution 60,000-90,000);
* ``factor``: 27 x 13 x 7 models of 120,000 pixels with blackbody continua and per-model maxima, 0.6 GB (a part of
  the axes of the 80 x 26 x 13 grid; 128-particle swarms, a 40-column linear continuum).

The grids are the same for every seed and are kept for the process, as a user's program keeps its
interpolator; stars, noise, labels and swarm seeds come from the seed.  Line spectra are exp(-optical depth), so
no pixel is black and chi2 is well conditioned for every label.

Swarm fits run a few iterations of the usual 100-300: a swarm's path hangs on comparisons of nearly equal costs, so
the labels of long fits differ between any two roundings.  What a long fit does most of the time, whole
contracted swarms, is covered by fits whose ranges are narrow from the start and by chi2 of contracted labels.

chi2 is returned in single precision: the models it is computed from are.
"""
import dataclasses
import math

import numpy as np
import torch

from pasta_b200 import pasta, synth

C_KMS = 299792.0
RESOLUTION = 85000.0
VSINI, RV = (0.0, 300.0), (-150.0, 150.0)


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the model of one label, as a notebook or an optimiser outside the framework asks for it (latency)
        dict(name="model one label", kind="model", grid="small", pixels=15000, labels=1, swarm="spread"),
        # models of a list of labels, returned whole (plots, training sets)
        dict(name="models 61 labels", kind="model", grid="survey", pixels=37501, labels=61, swarm="spread"),
        # one iteration of an outside sampler on one star: chi2 of a 40-particle swarm
        dict(name="chi2 small swarm", kind="chi2", grid="small", pixels=15000, labels=40, swarm="near", continuum="chunk",
             chunks=5, degree=8),
        # an early swarm or a coarse search: labels over many grid cubes
        dict(name="chi2 spread labels", kind="chi2", grid="survey", pixels=37501, labels=2500, swarm="spread",
             continuum="chunk", chunks=8, degree=5),
        # a posterior or a late swarm: many labels within a cube, the longest spectrum (the largest case)
        dict(name="chi2 contracted labels", kind="chi2", grid="survey", pixels=60000, labels=16001, swarm="contracted",
             continuum="chunk", chunks=8, degree=5),
        # wavelength-dependent resolution
        dict(name="chi2 variable resolution", kind="chi2_variable", grid="survey", pixels=23456, labels=1000, swarm="near",
             continuum="chunk", chunks=8, degree=5),
        # a design-matrix continuum on grids that carry the absolute flux
        dict(name="chi2 linear continuum", kind="chi2", grid="factor", pixels=30007, labels=2048, swarm="contracted",
             continuum="linear", columns=40),
        # two stars in one spectrum
        dict(name="chi2 binary", kind="binary", grid="small", pixels=15000, labels=160, swarm="near", continuum="chunk",
             chunks=5, degree=8),
        # one star, one swarm
        dict(name="fit one star", kind="fit", grid="small", stars=1, pixels_lo=15000, pixels_hi=15000, particles=40,
             iterations=10, swarm="spread", chunks=5, degree=8),
        # a batch of ragged spectra, swarms over the whole grid
        dict(name="fits spread swarms", kind="fit_many", grid="survey", stars=48, pixels_lo=10000, pixels_hi=60000,
             particles=64, iterations=4, swarm="spread", chunks=8, degree=5),
        # a batch of ragged spectra refined within narrow ranges
        dict(name="fits narrow ranges", kind="fit_many", grid="survey", stars=128, pixels_lo=10000, pixels_hi=60000,
             particles=64, iterations=4, swarm="contracted", chunks=8, degree=5),
        # the server: more requests than slots, each with its own continuum settings (chunks 4-12, degree 3-8)
        dict(name="served fits", kind="served", grid="survey", stars=96, slots=40, pixels_lo=10000, pixels_hi=60000,
             particles=64, iterations=4, swarm="contracted", chunks=0, degree=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "chi2", "chi2", "chi2", "chi2_variable", "linear", "binary", "fit", "fit_many", "served"])
    swarm = rng.choice(["spread", "near", "contracted"])
    grid = rng.choice(["small", "survey"])
    top = 18000 if grid == "small" else 60000
    if kind == "model":
        return dict(kind=kind, grid=grid, pixels=rng.randint(5000, top), labels=_log_int(rng, 1, 96), swarm=swarm)
    if kind == "linear":
        return dict(kind="chi2", grid="factor", pixels=rng.randint(10000, 40000), labels=_log_int(rng, 8, 3000), swarm=swarm,
                    continuum="linear", columns=rng.randint(4, 48))
    if kind in ("chi2", "chi2_variable", "binary"):
        if kind == "binary":
            grid, top = "small", 18000
        most = dict(chi2=12000, chi2_variable=1500, binary=600)[kind] if swarm != "spread" else 600
        return dict(kind=kind, grid=grid, pixels=rng.randint(5000, top), labels=_log_int(rng, 1, most), swarm=swarm,
                    continuum="chunk", chunks=rng.randint(4, 12), degree=rng.randint(3, 8))
    case = dict(kind=kind, grid=grid, stars=_log_int(rng, 2, 64), pixels_lo=min(10000, top // 2), pixels_hi=top,
                particles=rng.randint(17, 80), iterations=rng.randint(2, 4), swarm=rng.choice(["spread", "contracted"]),
                chunks=rng.randint(4, 12), degree=rng.randint(3, 8))
    if kind == "fit":
        case.update(stars=1, pixels_lo=rng.randint(5000, top))
        case.update(pixels_hi=case["pixels_lo"])
    if kind == "served":
        case.update(slots=rng.randint(2, 48), chunks=0, degree=0)
    return case


# ------------------------------------------------------------------- grids
_KEPT = {}


def _spec(grid):
    if grid == "small":
        return synth.config0_grid()
    if grid == "survey":
        return synth.config1_grid()
    s = synth.config4_grid()
    return dataclasses.replace(s, teffs=s.teffs[20:47], ms=s.ms[8:21], loggs=s.loggs[4:11])


def _kept(key, make):
    if key not in _KEPT:
        _KEPT[key] = make()
    return _KEPT[key]


class _Lines:
    """Optical depth of a line list: strengths linear in the labels, Gaussian profiles."""

    def __init__(self, spec, count=400):
        rng = np.random.default_rng([77, spec.n_px, len(spec.teffs)])
        self.wl = torch.tensor(spec.wl(), device="cuda")
        centre = torch.tensor(rng.uniform(spec.wl_lo, spec.wl_hi, count), device="cuda")[:, None]
        width = torch.tensor(rng.uniform(0.05, 0.3, count), device="cuda")[:, None]
        self.profiles = torch.exp(-0.5 * ((self.wl[None, :] - centre) / width) ** 2)
        self.at0 = rng.uniform(0.05, 0.6, count)
        self.slope = rng.uniform(-0.3, 0.3, (3, count))
        self.lo = np.array([spec.teffs.min(), spec.ms.min(), spec.loggs.min()])
        self.hi = np.array([spec.teffs.max(), spec.ms.max(), spec.loggs.max()])
        self.factor = spec.includes_factor

    def spectrum(self, tml):
        x = (np.atleast_2d(tml) - self.lo) / (self.hi - self.lo)
        depth = torch.tensor(np.clip(self.at0 + x @ self.slope, 0.0, 1.0), device="cuda")
        f = torch.exp(-(depth @ self.profiles))
        if self.factor:
            f = f * self.continuum(tml)
        return f

    def continuum(self, tml):
        """Unnormalised continua: blackbodies in units of a 5772 K one at 5000 A."""
        t = torch.tensor(np.atleast_2d(tml)[:, 0], device="cuda")[:, None]
        return (5000.0 / self.wl) ** 5 * math.expm1(synth.HC_K / (5000.0 * 5772.0)) / torch.expm1(
            synth.HC_K / (self.wl * t))


def _quantised(f):
    """uint16 spectra of rows f, scaled by their maxima when those are over 1."""
    return torch.round(f * 65535.0).to(torch.int32).cpu().numpy().astype(np.uint16)


def _arrays(grid):
    """(labels, spectra, maxima or None) of a grid, and of its continuum grid under ``grid + " continua"``."""
    def make():
        spec = _spec(grid.split()[0])
        lines, labels = _Lines(spec), synth.gridpoints(spec)
        scaled = spec.includes_factor or grid.endswith("continua")
        spectra, maxima = np.empty((len(labels), spec.n_px), np.uint16), np.ones(len(labels), np.float32)
        for a in range(0, len(labels), 512):
            part = labels[a:a + 512]
            f = lines.continuum(part) if grid.endswith("continua") else lines.spectrum(part)
            if scaled:
                mx = f.max(dim=1, keepdim=True).values.float()
                maxima[a:a + 512] = mx[:, 0].cpu().numpy()
                f = torch.clamp(f / mx, max=1.0)
            spectra[a:a + 512] = _quantised(f)
        return labels, spectra, maxima if scaled else None
    return _kept(("arrays", grid), make)


def _wl_grid(spec):
    return pasta.WlGrid(spec.log_first, spec.log_step, spec.n_px, log=True)


def _interpolator(grid):
    return _kept(("interpolator", grid), lambda: pasta.InMemInterpolator.from_arrays(
        *_arrays(grid), _wl_grid(_spec(grid.split()[0]))))


# ------------------------------------------------------- stars and labels
def _widths(spec, vsini):
    """Taps of the rotation kernel (odd) at each vsini."""
    dv = math.log(10.0) * spec.log_step
    q = 4.0 * (0.6 - 1.0) / (math.pi * 0.6)
    n = np.ceil(2.0 * np.asarray(vsini) / C_KMS / dv * math.sqrt(1.0 + q * q)).astype(np.int64) + 2
    return n + 1 - n % 2


def _gaussian(sigma, taps):
    x = torch.arange(taps, dtype=torch.float64, device="cuda") - (taps - 1) / 2
    g = torch.exp(-0.5 * (x / sigma[..., None]) ** 2)
    return g / g.sum(-1, keepdim=True)


def _odd(six_sigma):
    n = math.ceil(six_sigma)
    return n + 1 - n % 2


def _fixed_sigma(spec):
    return 1.0 / (math.log(10.0) * 2.355 * RESOLUTION * spec.log_step)


def _sigmas(case, spec, wl):
    """Gaussian sigma in Angstrom per observed pixel, R from 60,000 to 90,000."""
    return (wl / np.linspace(60000.0, 90000.0, len(wl)) / 2.355).astype(np.float32)


def _rotated(spec, rows, vsini, taps_extra=None):
    """Rows convolved with the limb-darkened rotation profile of each vsini (and one more kernel)."""
    n = spec.n_px
    nf = 1 << (n + 4096 - 1).bit_length()
    m = torch.tensor(_widths(spec, vsini), device="cuda")[:, None]
    dv = math.log(10.0) * spec.log_step
    t = torch.arange(int(m.max()), dtype=torch.float64, device="cuda")[None, :]
    vrot = torch.tensor(np.asarray(vsini, np.float64), device="cuda")[:, None] / C_KMS
    y = 1.0 - ((t * dv - (m - 1) * dv / 2.0) / vrot) ** 2
    y = torch.where((t < m) & (y > 0), y, torch.zeros_like(y))
    k = 2.0 * 0.4 * torch.sqrt(y) + math.pi * 0.3 * y
    k = k / k.sum(1, keepdim=True)
    big = torch.zeros((len(rows), nf), dtype=torch.float64, device="cuda")
    at = (torch.arange(k.shape[1], device="cuda")[None, :] - (m - 1) // 2) % nf
    big.scatter_(1, at, k)
    f = torch.fft.rfft(rows, nf) * torch.fft.rfft(big)
    if taps_extra is not None:
        h = (len(taps_extra) - 1) // 2
        one = torch.zeros(nf, dtype=torch.float64, device="cuda")
        one[:h + 1], one[nf - h:] = taps_extra[h:], taps_extra[:h]
        f = f * torch.fft.rfft(one)
    return torch.fft.irfft(f, nf)[:, :n]


def _broadened(case, spec, rows, vsini, wl):
    if case["kind"] != "chi2_variable":
        s = _fixed_sigma(spec)
        g = _gaussian(torch.tensor(s, dtype=torch.float64, device="cuda"), _odd(6.0 * s))
        return _rotated(spec, rows, vsini, g)
    # one Gaussian per synthetic pixel; sigma is interpolated from the observed pixels, and extrapolated below the first
    f = _rotated(spec, rows, vsini)
    synth_wl, sig = spec.wl(), _sigmas(case, spec, wl).astype(np.float64)
    s = np.interp(synth_wl, wl, sig)
    s = np.where(synth_wl < wl[0], sig[0] + (synth_wl - wl[0]) / (wl[1] - wl[0]) * (sig[1] - sig[0]), s)
    s = s / (math.log(10.0) * spec.log_step * synth_wl)
    taps = _odd(6.0 * s.max())
    g, h = _gaussian(torch.tensor(s, device="cuda"), taps), (taps - 1) // 2
    out = f.clone()
    out[:, h:spec.n_px - h] = torch.einsum("bnk,nk->bn", f.unfold(1, taps, 1), g[h:spec.n_px - h])
    return out


def _at_observed(spec, rows, wl, rv):
    """Linear resampling at the shifted observed pixels; the weight is that of the index rounded to single precision."""
    index = torch.tensor((np.log10(wl) - spec.log_first) / spec.log_step, device="cuda")[None, :] + torch.tensor(
        np.log10(1.0 - np.asarray(rv) / C_KMS) / spec.log_step, device="cuda")[:, None]
    j = torch.floor(index).long()
    w = (index.float() - j.float()).double()
    return (1.0 - w) * torch.gather(rows, 1, j) + w * torch.gather(rows, 1, j + 1)


_BOX = {  # half widths of the labels' box around a star: teff (relative), m, logg, vsini, rv
    "spread": (0.25, 0.5, 0.8, 60.0, 60.0), "near": (0.03, 0.1, 0.2, 20.0, 5.0),
    "contracted": (0.0015, 0.004, 0.01, 1.5, 0.4)}


def _star_label(spec, rng, vsini_hi=260.0):
    lo = np.array([spec.teffs.min(), spec.ms.min(), spec.loggs.min()])
    hi = np.array([spec.teffs.max(), spec.ms.max(), spec.loggs.max()])
    return np.concatenate([lo + (hi - lo) * rng.uniform(0.03, 0.97, 3), [rng.uniform(20.0, vsini_hi), rng.uniform(-80.0, 80.0)]])


def _labels_around(spec, star, swarm, count, rng):
    half = np.array(_BOX[swarm])
    half[0] *= star[0]
    lab = star + half * rng.uniform(-1.0, 1.0, (count, 5))
    for k, v in enumerate((spec.teffs, spec.ms, spec.loggs)):
        edge = 1e-3 * (v.max() - v.min())
        lab[:, k] = np.clip(lab[:, k], v.min() + edge, v.max() - edge)
    lab[:, 3] = np.clip(lab[:, 3], 10.0, 299.0)
    return lab


def _observed_wl(spec, n):
    lo, hi = synth.observed_window(spec, 150.0, 300.0, 60000.0)
    return np.geomspace(lo, hi, n)


def _noisy(model, rng):
    """Response and noise on a model at the observed pixels: (flux, var)."""
    n = len(model)
    x = np.linspace(-1.0, 1.0, n)
    a, b = rng.uniform(-0.2, 0.2, 2)
    signal = model * (1.0 + a * x + b * x * x)
    sigma = np.abs(signal) / rng.uniform(20.0, 200.0) + 1e-6
    return (signal + sigma * rng.standard_normal(n)).astype(np.float32), (sigma ** 2).astype(np.float32)


def _observe(case, spec, lines, label, n, rng):
    wl = _observed_wl(spec, n)
    rows = _broadened(case, spec, lines.spectrum(label[:3]), label[3:4], wl)
    return (wl,) + _noisy(_at_observed(spec, rows, wl, label[4:5])[0].cpu().numpy(), rng)


def _inputs(case, seed):
    """Everything of a case that comes from the seed, as host arrays."""
    spec, rng = _spec(case["grid"]), np.random.default_rng([seed, 5])
    lines = _Lines(spec)
    if case["kind"] == "model":
        star = _star_label(spec, rng)
        return dict(wl=_observed_wl(spec, case["pixels"]), labels=_labels_around(spec, star, case["swarm"], case["labels"], rng))
    if case["kind"] == "binary":
        a, b = _star_label(spec, rng), _star_label(spec, rng)
        ratio = rng.uniform(0.3, 1.0)
        wl = _observed_wl(spec, case["pixels"])
        n1 = _broadened(case, spec, lines.spectrum(a[:3]), a[3:4], wl)
        n2 = _broadened(case, spec, lines.spectrum(b[:3]), b[3:4], wl)
        model = _binary(spec, wl, n1, lines.continuum(a[:3]), a[4:5], n2, lines.continuum(b[:3]), b[4:5], np.array([ratio]))
        flux, var = _noisy(model[0].cpu().numpy(), rng)
        labels = np.concatenate([_labels_around(spec, a, case["swarm"], case["labels"], rng),
                                 _labels_around(spec, b, case["swarm"], case["labels"], rng),
                                 ratio * rng.uniform(0.8, 1.2, (case["labels"], 1))], axis=1)
        return dict(wl=wl, flux=flux, var=var, labels=labels)
    if case["kind"] in ("chi2", "chi2_variable"):
        star = _star_label(spec, rng)
        wl, flux, var = _observe(case, spec, lines, star, case["pixels"], rng)
        return dict(wl=wl, flux=flux, var=var, labels=_labels_around(spec, star, case["swarm"], case["labels"], rng))
    centre = _star_label(spec, rng, 200.0)
    stars = []
    for i in range(case["stars"]):
        label = (_star_label(spec, rng) if case["swarm"] == "spread" else
                 _labels_around(spec, centre, "contracted", 1, rng)[0])
        n = rng.integers(case["pixels_lo"], case["pixels_hi"] + 1)
        chunks, degree = case["chunks"] or 4 + i % 9, case["degree"] or 3 + i % 6
        stars.append(_observe(case, spec, lines, label, int(n), rng) + (chunks, degree, int(rng.integers(1 << 60))))
    return dict(stars=stars, centre=centre)


# ---------------------------------------------------------------- the calls
def _dispersion(case, spec, wl):
    if case["kind"] == "chi2_variable":
        return pasta.VariableResolutionDispersion(wl, _sigmas(case, spec, wl), _wl_grid(spec))
    return pasta.FixedResolutionDispersion(wl, RESOLUTION, _wl_grid(spec))


def _continuum(case, wl):
    if case.get("continuum") == "linear":
        return pasta.LinearModelContinuumFitter(synth.legendre_design(wl, case["columns"]))
    return pasta.ChunkContinuumFitter(wl, case["chunks"], case["degree"], 0.2)


def _ranges(case, centre):
    """Search ranges of a fit: the whole grid, or narrow ranges around the stars' common centre."""
    if case["swarm"] == "spread":
        return dict(vsini=VSINI, rv=RV, constraints=None)
    half = 2.0 * np.array(_BOX["contracted"])
    half[0] *= centre[0]
    return dict(vsini=(centre[3] - half[3], centre[3] + half[3]), rv=(centre[4] - half[4], centre[4] + half[4]),
                constraints=[pasta.RangeConstraint(k, centre[k] - half[k], centre[k] + half[k]) for k in range(3)])


def prepare(case, seed):
    spec, data = _spec(case["grid"]), _inputs(case, seed)
    interp = _interpolator(case["grid"])
    state = dict(case=case, interp=interp, data=data)
    if case["kind"] == "model":
        state.update(dispersion=_dispersion(case, spec, data["wl"]))
        return state
    if "stars" in data:
        stars = data["stars"]
        state.update(dispersions=[_dispersion(case, spec, s[0]) for s in stars],
                     continua=[pasta.ChunkContinuumFitter(s[0], s[3], s[4], 0.2) for s in stars],
                     settings=pasta.PSOSettings(case["particles"], case["iterations"]), ranges=_ranges(case, data["centre"]))
        if case["kind"] == "served":
            state.update(server=pasta.Server(interp, max_slots=case["slots"]))
        if case["kind"] == "fit":
            state.update(fitter=interp.get_fitter(state["dispersions"][0], state["continua"][0], state["settings"],
                                                  state["ranges"]["vsini"], state["ranges"]["rv"]))
        return state
    disp, cont = _dispersion(case, spec, data["wl"]), _continuum(case, data["wl"])
    settings = pasta.PSOSettings(40, 100)
    if case["kind"] == "binary":
        state.update(continua=_interpolator(case["grid"] + " continua"),
                     fitter=interp.get_binary_fitter(disp, cont, settings, VSINI, RV))
    else:
        state.update(fitter=interp.get_fitter(disp, cont, settings, VSINI, RV))
    return state


def _results(results):
    return dict(labels=np.array([r.label.as_list() for r in results]),
                chi2=np.array([r.chi2 for r in results], np.float32),
                continuum=np.concatenate([np.asarray(r.continuum_params, np.float32) for r in results]))


def run(state):
    case, interp, data = state["case"], state["interp"], state["data"]
    kind = case["kind"]
    if kind == "model":
        if case["labels"] == 1:
            return interp.produce_model(state["dispersion"], *data["labels"][0])
        return interp.produce_model_bulk(state["dispersion"], data["labels"])
    if kind in ("chi2", "chi2_variable"):
        return np.array(state["fitter"].chi2(interp, data["flux"], data["var"], data["labels"]), np.float32)
    if kind == "binary":
        return np.array(state["fitter"].chi2(interp, state["continua"], data["flux"], data["var"], data["labels"]), np.float32)
    stars, ranges = data["stars"], state["ranges"]
    if kind == "fit":
        _, flux, var, _, _, seed = stars[0]
        return _results([state["fitter"].fit(interp, flux, var, constraints=ranges["constraints"], seed=seed)])
    if kind == "fit_many":
        return _results(pasta.fit_many(interp, state["dispersions"], state["continua"], state["settings"],
                                       [s[1] for s in stars], [s[2] for s in stars], ranges["vsini"], ranges["rv"],
                                       seeds=[s[5] for s in stars], constraints=ranges["constraints"]))
    server = state["server"]
    order = {}
    for i, (s, d, c) in enumerate(zip(stars, state["dispersions"], state["continua"])):
        order[server.submit(d, c, state["settings"], s[1], s[2], ranges["vsini"], ranges["rv"], seed=s[5],
                            constraints=ranges["constraints"])] = i
    got = [None] * len(stars)
    while any(r is None for r in got):
        server.step()
        for rid, _, r in server.poll():
            got[order[rid]] = r
    return _results(got)


def work(case):
    """Bytes: the grid rows and spectra a pass has to read once, its labels and its outputs.  Operations: the 64-row
    interpolation, the broadening as 2048-point real transforms there and back, the resampling and the continuum."""
    spec = _spec(case["grid"])
    stars = case.get("stars", 1)
    pixels = case.get("pixels") or (case["pixels_lo"] + case["pixels_hi"]) / 2
    evals = case.get("labels") or stars * case["particles"] * (case["iterations"] + 1)
    parts = 2 if case["kind"] == "binary" else 1
    models = len(spec.teffs) * len(spec.ms) * len(spec.loggs)
    rows = 64 * parts if case["swarm"] == "contracted" else min(models, 64 * evals * parts)
    out = 4 * pixels * evals if case["kind"] == "model" else 4 * evals
    fit = 0 if case["kind"] == "model" else 4 * case["columns"] if case.get("continuum") == "linear" else 2 * ((case["degree"] or 6) + 1) + 2 * (case["degree"] or 6)
    return dict(bytes=float(2 * spec.n_px * rows + 16 * pixels * stars + 40 * evals * parts + out),
                flops=float(evals * (parts * spec.n_px * (2 * 64 + 2 * 2.5 * 11) + pixels * (4 * parts + fit + 8))))


# -------------------------------------------------------- in double precision
def _lagrange(values, x):
    """Four grid points around x (three at the ends) and their Lagrange weights, padded with weight 0."""
    i = int(np.searchsorted(values, x))
    at = [k for k in range(i - 2, i + 2) if 0 <= k < len(values)]
    w = [math.prod((x - values[q]) / (values[p] - values[q]) for q in at if q != p) for p in at]
    return at + [at[0]] * (4 - len(at)), w + [0.0] * (4 - len(w))


def _linear(values, x):
    i = int(np.searchsorted(values, x))
    t = (x - values[i - 1]) / (values[i] - values[i - 1])
    return [i - 1, i], [1.0 - t, t]


def _interpolated(grid, tml, around):
    """Rows of the grid interpolated at labels, in double."""
    spec = _spec(grid.split()[0])
    _, spectra, maxima = _arrays(grid)
    dev = _kept(("device", grid), lambda: torch.tensor(spectra.view(np.int16), device="cuda"))
    cols, ws = [], []
    for t, m, g in tml:
        (ti, tw), (mi, mw), (gi, gw) = around(spec.teffs, t), around(spec.ms, m), around(spec.loggs, g)
        cols.append([(a * len(spec.loggs) + b) * len(spec.ms) + c for a in ti for b in gi for c in mi])
        ws.append([x * y * z for x in tw for y in gw for z in mw])
    cols, ws = np.array(cols), np.array(ws)
    ws = ws / 65535.0 * (1.0 if maxima is None else maxima[cols].astype(np.float64))
    rows = (dev[torch.tensor(cols, device="cuda")].int() & 0xFFFF).double()
    return torch.einsum("bk,bkn->bn", torch.tensor(ws, device="cuda"), rows)


def _models(case, spec, wl, labels):
    rows = _broadened(case, spec, _interpolated(case["grid"], labels[:, :3], _lagrange), labels[:, 3], wl)
    return _at_observed(spec, rows, wl, labels[:, 4])


def _binary(spec, wl, n1, c1, rv1, n2, c2, rv2, ratio):
    """Two normalised rows weighted by their continua, at the observed pixels."""
    lr = torch.tensor(ratio, device="cuda")[:, None] * c1.mean(1, keepdim=True) / c2.mean(1, keepdim=True)
    a, b = _at_observed(spec, n1, wl, rv1), _at_observed(spec, n2, wl, rv2)
    ca, cb = _at_observed(spec, c1, wl, rv1), _at_observed(spec, c2, wl, rv2)
    return (a * ca + lr * b * cb) / (ca + lr * cb)


def _chunk_chi2(wl, chunks, degree, overlap=0.2):
    """Chi2 against (flux, var) rows of models: chunk polynomials of flux / model, blended where they overlap."""
    n = len(wl)
    edge = lambda i: min(max(i / chunks * (wl[-1] - wl[0]) + wl[0], wl[0]), wl[-1])  # noqa: E731
    start = [0 if c == 0 else int(np.searchsorted(wl, edge(c - overlap), "right")) for c in range(chunks)]
    stop = [n if c == chunks - 1 else int(np.searchsorted(wl, edge(c + 1 + overlap), "left")) for c in range(chunks)]
    bases = []
    for a, b in zip(start, stop):
        x = (wl[a:b] - wl[a]) / (wl[b - 1] - wl[a]) * 2.0 - 1.0
        q, _ = np.linalg.qr(np.polynomial.legendre.legvander(x, degree))
        bases.append(torch.tensor(q, device="cuda"))
    fade = []
    for c in range(1, chunks):
        x = wl[start[c]:stop[c - 1]]
        fade.append(torch.tensor(np.sin((x - x[-1]) / (x[0] - x[-1]) * math.pi / 2.0) ** 2, device="cuda"))

    def chi2(model, flux, var):
        y = flux / model
        fits = [(y[:, a:b] @ q) @ q.T for a, b, q in zip(start, stop, bases)]
        cont = torch.empty_like(y)
        for c in range(chunks):
            lo = start[c] if c == 0 else stop[c - 1]
            hi = n if c == chunks - 1 else start[c + 1]
            cont[:, lo:hi] = fits[c][:, lo - start[c]:hi - start[c]]
            if c:
                a, b = start[c], stop[c - 1]
                f = fade[c - 1]
                cont[:, a:b] = fits[c - 1][:, a - start[c - 1]:b - start[c - 1]] * f + fits[c][:, :b - a] * (1.0 - f)
        r = (flux - cont * model)[:, 50:n - 50]
        return (r * r / var[50:n - 50]).sum(1) / (n - 100)
    return chi2


def _linear_chi2(wl, columns):
    n = len(wl)
    q, _ = np.linalg.qr(synth.legendre_design(wl, columns).astype(np.float64))
    q = torch.tensor(q, device="cuda")

    def chi2(model, flux, var):
        y = flux / model
        r = ((y @ q) @ q.T - y)[:, 50:n - 50]
        return (r * r / var[50:n - 50]).sum(1) / n
    return chi2


def exact(case, seed):
    if case["kind"] in ("fit", "fit_many", "served"):
        return None  # a swarm's path has no value of its own in 64 bits
    spec, data = _spec(case["grid"]), _inputs(case, seed)
    wl, labels = data["wl"], data["labels"]
    parts, out = 32 if spec.n_px <= 80000 else 16, []
    if case["kind"] == "model":
        for a in range(0, len(labels), parts):
            out.append(_models(case, spec, wl, labels[a:a + parts]).cpu().numpy())
        out = np.concatenate(out)
        return out[0] if case["labels"] == 1 else out
    chi2 = _linear_chi2(wl, case["columns"]) if case["continuum"] == "linear" else _chunk_chi2(wl, case["chunks"], case["degree"])
    flux, var = (torch.tensor(data[k], device="cuda").double() for k in ("flux", "var"))
    for a in range(0, len(labels), parts):
        lab = labels[a:a + parts]
        if case["kind"] == "binary":
            rows = [_broadened(case, spec, _interpolated(case["grid"], lab[:, k:k + 3], _lagrange), lab[:, k + 3], wl) for k in (0, 5)]
            conts = [_interpolated(case["grid"] + " continua", lab[:, k:k + 3], _linear) for k in (0, 5)]
            model = _binary(spec, wl, rows[0], conts[0], lab[:, 4], rows[1], conts[1], lab[:, 9], lab[:, 10])
        else:
            model = _models(case, spec, wl, lab)
        out.append(chi2(model, flux, var).cpu().numpy())
    return np.concatenate(out)
