"""The calls that programs built on this package spend their time in, at the sizes they use.

Paths (a case's "path"):

* ``pipeline``   one ``Context.phase_pipeline`` call: region maps, active-region integration,
                 convolution and normalisation of every phase of a star.  From host arrays with
                 the raw deficits (what ``driver.run`` does, in the plain form by default) or on
                 device tensors (what a program that keeps its spectra on the GPU does).
* ``quiet``      one ``Context.quiet_disk`` call: the quiet star's disk sum, twice per star.
* ``resolution`` one ``Context.lower_resolution`` call on a quiet spectrum.
* ``deficits_grad``, ``quiet_grad``, ``resolution_grad``, ``rv_fit_grad``: forward and backward
                 of the differentiable form's layers (a fit's step runs all four).
* ``rv_fit``     mask CCF, then Gaussian and bisector fit, of all the spectra of a star.
* ``batch``      one ``Batch.run``: many stars that share their seed spectra.

Inputs follow the generator of ``soap_gpu_gb300.synth``: continuum 1 minus Gaussian lines
(depth U(0.05, 0.9), sigma U(0.03, 0.08) A, about two lines per A), a cubic bisector per mu bin,
spots and faculae of 0.3 to 3 % of the hemisphere, all drawn from the seed.
"""
import ctypes
import math

import numpy as np
import torch

from soap_gpu_gb300 import differentiable as df
from soap_gpu_gb300._lib import Activity, Star
from soap_gpu_gb300.api import Batch, Context

C = 299792458.0
PI = 3.141592653589793238463
R_KM = 696000.0
T_STAR, DT_SPOT, DT_FAC, NRHO = 5778, 663, 250, 20
U1, U2, OMEGA = 0.29, 0.34, -0.18
LB = (0.19, -0.42, 0.36, -0.13)          # facula limb-brightening cubic in mu
SIGMA_V = C / 115000.0 / (2 * math.sqrt(2 * math.log(2)))   # R = 115000
PIPELINE = dict(path="pipeline", vsini=2.0, incl=90.0)


def listed():
    return [
        # the driver's call on a short spectrum: the plain form, host arrays, raw deficits wanted
        dict(PIPELINE, name="driver_100_20k", form="plain64", host=True, raw=True, grid=100, n=20000, step=0.005,
             n_mu=10, n_phase=25, n_region=1),
        # the same star resident on the GPU in the fast form: launches and latency
        dict(PIPELINE, name="step_100_20k", form="fast32", host=False, raw=False, grid=100, n=20000, step=0.005,
             n_mu=10, n_phase=25, n_region=1),
        # the full spectrum (3800-6900 A) of a finely sampled star over a whole rotation
        dict(PIPELINE, name="step_300_310k", form="fast32", host=False, raw=False, grid=300, n=310000, step=0.01,
             n_mu=20, n_phase=100, n_region=2),
        # an uneven grid and pixel count in the plain form, a few phases of an inclined star
        dict(PIPELINE, name="step_151_60001_plain", form="plain64", host=False, raw=False, grid=151, n=60001,
             step=0.01, n_mu=7, n_phase=11, n_region=3, vsini=5.0, incl=60.0),
        # the quiet star of a medium-sized disk in the plain form
        dict(name="quiet_200_100k", path="quiet", form="plain64", grid=200, n=100000, step=0.01, n_mu=10, vsini=2.0,
             incl=90.0),
        # the quiet spectrum of the whole range brought to the instrument's resolution
        dict(name="resolution_310k", path="resolution", form="plain64", n=310000, step=0.01, n_spec=1),
        # one chunk of a fit's phases: deficits and their gradients
        dict(name="deficits_grad_200_100k", path="deficits_grad", grid=200, n=100000, step=0.01, n_mu=10, n_phase=5,
             n_region=3, vsini=2.0, incl=90.0),
        # the quiet spectrum and its gradients
        dict(name="quiet_grad_100_50k", path="quiet_grad", grid=100, n=50000, step=0.01, n_mu=10, vsini=4.0,
             incl=75.0),
        # the resolution step of one chunk of phases and its gradients
        dict(name="resolution_grad_100k", path="resolution_grad", n=100000, step=0.01, n_spec=10),
        # the RV series of a star: 3 types x 100 phases and the quiet spectra
        dict(name="rv_fit_310k", path="rv_fit", n=310000, step=0.01, n_spec=303, n_lines=4000, n_v=161),
        # the RV layer of one chunk of phases and its gradients
        dict(name="rv_fit_grad_100k", path="rv_fit_grad", n=100000, step=0.01, n_spec=10, n_lines=1000, n_v=81),
        # several stars of uneven grids, regions and phases over shared seeds
        dict(name="batch_6_stars_310k", path="batch", n=310000, step=0.01, n_mu=20, n_star=6, grid=250, n_phase=60),
    ]


def draw(rng):
    lg = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    path = rng.choice(("pipeline", "pipeline", "pipeline", "quiet", "resolution", "deficits_grad", "quiet_grad",
                       "resolution_grad", "rv_fit", "rv_fit_grad", "batch"))
    step = rng.choice((0.005, 0.01))
    star = dict(vsini=round(rng.uniform(1.0, 10.0), 3), incl=round(rng.uniform(30.0, 90.0), 2))
    if path == "pipeline":
        form = rng.choice(("fast32", "fast32", "plain64", "fast64"))
        n, grid, host = lg(6000, 310000), lg(40, 300), rng.random() < 0.25
        top = 100 if form == "fast32" else max(1, min(100, int(2.5e9 / (0.02 * grid * grid * n))))
        if host:
            top = max(1, min(top, int(1.5e6 / n)))
        return dict(path=path, form=form, host=host, raw=host or rng.random() < 0.3, grid=grid, n=n, step=step,
                    n_mu=rng.randint(4, 20), n_phase=rng.randint(1, top), n_region=rng.randint(1, 4), **star)
    if path == "quiet":
        form = rng.choice(("plain64", "fast32", "fast64"))
        grid = lg(40, 300)
        top = 310000 if form == "fast32" else min(310000, int(3.2e9 / (0.79 * grid * grid)))
        return dict(path=path, form=form, grid=grid, n=lg(6000, top), step=step, n_mu=rng.randint(4, 20), **star)
    if path == "resolution":
        return dict(path=path, form=rng.choice(("plain64", "plain64", "fast64")), n=lg(6000, 310000), step=step,
                    n_spec=rng.choice((1, 1, 2, 3)))
    if path == "deficits_grad":
        grid = lg(60, 200)
        n = lg(6000, 100000)
        return dict(path=path, grid=grid, n=n, step=step, n_mu=rng.randint(4, 12),
                    n_phase=rng.randint(1, 5), n_region=rng.randint(1, 3), **star)
    if path == "quiet_grad":
        return dict(path=path, grid=lg(40, 130), n=lg(6000, 50000), step=step, n_mu=rng.randint(4, 12), **star)
    if path == "resolution_grad":
        return dict(path=path, n=lg(6000, 100000), step=step, n_spec=rng.randint(1, 20))
    if path == "rv_fit":
        n = lg(30000, 310000)
        return dict(path=path, n=n, step=step, n_spec=lg(3, 303), n_lines=int(n * step * 1.2),
                    n_v=rng.choice((81, 161)))
    if path == "rv_fit_grad":
        n = lg(30000, 100000)
        return dict(path=path, n=n, step=step, n_spec=rng.randint(1, 20), n_lines=int(n * step * 1.0),
                    n_v=rng.choice((81, 161)))
    return dict(path="batch", n=lg(20000, 310000), step=step, n_mu=rng.randint(6, 20), n_star=rng.randint(2, 6),
                grid=rng.randint(60, 250), n_phase=rng.randint(8, 60))


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
_ctx = None


def _context():
    """The one library context that a program keeps open."""
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _n_eff(n):
    return n // 512 * 512


def _wave(case):
    return (3800.0 if case["n"] > 150000 else 5000.0) + np.arange(case["n"]) * case["step"]


def _lines(rng, wave, step):
    """Centres, depths and sigmas of the lines, about two per A."""
    count = max(8, int(2 * (wave[-1] - wave[0])))
    c = np.sort(rng.uniform(wave[0] + 0.5, wave[-1] - 0.5, count))
    return c, rng.uniform(0.05, 0.9, count), rng.uniform(0.03, 0.08, count)


def _spectrum(wave, step, c, d, s):
    half = int(math.ceil(9 * 0.08 / step))
    j = np.rint((c - wave[0]) / step).astype(np.int64)[:, None] + np.arange(-half, half + 1)[None, :]
    ok = (j >= 0) & (j < wave.size)
    x = wave[np.clip(j, 0, wave.size - 1)] - c[:, None]
    v = np.where(ok, d[:, None] * np.exp(-x * x / (2 * s[:, None] ** 2)), 0.0)
    return np.clip(1.0 - np.bincount(np.clip(j, 0, wave.size - 1).ravel(), v.ravel(), wave.size), 0.0, None)


def _bisector(wave, flux, coef):
    """Rows of `flux` shifted by the velocity polynomial `coef` (n_mu x 4) of the flux itself."""
    rows = []
    for c in coef:
        v = ((c[0] * flux + c[1]) * flux + c[2]) * flux + c[3]
        new = wave + wave * (torch.sqrt((1 + v / C) / (1 - v / C)) - 1)
        k = torch.searchsorted(new, wave).clamp(1, wave.numel() - 1)
        x0, x1, y0, y1 = new[k - 1], new[k], flux[k - 1], flux[k]
        y = y0 + (wave - x0) * ((y1 - y0) / (x1 - x0))
        rows.append(torch.where((wave > new[0]) & (wave < new[-1]), y, torch.zeros_like(y)))
    return torch.stack(rows)


def _cubes(rng, wave, step, n_mu):
    c, d, s = _lines(rng, wave, step)
    ds, fs = rng.uniform(0.9, 1.2, c.size), rng.uniform(0.95, 1.05, c.size)
    coef = rng.uniform(-300.0, 300.0, (n_mu, 4))
    w = _dev(wave)
    q = _dev(_spectrum(wave, step, c, d, s))
    sp = _dev(_spectrum(wave, step, c, np.minimum(d * ds, 0.99), s))
    fa = _dev(_spectrum(wave, step, c, np.minimum(d * fs, 0.99), s))
    tilt = 1 + 0.2 * (w - w.mean()) / (w[-1] - w[0])
    qn = _bisector(w, q, coef)
    level = _dev(rng.uniform(0.9, 1.1, (n_mu, 1)))
    return dict(q_norm=qn, q_sed=qn * tilt * level, spot_norm=_bisector(w, sp, coef * 0.5),
                fac_norm=_bisector(w, fa, coef * 0.7), spot_sed=0.3 + 0.05 * tilt, fac_sed=1.0 + 0.05 * tilt)


def _mu_boundary(n_mu):
    return np.linspace(0.95, 0.15, n_mu - 1)


def _regions(rng, count):
    f = rng.uniform(0.003, 0.03, count)
    return np.column_stack([rng.uniform(-50, 50, count), rng.uniform(0, 360, count), np.sqrt(f),
                            rng.integers(0, 2, count).astype(float)])


def _star_regions(rng, case):
    reg = _regions(rng, case["n_region"])
    reg[0, 1] = 180.0 + rng.uniform(-20, 20)      # one region crosses the disk around phase 0.5
    reg[0, 0] = rng.uniform(-20, 40)
    n_ph = case["n_phase"]
    ph = np.arange(n_ph) / max(n_ph, 1) if n_ph > 2 else 0.5 + 0.05 * np.arange(n_ph)
    return reg, ph


def _period(vsini):
    return 2 * PI * R_KM / (vsini * 86400.0)


def _star(case, grid=None):
    return Star(int(grid or case["grid"]), _period(case["vsini"]), OMEGA, case["incl"], R_KM, U1, U2,
                (ctypes.c_double * 4)(*LB))


ACT = Activity(T_STAR, DT_SPOT, DT_FAC, NRHO, 0)


def _maps_np(grid, vsini, incl, n_mu):
    """Velocity [km/s], limb darkening, mu, mu bin and limb brightening of the disk's cells."""
    w0 = 360.0 / _period(vsini)
    w1 = w0 * OMEGA
    k = np.arange(grid, dtype=np.float64)
    th = -90.0 + k * (180.0 / grid)
    s = np.sin(th * PI / 180)
    ov = (w0 + w1 * (s * s)) * PI / (180 * 24 * 3600) * R_KM
    y, z = (-1. + k * (2. / grid))[:, None], (-1. + k * (2. / grid))[None, :]
    delta = y * ov[None, :] * math.sin(incl * PI / 180.)
    r2 = y * y + z * z
    vis = r2 <= 1.
    mu = np.sqrt(np.where(vis, 1. - r2, 0.0))
    om = 1. - mu
    limb = 1. - U1 * om - U2 * om * om
    lb = LB[0] + LB[1] * mu + LB[2] * mu * mu + LB[3] * mu * mu * mu
    above = mu[..., None] > _mu_boundary(n_mu)
    region = np.where(above.any(-1), above.argmax(-1), n_mu - 1)
    flat = lambda a, f: np.where(vis, a, f).ravel()
    return dict(delta=flat(delta, -999.), limb=flat(limb, -999.), mu=flat(mu, -999.), region=flat(region, 0),
                lb=flat(lb, -999.))


def _broadened(wave, rows, m, n_eff):
    """A quiet spectrum of about the disk's velocities: the rows of each mu bin at nine shifts,
    with the limb weights of the cells that move so."""
    vis = m["limb"] > -998.
    d, l, r = m["delta"][vis], m["limb"][vis], m["region"][vis]
    top = max(np.abs(d).max(), 1e-9)
    v = np.rint(d / top * 4).astype(int)
    out = torch.zeros_like(rows[0])
    x = torch.arange(rows.shape[1], device=rows.device, dtype=torch.float64)
    step = float(wave[1] - wave[0])
    for k in range(-4, 5):
        pos = (x - (k / 4 * top * 1000 / C) * _dev(wave) / step).clamp(0, rows.shape[1] - 1.001)
        i = pos.floor().long()
        f = pos - i
        for b in range(rows.shape[0]):
            w = float(l[(v == k) & (r == b)].sum())
            if w:
                out = out + w * (rows[b][i] * (1 - f) + rows[b][i + 1] * f)
    out[n_eff:] = 0.0
    return out


def _low_spectra(rng, wave, step, count, n_eff):
    """Normalised spectra of a star at the instrument's resolution, each a little shifted and deformed."""
    c, d, s = _lines(rng, wave, step)
    s = np.sqrt(s * s + (c * (SIGMA_V / C)) ** 2 + 0.02 ** 2)
    base = _dev(_spectrum(wave, step, c, d * 0.8, s))
    base = base / base.max()
    x = torch.arange(wave.size, device="cuda", dtype=torch.float64)
    out = torch.empty((count, n_eff), dtype=torch.float64, device="cuda")
    amp, ph = rng.uniform(-0.3, 0.3, count), rng.uniform(0, 6.28, count)
    for q in range(count):
        pos = (x + float(amp[q])).clamp(0, wave.size - 1.001)
        i = pos.floor().long()
        f = pos - i
        y = base[i] * (1 - f) + base[i + 1] * f
        out[q] = (y * (1 + 1e-3 * torch.sin(x * 1e-3 + float(ph[q]))))[:n_eff]
    return out, c, d


def _mask(wave_trim, c, d, count):
    lo, hi = wave_trim[0] + 0.5, wave_trim[-1] - 0.5
    k = np.nonzero((c > lo) & (c < hi))[0]
    pick = np.sort(k[np.argsort(-d[k])][:count])
    return c[pick], np.ones(pick.size)


def _velocities(n_v):
    return np.linspace(-20000.0, 20000.0, n_v)


def _g(rng, *shape):
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    return torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")


def _inputs(case, seed):
    """The tensors that `prepare` hands over and `exact` computes from."""
    rng = np.random.default_rng(seed)
    n_eff = _n_eff(case["n"])
    wave = _wave(case)
    p = dict(wave=wave, n_eff=n_eff)
    path = case["path"]
    if path in ("pipeline", "quiet", "deficits_grad", "quiet_grad", "batch"):
        p["cubes"] = _cubes(rng, wave, case["step"], case["n_mu"])
    if path in ("pipeline", "deficits_grad"):
        p["regions"], p["phases"] = _star_regions(rng, case)
    if path == "pipeline":
        m = _maps_np(case["grid"], case["vsini"], case["incl"], case["n_mu"])
        p["quiet_norm"] = _broadened(wave, p["cubes"]["q_norm"], m, n_eff)
        p["quiet_sed"] = _broadened(wave, p["cubes"]["q_sed"], m, n_eff)
    elif path == "deficits_grad":
        p["g"] = _g(rng, case["n_phase"], 3, case["n"])
    elif path == "quiet_grad":
        p["g"] = _g(rng, case["n"])
    elif path in ("resolution", "resolution_grad"):
        c, d, s = _lines(rng, wave, case["step"])
        s = np.sqrt(s * s + 0.03 ** 2)
        base = _dev(_spectrum(wave, case["step"], c, d, s)) * (1000.0 + 0.02 * (_dev(wave) - 5000.0))
        base[n_eff:] = 0.0
        k = _dev(rng.uniform(0.002, 0.02, (case["n_spec"], 1)))
        x = torch.arange(case["n"], device="cuda", dtype=torch.float64)[None, :]
        spec = base[None, :] * k * (1 + 0.05 * torch.sin(x * _dev(rng.uniform(1e-3, 1e-2, (case["n_spec"], 1)))))
        p["base"], p["spec"] = base, (spec if path == "resolution_grad" else base[None, :] - spec)
        if path == "resolution_grad":
            p["g"] = _g(rng, case["n_spec"], n_eff)
    elif path in ("rv_fit", "rv_fit_grad"):
        low, c, d = _low_spectra(rng, wave, case["step"], case["n_spec"], n_eff)
        p["wave_trim"] = wave[:n_eff][210:-210]
        p["spectra"] = low[:, 210:-210].contiguous()
        p["lines"] = _mask(p["wave_trim"], c, d, case["n_lines"])
        if path == "rv_fit_grad":
            p["g"] = _g(rng, case["n_spec"], 5)
    elif path == "batch":
        stars = []
        for q in range(case["n_star"]):     # grids and phases from half and a third of the largest up to it
            part = (q + 1) / case["n_star"]
            grid = max(40, int(case["grid"] * (0.5 + 0.5 * part)))
            n_ph = max(1, int(case["n_phase"] * (1 / 3 + 2 / 3 * part)))
            reg = _regions(rng, int(rng.integers(1, 7)))
            st = Star(grid, _period(float(rng.uniform(1.0, 10.0))), OMEGA, 90.0, R_KM, U1, U2,
                      (ctypes.c_double * 4)(*LB))
            stars.append((st, np.arange(n_ph) / n_ph, [reg] * n_ph))
        p["stars"] = stars
    return p


def prepare(case, seed):
    ctx = _context()
    p = _inputs(case, seed)
    path, step, n_eff = case["path"], case["step"], p["n_eff"]
    w = _dev(p["wave"])
    st = dict(case=case, ctx=ctx, n_eff=n_eff, wave=w)
    if path in ("pipeline", "quiet"):
        mu_b = _mu_boundary(case["n_mu"])
        st["maps"] = ctx.disk_maps(case["grid"], _period(case["vsini"]), OMEGA, case["incl"], R_KM, U1, U2,
                                   mu_b if case.get("host") else _dev(mu_b), LB)
    if path == "pipeline":
        st.update(cubes=p["cubes"], quiet=(p["quiet_sed"], p["quiet_norm"]), star=_star(case), phases=p["phases"],
                  regions=[p["regions"]] * case["n_phase"])
        if case["host"]:
            st["wave"] = p["wave"]
            st["cubes"] = {k: v.cpu().numpy() for k, v in p["cubes"].items()}
            st["quiet"] = tuple(q.cpu().numpy() for q in st["quiet"])
    elif path == "quiet":
        st["cube"] = p["cubes"]["q_norm"]
    elif path == "resolution":
        st["spec"] = p["spec"]
    elif path in ("deficits_grad", "quiet_grad"):
        reg, ph = (p["regions"], p["phases"]) if path == "deficits_grad" else (np.zeros((0, 4)), np.array([0.5]))
        st["setup"] = df.IntegrationSetup.build(
            ctx, p["wave"], n_eff, case["grid"], _period(case["vsini"]), OMEGA, case["incl"], R_KM,
            _mu_boundary(case["n_mu"]), LB, ph, [reg] * len(ph), ACT, step)
        st["params"] = _dev([U1, U2, case["vsini"], case["incl"]]).requires_grad_()
        names = df.CUBE_KEYS if path == "deficits_grad" else ("q_norm",)
        st["cubes"] = [p["cubes"][k].requires_grad_() for k in names]
        st["g"] = p["g"]
    elif path == "resolution_grad":
        st["setup"] = df.ResolutionSetup(ctx, w, n_eff, SIGMA_V, step_mult=step, step_exp=step)
        st["spec"], st["base"], st["g"] = p["spec"].requires_grad_(), p["base"].requires_grad_(), p["g"]
    elif path in ("rv_fit", "rv_fit_grad"):
        lw, wt = (_dev(a) for a in p["lines"])
        st["mask"] = (_dev(_velocities(case["n_v"])), lw, wt, _dev(p["wave_trim"]))
        st["spectra"] = p["spectra"]
        if path == "rv_fit_grad":
            st["setup"] = df.CcfSetup(ctx, *st["mask"], step, mask_step=step, index_old=int(100.0 / step))
            st["spectra"], st["g"] = p["spectra"].requires_grad_(), p["g"]
    else:
        stars, phases, regions = zip(*p["stars"])
        st["batch"] = Batch(ctx, w, n_eff, p["cubes"], _mu_boundary(case["n_mu"]), step, ACT, SIGMA_V, list(stars),
                            list(phases), list(regions))
    return st


def run(st):
    case, ctx, step, n_eff = st["case"], st["ctx"], st["case"]["step"], st["n_eff"]
    path = case["path"]
    if path == "pipeline":
        return ctx.phase_pipeline(case["form"], st["wave"], n_eff, st["star"], st["maps"], st["cubes"], step, ACT,
                                  st["phases"], st["regions"], st["quiet"][0], st["quiet"][1], SIGMA_V,
                                  conv_step=step, want_raw=case["raw"])
    if path == "quiet":
        return ctx.quiet_disk(case["form"], st["wave"], st["cube"], n_eff, st["maps"], case["grid"], step)
    if path == "resolution":
        return ctx.lower_resolution(case["form"], st["wave"], st["spec"], n_eff, SIGMA_V, step_mult=step,
                                    step_exp=step)
    if path == "deficits_grad":
        out = df.deficit_spectra(st["params"], *st["cubes"], st["setup"])
        return out, torch.autograd.grad(out, [st["params"], *st["cubes"]], st["g"])
    if path == "quiet_grad":
        out = df.quiet_spectrum(st["params"], st["cubes"][0], st["setup"])
        return out, torch.autograd.grad(out, [st["params"], st["cubes"][0]], st["g"])
    if path == "resolution_grad":
        out = df.lower_resolution(st["spec"], st["base"], st["setup"])
        return out, torch.autograd.grad(out, [st["spec"], st["base"]], st["g"])
    if path == "rv_fit":
        ccf = ctx.ccf("plain64", *st["mask"], step, st["spectra"], mask_step=step, index_old=int(100.0 / step))
        fit = ctx.gauss_bis(st["mask"][0], ccf)
        return ccf, fit
    if path == "rv_fit_grad":
        par = df.gauss_fit_bis(df.normalised_ccf(st["spectra"], st["setup"]), st["setup"])
        return par, torch.autograd.grad(par, [st["spectra"]], st["g"])
    return st["batch"].run()


# ---------------------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------------------
def _active(case):
    """Active cells of all phases, about: a region of 1.65 % of the hemisphere is in view half
    of the time and covers about 0.6 of its area in the disk's cells."""
    return 0.5 * case["n_phase"] * case["n_region"] * 0.0165 * 2 * 0.6 * 0.7854 * case["grid"] ** 2


def work(case):
    path, n = case["path"], case["n"]
    taps = 2 * 9 * SIGMA_V / C * 5000.0 / case["step"]      # +- 9 sigma of the instrument
    if path == "pipeline":
        rows = 4 * case["n_mu"] * n * 8
        out = case["n_phase"] * 3 * n * 8 * (2 if case["raw"] else 1)
        flops = 6.0 * case["n_phase"] * n * taps
        if case["form"] == "plain64":       # three interpolations and three sums per active cell and pixel
            flops += 26.0 * _active(case) * n
        return dict(bytes=rows + 5 * n * 8 + 36 * case["grid"] ** 2 + out, flops=flops)
    if path == "quiet":
        cells = 0.7854 * case["grid"] ** 2
        return dict(bytes=(case["n_mu"] + 2) * n * 8 + 20 * case["grid"] ** 2,
                    flops=10.0 * cells * n if case["form"] == "plain64" else 0)
    if path == "resolution":
        return dict(bytes=(2 * case["n_spec"] + 1) * n * 8, flops=2.0 * case["n_spec"] * n * taps)
    if path == "deficits_grad":
        return dict(bytes=(8 * case["n_mu"] + 5 + 6 * case["n_phase"]) * n * 8 + 16 * case["n_phase"] * case["grid"] ** 2,
                    flops=26.0 * _active(case) * n)
    if path == "quiet_grad":
        return dict(bytes=(2 * case["n_mu"] + 3) * n * 8 + 36 * case["grid"] ** 2,
                    flops=10.0 * 0.7854 * case["grid"] ** 2 * n)
    if path == "resolution_grad":
        return dict(bytes=(4 * case["n_spec"] + 3) * n * 8, flops=4.0 * case["n_spec"] * n * taps)
    if path == "rv_fit":       # the mask holds about four pixels per line and velocity
        nnz = 4.0 * case["n_lines"] * case["n_v"]
        return dict(bytes=case["n_spec"] * n * 8 + 12 * nnz, flops=2.0 * nnz * case["n_spec"])
    if path == "rv_fit_grad":
        nnz = 4.0 * case["n_lines"] * case["n_v"]
        return dict(bytes=2 * case["n_spec"] * n * 8 + 12 * nnz, flops=4.0 * nnz * case["n_spec"])
    ph = case["n_star"] * case["n_phase"] * 0.67
    return dict(bytes=4 * case["n_mu"] * n * 8 + ph * 3 * n * 8, flops=6.0 * ph * n * taps)


# ---------------------------------------------------------------------------------------
# the same outputs in plain torch and numpy, in 64 bits
# ---------------------------------------------------------------------------------------
class _Cells:
    """Some cells' owner intervals and interpolation weights at every output pixel."""

    def __init__(self, wave, n_eff, step, delta):
        d = delta[:, None]
        b = d * 1000. / C
        sq = torch.sqrt((1 + b) / (1 - b))
        fb = -1 * (1 - sq)
        off = fb * wave[0] / step
        j = torch.arange(n_eff, device=wave.device)
        first = torch.ceil(j.double()[None, :] * (1 + fb) + off).long().contiguous()
        o = torch.searchsorted(first, j[None, :].expand(d.shape[0], -1).contiguous(), right=True) - 1
        still = d == 0
        o = torch.where(still, j[None, :], o)
        self.ok = (o >= 0) & ((o <= n_eff - 2) | still)
        self.o = o.clamp(0, n_eff - 2)
        l0, l1 = wave[self.o], wave[self.o + 1]
        s0, s1 = l0 + (-1 * l0) * (1 - sq), l1 + (-1 * l1) * (1 - sq)
        self.dd = s1 - s0
        self.w = torch.where(still, (j[None, :] - self.o).double(), (wave[:n_eff] - s0) / self.dd)
        # the weight without the cancellation in l_j - l'_o: the adjoints' exact value
        fine = ((wave[:n_eff] - l0) - l0 * fb) / ((l1 - l0) * sq)
        self.fine = torch.where(still, (j[None, :] - self.o).double(), fine)
        omb = 1 - b
        self.dw = -wave[:n_eff] * (1000. / C) / (sq ** 3 * omb ** 2) / (l1 - l0)     # d weight / d velocity

    def at(self, rows, row, fine=False):
        """Values of the cells' rows (n_mu x n), and the differences across their intervals."""
        a = rows[row[:, None], self.o]
        e = rows[row[:, None], self.o + 1] - a
        zero = torch.zeros_like(a)
        return (torch.where(self.ok, a + e * (self.fine if fine else self.w), zero),
                torch.where(self.ok, e, zero))


def _region_maps(case, regions, phases, grid, incl):
    """Temperature and type of every cell, phase by phase (-9999 outside of the regions)."""
    inc = incl * PI / 180.
    k = np.arange(grid, dtype=np.float64)
    y, z = (-1. + k * (2. / grid))[:, None], (-1. + k * (2. / grid))[None, :]
    r2 = z * z + y * y
    xa = np.sqrt(np.maximum(1. - (y * y + z * z), 0.0))
    step = 2. / grid
    for ph in phases:
        t, b = np.full((grid, grid), -9999.0), np.full((grid, grid), -9999.0)
        for lat, lon, s, typ in regions:
            la, lo = lat * PI / 180., lon * PI / 180.
            rho = -PI + np.arange(NRHO) * (2. * PI / (NRHO - 1))
            rim = np.stack([np.full(NRHO, math.sqrt(1 - s * s)), s * np.cos(rho), s * np.sin(rho)])
            bb, g, b2 = -la, lo, PI / 2. - inc
            cb, sb, cg, sg, c2, s2 = (f(v) for v in (bb, g, b2) for f in (math.cos, math.sin))
            rot = np.array([[c2 * cg * cb - sb * s2, -sg * c2, c2 * cg * sb + s2 * cb], [sg * cb, cg, sg * sb],
                            [-s2 * cg * cb - c2 * sb, s2 * sg, -s2 * cg * sb + c2 * cb]])
            cp, sp = math.cos(-ph * 2 * PI), math.sin(-ph * 2 * PI)
            ax = np.array([math.cos(inc), 0.0, math.sin(inc)])
            sk = np.array([[0, ax[2], -ax[1]], [-ax[2], 0, ax[0]], [ax[1], -ax[0], 0]])
            turn = (1 - cp) * np.outer(ax, ax) + cp * np.eye(3) + sp * sk
            v = turn @ (rot @ rim)
            on = v[0] >= 0
            if not on.any():
                continue
            ylo, yhi, zlo, zhi = (min(1, v[1][on].min()), max(-1, v[1][on].max()), min(1, v[2][on].min()),
                                  max(-1, v[2][on].max()))
            if not on.all():
                if ylo * yhi < 0:
                    zlo, zhi = (-1, zhi) if zlo < 0 else (zlo, 1)
                if zlo * zhi < 0:
                    ylo, yhi = (-1, yhi) if ylo < 0 else (ylo, 1)
            box = np.zeros((grid, grid), bool)
            box[max(0, math.floor((1. + ylo) / step)):max(0, math.ceil((1. + yhi) / step)),
                max(0, math.floor((1. + zlo) / step)):max(0, math.ceil((1. + zhi) / step))] = True
            g2 = (ph - 1.0) * (2 * PI)
            c, sn, ci, si = math.cos(g2), math.sin(g2), math.cos(inc), math.sin(inc)
            back = np.array([[(1 - c) * ci * ci + c, sn * si, (1 - c) * ci * si], [-sn * si, c, sn * ci],
                             [(1 - c) * si * ci, -sn * ci, (1 - c) * si * si + c]])
            cg, sg, cb, sb = math.cos(-lo), math.sin(-lo), math.cos(la), math.sin(la)
            c2, s2 = math.cos(-(PI / 2. - inc)), math.sin(-(PI / 2. - inc))
            row = np.array([cb * cg * c2 - s2 * sb, -sg * cb, cb * cg * s2 + sb * c2]) @ back
            x = row[0] * xa + row[1] * y + row[2] * z
            hit = box & (r2 < 1.) & (x * x >= 1. - s * s)
            if typ == 0:
                t[hit], b[hit] = T_STAR - DT_SPOT, 0.0
            else:
                tf = T_STAR + DT_FAC + 0.9 - 407.7 * xa + 190.9 * (xa * xa)
                t[hit], b[hit] = np.trunc(tf)[hit], 1.0
        yield t.ravel(), b.ravel()


def _chunk(n):
    return max(1, int(6e6 / n))


def _deficits(case, p, limit=2.5e10):
    """Deficits (phases x (tot, flux, bconv) x n_eff), None where it would take too long."""
    m = _maps_np(case["grid"], case["vsini"], case["incl"], case["n_mu"])
    maps = list(_region_maps(case, p["regions"], p["phases"], case["grid"], case["incl"]))
    if sum(int((b >= 0).sum()) for _, b in maps) * p["n_eff"] > limit:
        return None
    c, n_eff = p["cubes"], p["n_eff"]
    w = _dev(p["wave"])
    out = torch.zeros((len(maps), 3, n_eff), dtype=torch.float64, device="cuda")
    for k, (t, b) in enumerate(maps):
        for typ, cube, sed in ((0, "spot_norm", "spot_sed"), (1, "fac_norm", "fac_sed")):
            idx = np.nonzero(b == typ)[0]
            for c0 in range(0, idx.size, _chunk(n_eff)):
                i = idx[c0:c0 + _chunk(n_eff)]
                g = _Cells(w, n_eff, case["step"], _dev(m["delta"][i]))
                row = torch.as_tensor(m["region"][i], device="cuda")
                lim = _dev(m["limb"][i])[:, None]
                q, s, a = (g.at(c[f], row)[0] * lim for f in ("q_norm", "q_sed", cube))
                inten = c[sed][None, :n_eff] * (1.0 if typ == 0 else _dev(1.0 + m["lb"][i])[:, None])
                out[k, 0] += (s - inten * a).sum(0)
                out[k, 1] += (s - inten * q).sum(0)
                out[k, 2] += (q - a).sum(0)
    return out


def _sigma(lam):
    b = SIGMA_V / C
    return -1 * lam * (1 - math.sqrt((1 + b) / (1 - b)))


def _low(case, wave, spec, n_eff):
    """Convolved and normalised spectra, their minimum and the convolution's maximum."""
    n = spec.shape[1]
    b = SIGMA_V / C
    d32 = -1 * wave[0] * (1 - float(np.sqrt(np.float32((1 + b) / (1 - b)))))
    half = 50.0 * d32 / (wave[1] - wave[0])
    wid = int(math.ceil(half) if half - math.floor(half) >= 0.5 else math.floor(half))
    lam = _dev(wave)[:n_eff]
    sig = _sigma(lam)
    i = torch.arange(n_eff, device="cuda")
    inside = (i > wid) & (i + wid < n - 1)
    conv = torch.zeros((spec.shape[0], n_eff), dtype=torch.float64, device="cuda")
    for d in range(-wid, wid - 1):
        e = torch.exp(-(d * d) * case["step"] * case["step"] / (2 * sig * sig)) / (sig * math.sqrt(2 * PI))
        conv += case["step"] * (1 - spec[:, (i + d).clamp(0, n - 1)]) * torch.where(inside, e, torch.zeros_like(e))
    mn = spec.min(1).values
    mx = torch.where(conv != 0, conv, torch.full_like(conv, -60000.0)).max(1).values
    return 1 - conv * ((1 - mn) / mx)[:, None], torch.stack([mn, mx], 1), conv, wid, sig, inside


def _exact_pipeline(case, p):
    d = _deficits(case, p)
    if d is None:
        return None
    n_eff = p["n_eff"]
    low = torch.empty_like(d)
    full = torch.zeros((3, case["n"]), dtype=torch.float64, device="cuda")
    for k in range(d.shape[0]):
        full[:, :n_eff] = d[k]
        base = torch.stack([p["quiet_sed"], p["quiet_sed"], p["quiet_norm"]])
        low[k] = _low(case, p["wave"], base - full, n_eff)[0]
    return (low, d) if case["raw"] else low


def _all_cells(case, p, cube, g=None):
    """The quiet sum of a cube; with `g` the gradients of its product with g too."""
    m = _maps_np(case["grid"], case["vsini"], case["incl"], case["n_mu"])
    n_eff, w = p["n_eff"], _dev(p["wave"])
    idx = np.nonzero(m["limb"] > -998.)[0]
    if idx.size * n_eff > (8e9 if g is None else 2e9):
        return None
    out = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
    grad = torch.zeros_like(cube)
    gl, gd = [], []
    for c0 in range(0, idx.size, _chunk(n_eff)):
        i = idx[c0:c0 + _chunk(n_eff)]
        k = _Cells(w, n_eff, case["step"], _dev(m["delta"][i]))
        row = torch.as_tensor(m["region"][i], device="cuda")
        lim = _dev(m["limb"][i])[:, None]
        v, e = k.at(cube, row)
        out[:n_eff] += (v * lim).sum(0)
        if g is not None:
            _scatter(grad, k, row, lim * g[None, :n_eff])
            gl.append((k.at(cube, row, True)[0] * g[:n_eff]).sum(1))
            gd.append((e * k.dw * g[:n_eff]).sum(1) * lim[:, 0])
    if g is None:
        return out
    return out, (_param_grad(case, m, idx, torch.cat(gl), torch.cat(gd)), grad)


def _scatter(grad, k, row, h):
    """grad[row, o] and grad[row, o + 1] += the shares of h at every pixel."""
    n = grad.shape[1]
    h = torch.where(k.ok, h, torch.zeros_like(h))
    at = (row[:, None] * n + k.o).reshape(-1)
    grad.view(-1).index_add_(0, at, (h * (1 - k.fine)).reshape(-1))
    grad.view(-1).index_add_(0, at + 1, (h * k.fine).reshape(-1))


def _param_grad(case, m, idx, gl, gd):
    om, dl = _dev(1.0 - m["mu"][idx]), _dev(m["delta"][idx])
    r = case["incl"] * PI / 180.
    gv = (gd * dl).sum()
    return torch.stack([-(gl * om).sum(), -(gl * om * om).sum(), gv / case["vsini"],
                        gv * (PI / 180.) * math.cos(r) / math.sin(r)])


def _exact_deficits_grad(case, p):
    d = _deficits(case, p, 3e9)
    if d is None:
        return None
    c, n_eff, w = p["cubes"], p["n_eff"], _dev(p["wave"])
    out = torch.zeros((case["n_phase"], 3, case["n"]), dtype=torch.float64, device="cuda")
    out[:, 0, :n_eff], out[:, 1, :n_eff], out[:, 2, :n_eff] = d[:, 1], d[:, 2], d[:, 0]
    m = _maps_np(case["grid"], case["vsini"], case["incl"], case["n_mu"])
    gr = {k: torch.zeros_like(v) for k, v in c.items()}
    gm = case["grid"] ** 2
    gl, gd = (torch.zeros(gm, dtype=torch.float64, device="cuda") for _ in range(2))
    for k, (t, b) in enumerate(_region_maps(case, p["regions"], p["phases"], case["grid"], case["incl"])):
        gf, gb, gt = (p["g"][k, q, :n_eff][None, :] for q in range(3))
        for typ, cube, sed in ((0, "spot_norm", "spot_sed"), (1, "fac_norm", "fac_sed")):
            idx = np.nonzero(b == typ)[0]
            for c0 in range(0, idx.size, _chunk(n_eff)):
                i = idx[c0:c0 + _chunk(n_eff)]
                g = _Cells(w, n_eff, case["step"], _dev(m["delta"][i]))
                row, lim = torch.as_tensor(m["region"][i], device="cuda"), _dev(m["limb"][i])[:, None]
                ratio = 1.0 if typ == 0 else _dev(1.0 + m["lb"][i])[:, None]
                inten = c[sed][None, :n_eff] * ratio
                hs, hq, ha = gf + gt, gb - inten * gf, -gb - inten * gt
                (q, eq), (s, es), (a, ea) = (g.at(c[f], row, True) for f in ("q_norm", "q_sed", cube))
                _scatter(gr["q_sed"], g, row, lim * hs)
                _scatter(gr["q_norm"], g, row, lim * hq)
                _scatter(gr[cube], g, row, lim * ha)
                gr[sed][:n_eff] += (-ratio * lim * (q * gf + a * gt)).sum(0)
                at = torch.as_tensor(i, device="cuda")
                gl[at] += (s * hs + q * hq + a * ha).sum(1)
                gd[at] += ((es * hs + eq * hq + ea * ha) * g.dw).sum(1) * lim[:, 0]
    idx = np.nonzero(m["limb"] > -998.)[0]
    at = torch.as_tensor(idx, device="cuda")
    return out, (_param_grad(case, m, idx, gl[at], gd[at]), *[gr[k] for k in df.CUBE_KEYS])


def _first(hit):
    """The first true column of each row."""
    at = torch.arange(hit.shape[1], device=hit.device)
    return torch.where(hit, at, hit.shape[1]).min(1).values


def _exact_resolution_grad(case, p):
    n, n_eff, wave = case["n"], p["n_eff"], p["wave"]
    a = p["base"][None, :] - p["spec"]
    out, mm, conv, wid, sig, inside = _low(case, wave, a, n_eff)
    mn, mx, g = mm[:, 0], mm[:, 1], p["g"]
    s = (g * conv).sum(1)
    gc = -((1 - mn) / mx)[:, None] * g
    rows = torch.arange(a.shape[0], device="cuda")
    gc[rows, _first(conv == mx[:, None])] += s * (1 - mn) / (mx * mx)
    ga = torch.zeros_like(a)
    i = torch.arange(n_eff, device="cuda")
    gc = torch.where(inside, gc, torch.zeros_like(gc))
    for d in range(-wid, wid - 1):
        k = case["step"] * torch.exp(-(d * d) * case["step"] * case["step"] / (2 * sig * sig)) / (sig * math.sqrt(2 * PI))
        lo, hi = max(0, -d), min(n_eff, n - d)
        ga[:, lo + d:hi + d] -= (k * gc)[:, lo:hi]
    ga[rows, _first(a == mn[:, None])] += s / mx
    return out, (-ga, ga.sum(0))


def _exact_ccf(case, p):
    """The normalised, apodised CCF from the dense mask, a velocity at a time."""
    wt, n = p["wave_trim"], p["wave_trim"].size
    lw, wg = p["lines"]
    step, ext = case["step"], int(100.0 / case["step"])
    grid = np.concatenate([np.linspace(wt[0] - step * ext, wt[0], ext), wt,
                           np.linspace(wt[-1], wt[-1] + step * ext, ext)])
    b = 820. / C
    k = math.sqrt((1 + b) / (1 - b)) - 1
    rows = []
    for v in _velocities(case["n_v"]):
        at = lw * (1 + v / C)
        hw = at * k
        beg, end = at - hw / 2, at + hw / 2
        lo = np.ceil((beg - grid.min()) / step).astype(int)
        hi = (np.ceil((end - grid.min()) / step) - 1).astype(int)
        mask = np.zeros(grid.size)
        fb = np.abs(grid[lo] - beg) / (grid[lo] - grid[lo - 1])
        fa = np.abs(grid[hi] - end) / (grid[hi + 1] - grid[hi])
        for q in range(lw.size):       # later lines overwrite
            mask[lo[q]:hi[q]] = wg[q]
            mask[lo[q] - 1] = wg[q] * fb[q]
            mask[hi[q]] = wg[q] * fa[q]
        rows.append(p["spectra"] @ _dev(mask[ext:-ext]))
    ccf = torch.stack(rows, 1)
    n_v = case["n_v"]
    period = int((n_v - 1) / 2.)
    length = int(period / 2.)
    ramp = 0.5 * np.cos(2 * PI / period * np.arange(length) - PI) + 0.5
    win = np.concatenate([np.zeros(5), ramp, np.ones(n_v - period - 10), ramp[::-1], np.zeros(5)])
    return 1 - (1 - ccf / ccf.max(1, keepdim=True).values) * _dev(win)[None, :]


def exact(case, seed):
    path = case["path"]
    if path in ("rv_fit_grad", "batch"):
        return None
    p = _inputs(case, seed)
    if path == "pipeline":
        return _exact_pipeline(case, p)
    if path == "quiet":
        return _all_cells(case, p, p["cubes"]["q_norm"])
    if path == "resolution":
        return _low(case, p["wave"], p["spec"], p["n_eff"])[:2]
    if path == "deficits_grad":
        return _exact_deficits_grad(case, p)
    if path == "quiet_grad":
        return _all_cells(case, p, p["cubes"]["q_norm"], p["g"])
    if path == "resolution_grad":
        return _exact_resolution_grad(case, p)
    return _exact_ccf(case, p), {k: None for k in ("model", "par", "depth", "bis", "iters")}
