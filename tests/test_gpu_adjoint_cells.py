"""The gradients of the per-phase integration, entry by entry, against sums over single cells in
numpy's extended precision: every cell's owner at every pixel and its interpolation weight

    w = (l_j - l'_o) / (S (l_{o+1} - l_o)),   l'_o = S l_o, S = sqrt((1 + b) / (1 - b)),

with l'_o rounded as the forward rounds it for the row gradients (they are the transpose of the
forward) and exact for the continuum, limb and velocity gradients."""
import numpy as np
import pytest

import oracle
from soap_gpu_gb300._lib import Activity

pytestmark = pytest.mark.gpu
C = 299792458.0
LD = np.longdouble
ROWS = ("q_norm", "q_sed", "spot_norm", "fac_norm")


def _maps(grid, vsini, n_mu):
    period = 2 * np.pi * 696000.0 / (vsini * 86400.0)
    return dict(oracle.disk_maps(grid, period, -0.18, 80.0, 696000.0, 0.3, 0.3, np.linspace(0.95, 0.15, n_mu - 1),
                                 (0.2, -0.4, 0.3, -0.1)))


def _reference(wave, n_eff, bi, maps, x, step, g):
    """The gradients and, for each entry, the sum of the magnitudes of what it is made of and the
    number of cells.  Temperatures of unit Planck ratio, faculae 1 + LB."""
    n, n_mu = wave.size, x["q_norm"].shape[0]
    j = np.arange(n_eff)
    lam = wave[:n_eff]
    out = {k: np.zeros(x[k].shape, LD) for k in x}
    out["limb"], out["delta"] = (np.zeros(maps["limb"].size, LD) for _ in range(2))
    mag = {k: np.zeros_like(v) for k, v in out.items()}
    cnt = {k: np.zeros(v.shape, int) for k, v in out.items()}

    def put(key, at, v, m):
        np.add.at(out[key], at, v)
        np.add.at(mag[key], at, m)
        np.add.at(cnt[key], at, 1)

    for p in range(bi.shape[0]):
        gF, gB, gT = (g[q, p, :n_eff].astype(LD) for q in range(3))
        for k in np.nonzero((bi[p] >= -0.5) & (bi[p] <= 1.5))[0]:
            d, L, b = maps["delta"][k], LD(maps["limb"][k]), int(maps["region"][k])
            be = d * 1000. / C
            S = np.sqrt((1 + be) / (1 - be))
            f = -1 * (1 - S)
            if d == 0.0:
                o = np.minimum(j, n_eff - 2)
                ok = np.ones(n_eff, bool)
                w = wr = (j - o).astype(LD)
            else:
                first = np.ceil(np.arange(n_eff) * (1 + f) + f * wave[0] / step)
                o = np.searchsorted(first, j, side="right") - 1
                ok = (o >= 0) & (o <= n_eff - 2)
                o = np.clip(o, 0, n_eff - 2)
                l0, dl = lam[o].astype(LD), lam[o + 1].astype(LD) - lam[o]
                w = ((lam - l0) - l0 * LD(f)) / (LD(S) * dl)
                wr = (lam - (lam[o] + (-1 * lam[o] * (1 - S))).astype(LD)) / (LD(S) * dl)
            typ = 0 if bi[p, k] == 0 else 1
            ratio = LD(1.0) if typ == 0 else LD(1.0 + maps["lb"][k])
            sed = "fac_sed" if typ else "spot_sed"
            cube = ROWS[2 + typ]
            I = ratio * x[sed][:n_eff]
            h = {"q_sed": (gF + gT, abs(gF) + abs(gT)), "q_norm": (gB - I * gF, abs(gB) + abs(I * gF)),
                 cube: (-gB - I * gT, abs(gB) + abs(I * gT))}
            glimb = glm = gdel = gdm = 0
            slope = -lam * LD(1000. / C) / (LD(S) ** 3 * (1 - LD(be)) ** 2) / (lam[o + 1].astype(LD) - lam[o])
            last = (d == 0.0) & (j == n_eff - 1)       # a cell at rest has no interval there
            for name, (hv, hm) in h.items():
                i = np.nonzero(ok & (hm != 0))[0]
                put(name, (b, o[i]), (L * (1 - wr) * hv)[i], abs(L) * hm[i])
                put(name, (b, o[i] + 1), (L * wr * hv)[i], abs(L) * hm[i])
                a, e = x[name][b, o].astype(LD), x[name][b, o + 1].astype(LD) - x[name][b, o]
                glimb += ((a + w * e) * hv * ok).sum()
                glm += ((abs(a) + abs(e)) * hm * ok).sum()
                gdel += (e * slope * hv * (ok & ~last)).sum() * L
                gdm += (abs(e * slope) * hm * (ok & ~last)).sum() * abs(L)
            put("limb", k, glimb, glm)
            put("delta", k, gdel, gdm)
            q, a = (x[r][b, o] + w * (x[r][b, o + 1].astype(LD) - x[r][b, o]) for r in ("q_norm", cube))
            m = abs(x["q_norm"][b, o]) + abs(x["q_norm"][b, o + 1]), abs(x[cube][b, o]) + abs(x[cube][b, o + 1])
            i = np.nonzero(ok)[0]
            put(sed, i, (-ratio * L * (q * gF + a * gT))[i], (abs(ratio * L) * (m[0] * abs(gF) + m[1] * abs(gT)))[i])
    return out, mag, cnt


def _inputs(rng, n, n_mu, grid, maps, n_phase=2):
    gm = grid * grid
    vis = np.nonzero(maps["limb"] > -998)[0]
    bi = np.full((n_phase, gm), -9999.0)
    bi[0, vis[::2]], bi[0, vis[1::4]] = 0.0, 1.0
    if n_phase > 1:
        bi[1, vis[::5]] = 1.0
    temp = np.where(bi == 0.0, 5115.0, np.where(bi == 1.0, 5900.0, -9999.0))
    x = {k: 1.0 + 0.3 * rng.uniform(-1, 1, (n_mu, n)) for k in ROWS}
    x["spot_sed"], x["fac_sed"] = 0.3 + 0.1 * np.arange(n) / n, 1.0 + 0.1 * np.arange(n) / n
    return bi, temp, x


# a cell of 1180 km/s crosses an integer position every tile of 256 pixels, one of 3000 km/s leaves the ranges
@pytest.mark.parametrize("vsini", [1300.0, 2500.0, 3500.0])
def test_cells_that_cross_several_integers_in_a_tile(ctx, vsini):
    """Every cell once at every pixel.  The positions are those of the forward; 1e-9 of an entry's
    magnitudes covers the rounding of l' (2 ulp(lambda) / step = 4e-10 of a weight)."""
    rng = np.random.default_rng(int(vsini))
    n, n_eff, n_mu, grid, step = 8000, 7990, 4, 12, 0.01
    wave = 5000.0 + step * np.arange(n)
    maps = _maps(grid, vsini, n_mu)
    bi, temp, x = _inputs(rng, n, n_mu, grid, maps)
    g = rng.standard_normal((3, 2, n))
    got = ctx.phase_integrate_adjoint(wave, n_eff, grid, temp, bi, maps, x, step, Activity(5778, 663, 250, 20, 0), *g)
    ref, mag, _ = _reference(wave, n_eff, bi, maps, x, step, g)
    for k in ref:
        assert np.all(np.abs(got[k] - ref[k]) <= 1e-9 * mag[k] + 1e-300), k


# rotators of a few to 400 km/s (beyond 290 km/s the residues of l' are summed cell by cell), a grid
# across 4096 A, limb factors over twelve orders of magnitude and beyond FP32's range
@pytest.mark.parametrize("lambda0,vsini,grid,limb", [(5000.0, 60.0, 40, "disk"), (4094.0, 9.0, 24, "disk"),
                                                     (6000.0, 4.0, 13, "wide"), (5000.0, 400.0, 16, "disk"),
                                                     (4090.0, 30.0, 20, "huge")])
def test_entries_carry_the_rounding_of_single_cells(ctx, lambda0, vsini, grid, limb):
    """Gradients that reach a few output pixels only, so that an entry of the rows is the sum over the
    cells of one offset.  A cell's term takes at most 16 roundings and the cells' sum one each: (16 +
    cells) u of the entry's magnitudes.  The limb and velocity gradients sum 6 tiles' pixels in 13
    steps each, over at most 6 shares: (16 + 13 + 12) u."""
    rng = np.random.default_rng(grid)
    n, n_eff, n_mu, step = 1400, 1390, 4, 0.01
    wave = lambda0 + step * np.arange(n)
    maps = _maps(grid, vsini, n_mu)
    vis = maps["limb"] > -998
    if limb == "wide":
        maps["limb"] = np.where(vis, maps["limb"] * 10.0 ** rng.uniform(-12, 0, vis.size), maps["limb"])
    if limb == "huge":
        maps["limb"] = np.where(vis, maps["limb"] * 1e60, maps["limb"])
    bi, temp, x = _inputs(rng, n, n_mu, grid, maps)
    g = np.zeros((3, 2, n))
    at = np.r_[0, 247, 248, 256, 700, 1023, n_eff - 1, rng.integers(0, n_eff, 8)]
    g[:, :, at] = rng.standard_normal((3, 2, at.size))
    got = ctx.phase_integrate_adjoint(wave, n_eff, grid, temp, bi, maps, x, step, Activity(5778, 663, 250, 20, 0), *g)
    ref, mag, cnt = _reference(wave, n_eff, bi, maps, x, step, g)
    u = 2.0 ** -53
    for k in ref:
        bound = (41 if k in ("limb", "delta") else 16 + cnt[k]) * u * mag[k]
        bad = np.abs(got[k] - ref[k]) > bound
        assert not bad.any(), (k, np.argwhere(bad)[:3], float(np.max(np.abs(got[k] - ref[k])[bad] / mag[k][bad]) / u))


@pytest.mark.parametrize("lambda0,vsini", [(5000.0, 2.0), (6000.0, 20.0), (4500.0, 200.0)])
def test_rounding_of_shifted_wavelengths_near_halves(ctx, lambda0, vsini):
    """The row gradients at every pixel: among some million (cell, pixel) pairs there are shifted
    wavelengths within 2^-21 of half an ulp, which have to be rounded as the forward rounds them (bound
    as above)."""
    rng = np.random.default_rng(3)
    n, n_eff, n_mu, grid, step = 1400, 1390, 4, 60, 0.01
    wave = lambda0 + step * np.arange(n)
    maps = _maps(grid, vsini, n_mu)
    bi, temp, x = _inputs(rng, n, n_mu, grid, maps, 1)
    g = rng.standard_normal((3, 1, n))
    got = ctx.phase_integrate_adjoint(wave, n_eff, grid, temp, bi, maps, x, step, Activity(5778, 663, 250, 20, 0), *g)
    ref, mag, cnt = _reference(wave, n_eff, bi, maps, x, step, g)
    for k in ROWS:
        bad = np.abs(got[k] - ref[k]) > (16 + cnt[k]) * 2.0 ** -53 * mag[k]
        assert not bad.any(), (k, int(bad.sum()), np.argwhere(bad)[:3])


@pytest.mark.parametrize("grid,n,n_phase,n_mu", [(1500, 200, 30, 1), (3000, 8400, 1, 1)])
def test_scratch_of_large_maps(grid, n, n_phase, n_mu):
    """Maps of millions of cells, a few of them active: the phases in groups that fit the scratch, or
    fewer shares of the pixels, with the gradients of per-cell sums (bounds as above, and one addition
    per phase); the workspace stays below 5.5 GB (over 6 for all phases and shares at a time)."""
    torch = pytest.importorskip("torch")
    from soap_gpu_gb300.api import Context
    rng = np.random.default_rng(grid)
    gm, step, n_eff = grid * grid, 0.01, n - 3
    wave = 5000.0 + step * np.arange(n)
    at = np.sort(rng.choice(gm, 40, replace=False))
    maps = dict(delta=np.full(gm, -999.0), limb=np.full(gm, -999.0), lb=np.zeros(gm), region=np.zeros(gm, np.int32))
    maps["delta"][at], maps["limb"][at] = rng.uniform(-3.0, 3.0, 40), rng.uniform(0.3, 1.0, 40)
    maps["lb"][at] = rng.uniform(-0.1, 0.2, 40)
    bi = np.full((n_phase, gm), -9999.0)
    for p in range(n_phase):
        on = rng.choice(at, 6, replace=False)
        bi[p, on[:3]], bi[p, on[3:]] = 0.0, 1.0
    temp = np.where(bi == 0.0, 5115.0, np.where(bi == 1.0, 5900.0, -9999.0))
    x = {k: 1.0 + 0.3 * rng.uniform(-1, 1, (n_mu, n)) for k in ROWS}
    x["spot_sed"], x["fac_sed"] = 0.3 + 0.1 * np.arange(n) / n, 1.0 + 0.1 * np.arange(n) / n
    g = rng.standard_normal((3, n_phase, n))
    dev = lambda a: torch.as_tensor(a, device="cuda:0")
    args = [dev(wave), n_eff, grid, dev(temp), dev(bi), {k: dev(v) for k, v in maps.items()}, {k: dev(v) for k, v in x.items()},
            step, Activity(5778, 663, 250, 20, 0), *(dev(v) for v in g)]
    torch.cuda.synchronize()
    with Context(0) as ctx:
        free = torch.cuda.mem_get_info()[0]
        got = {k: v.cpu().numpy() for k, v in ctx.phase_integrate_adjoint(*args).items()}
        assert free - torch.cuda.mem_get_info()[0] < 5.5e9
    ref, mag, cnt = _reference(wave, n_eff, bi, maps, x, step, g)
    for k in ref:
        bound = (41 + n_phase + (n >> 8) if k in ("limb", "delta") else 16 + n_phase + cnt[k]) * 2.0 ** -53 * mag[k]
        assert np.all(np.abs(got[k] - ref[k]) <= bound), k


def test_gradients_that_are_not_finite_stay_at_their_pixels(ctx):
    """Cells at rest copy their source: a NaN or infinite gradient of pixel j reaches source j of the
    rows that enter that output and no other, for a row of cells and for one evaluated by itself (Planck
    ratio)."""
    n, n_mu, grid, step, at = 700, 2, 4, 0.01, 300
    wave = 5000.0 + step * np.arange(n)
    gm = grid * grid
    maps = dict(delta=np.zeros(gm), limb=np.linspace(0.4, 1.0, gm), lb=np.full(gm, 0.1), region=np.zeros(gm, np.int32))
    rng = np.random.default_rng(1)
    x = {k: 1.0 + 0.3 * rng.uniform(-1, 1, (n_mu, n)) for k in ROWS}
    x["spot_sed"], x["fac_sed"] = 0.3 + 0.1 * np.arange(n) / n, 1.0 + 0.1 * np.arange(n) / n
    bi = np.tile(np.where(np.arange(gm) < 8, 0.0, 1.0), (1, 1))
    for t_spot in (5115.0, 5115.5):
        temp = np.where(bi == 0.0, t_spot, 5900.0)
        for q, hit in ((0, ("q_sed", "q_norm")), (1, ("q_norm", "spot_norm", "fac_norm")),
                       (2, ("q_sed", "spot_norm", "fac_norm"))):
            for bad in (np.nan, np.inf):
                g = rng.standard_normal((3, 1, n))
                g[q, 0, at] = bad
                got = ctx.phase_integrate_adjoint(wave, n, grid, temp, bi, maps, x, step,
                                                  Activity(5778, 663, 250, 20, 0), *g)
                for k in ROWS:
                    bad_at = np.argwhere(~np.isfinite(got[k])).tolist()
                    assert bad_at == ([[0, at]] if k in hit else []), (k, q, bad_at)
