"""The plain form's kernels at the sizes and values where their paths change.

Tolerance of the forward stages: 1e-12 of the spectrum's scale against the oracle, the plain
form's contract (the kernels keep the oracle's operations and their order; exp differs by less
than 1 ulp)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
C = 299792458.0


def _sigma_v(reso):
    return C / reso / (2 * np.sqrt(2 * np.log(2)))


def _spectra(kind, n, n_eff, n_spec, rng):
    x = np.arange(n)
    y = 1.0 - 0.6 * np.exp(-((x % 97) - 40.0) ** 2 / 18.0)
    y = y[None, :] * (1 + 0.01 * rng.uniform(-1, 1, (n_spec, n)))
    if kind == "unit":     # continuum exactly 1 between isolated lines, empty towards the ends
        y = 1.0 - 0.6 * np.exp(-((x % 311) - 150.0) ** 2 / 18.0) * (np.abs((x % 311) - 150) < 30)
        y = np.tile(y, (n_spec, 1)) - 1e-3 * np.arange(n_spec)[:, None] * (y < 1)
    if kind == "disk":
        y = 1500.0 * y
        y[:, n_eff:] = 0.0
    return y


@pytest.mark.parametrize("kind", ["disk", "unit", "hole"])
@pytest.mark.parametrize("n,n_spec,reso", [(700, 1, 115000.0), (1537, 3, 115000.0), (4100, 40, 60000.0),
                                           (9000, 2, 7000.0), (20000, 1, 1500.0)])
def test_plain_convolution(ctx, kind, n, n_spec, reso):
    """Tiles of 128 pixels and their remainders, one and many spectra, reaches from a few pixels
    to more than the tiled form's shared memory holds, windows that leave the short form."""
    rng = np.random.default_rng(n)
    step = 0.01
    wave = 5000.0 + step * np.arange(n)
    n_eff = n // 512 * 512
    sv = _sigma_v(reso)
    a = _spectra("disk" if kind == "hole" else kind, n, n_eff, n_spec, rng)
    wid = oracle.conv_halfwidth(wave, sv, 50.0)
    if 2 * wid + 2 >= n:
        pytest.skip("the window does not fit the spectrum")
    base = a[0] * 1.5
    hole = n_eff // 2 + 3
    spec = base[None, :] - a
    if kind == "hole":
        spec[-1, hole] = np.nan
    got, mm = ctx.lower_resolution("plain64", wave, spec, n_eff, sv, base=base, step_mult=step, step_exp=step)
    for s in range(n_spec):
        ref, _, ext = oracle.lower_resolution(wave, base - np.where(np.isnan(spec[s]), 0.0, spec[s]), n_eff, sv,
                                              step_mult=step, step_exp=step)
        if kind == "hole" and s == n_spec - 1:
            i = np.arange(n_eff)
            reached = (i > wid) & (i + wid < n - 1) & (i - wid <= hole) & (hole <= i + wid - 2)
            assert np.array_equal(np.isnan(got[s]), reached)
            continue
        assert np.allclose(mm[s], ext, rtol=1e-12, atol=0)
        assert np.max(np.abs(got[s] - ref)) <= 1e-12 * np.max(np.abs(ref))


def _disk(grid, vsini, lambda0, n_mu):
    lb = (0.2, -0.4, 0.3, -0.1)
    period = 2 * np.pi * 696000.0 / (vsini * 86400.0)
    return oracle.disk_maps(grid, period, -0.18, 80.0, 696000.0, 0.3, 0.3, np.linspace(0.95, 0.15, n_mu - 1), lb)


def _cube(n, n_mu, rng, kind):
    x = np.arange(n)
    y = 1.0 - 0.5 * np.exp(-((x % 61) - 30.0) ** 2 / 20.0)
    y = y[None, :] * (1 + 1e-3 * rng.uniform(-1, 1, (n_mu, n)))
    if kind == "flat":        # stretches of equal values, negative and positive zeros
        y[:, n // 4:n // 2] = 1.0
        y[:, n // 2:n // 2 + 40] = np.where(x[:40] % 3 == 0, -0.0, 0.0)
    if kind == "wild":        # infinities, NaN, tiny and huge neighbours
        for k, v in enumerate((np.inf, np.nan, -np.inf, 1e-310, 1e300, 2.0 ** -1000)):
            y[k % n_mu, n // 3 + 60 * k] = v
    return y


# grids inside a binade and across one (4096 A), an uneven one, ends of tiles of 62 pixels, one
# pixel count below a tile, slow and fast rotators (above 290 km/s the integer form has no range)
@pytest.mark.parametrize("lambda0,step,n,vsini,uneven,kind", [
    (5000.0, 0.01, 62 * 9 + 1, 4.0, False, "lines"), (5000.0, 0.005, 1300, 4.0, False, "flat"),
    (4092.0, 0.01, 1024, 10.0, False, "lines"), (3800.0, 0.01, 2050, 40.0, False, "wild"),
    (5000.0, 0.01, 1100, 400.0, False, "lines"), (5000.0, 0.01, 1100, 5.0, True, "lines"),
    (6000.0, 0.02, 41, 0.5, False, "lines"), (5000.0, 0.0078125, 700, 3.0, False, "lines")])
def test_plain_sums_are_the_sequential_ones(ctx, lambda0, step, n, vsini, uneven, kind):
    """Quiet disk and per-phase integration equal the oracle's loops bit for bit."""
    rng = np.random.default_rng(n)
    grid, n_mu = 14, 4
    n_eff = n if n < 62 else n - 7
    wave = lambda0 + step * np.arange(n)
    if uneven:
        wave = wave + step * 0.2 * np.sin(np.arange(n) / 50.0)
    maps = _disk(grid, vsini, lambda0, n_mu)
    vis = np.nonzero(maps["limb"] > -998)[0]
    cube = [_cube(n, n_mu, rng, kind) for _ in range(4)]
    with np.errstate(all="ignore"):
        ref = oracle.quiet_disk(wave, cube[0], n_eff, maps, grid, step)
        got = ctx.quiet_disk("plain64", wave, cube[0], n_eff, maps, grid, step)
        assert np.array_equal(got, ref, equal_nan=True)
        bi = np.full(grid * grid, -9999.0)
        bi[vis[::3]], bi[vis[1::3]] = 0.0, 1.0
        temp = np.where(bi == 0.0, 5115.0, np.where(bi == 1.0, 5900.0, -9999.0))
        sed = 0.3 + 0.1 * np.arange(n) / n, 1.0 + 0.1 * np.arange(n) / n
        from soap_gpu_gb300._lib import Activity
        names = ("q_norm", "q_sed", "spot_norm", "fac_norm")
        out = ctx.phase_integrate("plain64", wave, n_eff, grid, np.stack([temp, temp]), np.stack([bi, -9999.0 + 0 * bi]),
                                  maps, dict(zip(names, cube), spot_sed=sed[0], fac_sed=sed[1]), step,
                                  Activity(5778, 663, 250, 20, 0))
        want = oracle.phase_integrate(wave, n_eff, grid, temp, bi, maps, *cube, sed[0], sed[1], step)
    for o, r in zip(out, want):
        assert np.array_equal(o[0], r, equal_nan=True)
        assert not o[1].any()


# the adjoint's ranges of equal offsets: tiles of 31 and 256 pixels and their ends, cells at rest
# (even grids have a column of them), more than 64 offsets in a row, Planck ratios, uneven grids
@pytest.mark.parametrize("lambda0,step,n,vsini,grid,uneven,solar", [
    (5000.0, 0.01, 1300, 4.0, 14, False, False), (5000.0, 0.005, 249, 9.0, 13, False, False),
    (4092.0, 0.01, 1030, 10.0, 14, False, True), (6000.0, 0.01, 900, 60.0, 21, False, False),
    (5000.0, 0.01, 700, 5.0, 14, True, False), (5000.0, 0.01, 20, 2.0, 8, False, False)])
def test_adjoint_is_the_transpose(ctx, lambda0, step, n, vsini, grid, uneven, solar):
    """<W, J V> = <J^T W, V> over the cubes, the continuum rows and the limb map, in which the
    integration is linear.  Bound: the forward rounds its interpolation weights to 2 ulp(lambda) /
    step, at most 4e-10 here, so 1e-9 |W| |J V|.  The velocity gradient against a central difference
    in a common factor of the velocities, 1e-4 (relative step 1e-6, as in the parity of vsini)."""
    from soap_gpu_gb300._lib import Activity
    rng = np.random.default_rng(n)
    n_mu, n_eff = 4, n if n < 256 else n - 5
    wave = lambda0 + step * np.arange(n)
    if uneven:
        wave = wave + step * 0.2 * np.sin(np.arange(n) / 50.0)
    maps = _disk(grid, vsini, lambda0, n_mu)
    vis = np.nonzero(maps["limb"] > -998)[0]
    gm = grid * grid
    bi = np.full((2, gm), -9999.0)
    bi[0, vis[::2]], bi[0, vis[1::4]], bi[1, vis[::5]] = 0.0, 1.0, 1.0
    temp = np.where(bi == 0.0, 5115.0, np.where(bi == 1.0, 5900.0 + np.arange(gm) % 40, -9999.0))
    temp[0, vis[0]] = 5115.5                      # a spot whose Planck ratio is not 1
    act = Activity(5778, 663, 250, 20, int(solar))
    names = ("q_norm", "q_sed", "spot_norm", "fac_norm", "spot_sed", "fac_sed")
    x = dict(zip(names, [_cube(n, n_mu, rng, "lines") for _ in range(4)] +
                 [0.3 + 0.1 * np.arange(n) / n, 1.0 + 0.1 * np.arange(n) / n]))
    W = rng.standard_normal((3, 2, n))
    fwd = lambda m, c: np.stack(ctx.phase_integrate("plain64", wave, n_eff, grid, temp, bi, m, c, step, act))
    g = ctx.phase_integrate_adjoint(wave, n_eff, grid, temp, bi, maps, x, step, act, *W)
    close = lambda jv, rhs: abs((W * jv).sum() - rhs) <= 1e-9 * np.linalg.norm(W) * np.linalg.norm(jv)
    V = {k: rng.standard_normal(x[k].shape) for k in names[:4]}
    assert close(fwd(maps, dict(V, spot_sed=x["spot_sed"], fac_sed=x["fac_sed"])),
                 sum((g[k] * V[k]).sum() for k in V))
    S = {k: rng.standard_normal(n) for k in names[4:]}
    zero = {k: np.zeros(n) for k in S}
    assert close(fwd(maps, dict(x, **S)) - fwd(maps, dict(x, **zero)), sum((g[k] * S[k]).sum() for k in S))
    dl = rng.standard_normal(gm)
    assert close(fwd(dict(maps, limb=dl), x), (g["limb"] * dl).sum())
    h = 1e-6
    scaled = [fwd(dict(maps, delta=np.where(maps["limb"] > -998, maps["delta"] * (1 + s), -999.0)), x) for s in (h, -h)]
    jv = (scaled[0] - scaled[1]) / (2 * h)
    rhs = (g["delta"] * np.where(maps["limb"] > -998, maps["delta"], 0.0)).sum()
    assert abs((W * jv).sum() - rhs) <= 1e-4 * np.linalg.norm(W) * np.linalg.norm(jv)


@pytest.mark.parametrize("n,n_spec,reso", [(900, 1, 115000.0), (1537, 30, 60000.0), (9000, 2, 9000.0), (9000, 1, 7000.0)])
def test_resolution_adjoint_is_the_transposed_window(ctx, n, n_spec, reso):
    """The gradient against the transposed taps of the whole reference window in numpy.  Tolerance: at
    most 2 wid = 3000 terms, each with a few roundings, so 3000 x 4 x 1.1e-16 = 1.3e-12 of the sum of
    their magnitudes, which is below f max |g| x 1.01; 1e-11 of that leaves room for the shared factors.
    A NaN gradient reaches the whole window and no other spectrum."""
    rng = np.random.default_rng(n)
    step = 0.01
    wave = 5000.0 + step * np.arange(n)
    n_eff = n // 512 * 512
    sv = _sigma_v(reso)
    wid = oracle.conv_halfwidth(wave, sv, 50.0)
    a = _spectra("disk", n, n_eff, n_spec, rng)
    base = a[0] * 1.5
    spec = base[None, :] - a
    kw = dict(base=base, step_mult=step, step_exp=step)
    g = rng.standard_normal((n_spec, n_eff))
    gs, gb = ctx.lower_resolution_adjoint(wave, spec, n_eff, sv, g, **kw)
    b = sv / C
    sig = -1 * wave[:n_eff] * (1 - np.sqrt((1 + b) / (1 - b)))
    i = np.arange(n_eff)
    inside = (i > wid) & (i + wid < n - 1)
    for s in range(0, n_spec, 13):
        A = base - spec[s]
        _, conv, (mn, mx) = oracle.lower_resolution(wave, A, n_eff, sv, step_mult=step, step_exp=step)
        S = (g[s] * conv).sum()
        gc = -(1 - mn) / mx * g[s]
        gc[np.argmax(np.where(conv != 0, conv, -np.inf))] += S * (1 - mn) / mx ** 2
        ref = np.zeros(n)
        ref[np.argmin(A)] -= S / mx
        for d in range(-wid, wid - 1):
            k = np.where(inside, step * np.exp(-d * d * step * step / (2 * sig * sig)) / (sig * np.sqrt(2 * np.pi)), 0)
            lo, hi = max(0, -d), min(n_eff, n - d)
            ref[lo + d:hi + d] += (k * gc)[lo:hi]
        assert np.max(np.abs(gs[s] - ref)) <= 1e-11 * max(np.abs(gc).max(), abs(S / mx))
    assert np.allclose(gb, -gs.sum(0), rtol=1e-12, atol=1e-12 * np.abs(gs).max())
    mid = n_eff // 2
    g[-1, mid] = np.nan
    m = np.arange(n)
    gs = ctx.lower_resolution_adjoint(wave, spec, n_eff, sv, g, **kw)[0]
    assert np.isnan(gs[-1][(m >= mid - wid) & (m <= mid + wid - 2)]).all()
    assert not np.isnan(gs[:-1]).any()


# fewer and more points than the fit's threads, its bisector arrays in shared memory and in scratch
@pytest.mark.parametrize("n,n_spec,with_err", [(21, 1, False), (161, 5, True), (4001, 2, False)])
def test_fit_and_its_adjoint(ctx, n, n_spec, with_err):
    """The fit against the oracle's (the tolerances of test_gpu_parity: 1e-4 m/s, 1e-9 of the model);
    its adjoint against a central difference of the fitted velocity along a direction (1e-4 of the
    gradient's norm, as in test_gpu_ccf_adjoint)."""
    rng = np.random.default_rng(n)
    x = np.linspace(-20000.0, 20000.0, n)
    sig = rng.uniform(3000, 4500, (n_spec, 1))
    x0 = rng.uniform(-2000, 2000, (n_spec, 1))
    y = 1.05 - rng.uniform(0.1, 0.4, (n_spec, 1)) * np.exp(-(x - x0) ** 2 / (2 * sig * sig)) + 1e-4 * np.sin(x / 777.0)
    err = rng.uniform(0.5, 2.0, (n_spec, n)) if with_err else None
    got = ctx.gauss_bis(x, y, err)
    for s in range(n_spec):
        ref = oracle.gauss_bis(x, y[s], None if err is None else err[s])
        assert got["iters"][s] >= 0 and ref["iters"] >= 0
        assert np.max(np.abs(got["par"][s, 2:] - ref["par"][2:])) < 1e-4
        assert np.max(np.abs(got["bis"][s] - ref["bis"])) < 1e-4
        assert np.max(np.abs(got["model"][s] - ref["model"])) < 1e-9
    gp = np.zeros((n_spec, 5))
    gp[:, 3] = 1.0
    g = ctx.gauss_fit_adjoint(x, y, got["model"], got["par"], gp, err)
    v = rng.standard_normal(y.shape)
    h = 1e-4 / np.sqrt(n)
    d = (ctx.gauss_bis(x, y + h * v, err)["par"][:, 3] - ctx.gauss_bis(x, y - h * v, err)["par"][:, 3]) / (2 * h)
    assert np.all(np.abs(d - (g * v).sum(1)) <= 1e-4 * np.linalg.norm(g, axis=1) * np.linalg.norm(v, axis=1))


@pytest.mark.parametrize("n,n_phase,kind", [(62 * 608, 1, "lines"), (62 * 608 + 1, 2, "flat"), (62 * 66 + 5, 14, "lines"),
                                            (62 * 66, 14, "wild"), (62 * 66 - 1, 14, "flat")])
def test_plain_sums_of_many_tiles(ctx, n, n_phase, kind):
    """As above at the tile counts where the quiet sum goes from 16 warps per tile to two and the
    integration's products from the FP64 pipe to the integer ones; continuum rows and limb factors with
    zero, negative, tiny and non-finite values."""
    rng = np.random.default_rng(n)
    grid, n_mu, step, n_eff = 8, 3, 0.01, n - 3
    wave = 4090.0 + step * np.arange(n)   # across a binade
    maps = dict(_disk(grid, 9.0, 4090.0, n_mu))
    vis = np.nonzero(maps["limb"] > -998)[0]
    maps["limb"] = maps["limb"].copy()
    maps["limb"][vis[[1, 4, 7]]] = 0.0, -0.3, 1e-200
    cube = [_cube(n, n_mu, rng, kind) for _ in range(4)]
    sed = [0.3 + 0.1 * np.arange(n) / n, 1.0 + 0.1 * np.arange(n) / n]
    sed[0][[70, 300]] = 0.0, -0.2
    sed[1][[71, 301, 500]] = np.nan, np.inf, 1e-100
    bi = np.full(grid * grid, -9999.0)
    bi[vis[::2]], bi[vis[1::2]] = 0.0, 1.0
    temp = np.where(bi == 0.0, 5115.0, np.where(bi == 1.0, 5900.0, -9999.0))
    from soap_gpu_gb300._lib import Activity
    names = ("q_norm", "q_sed", "spot_norm", "fac_norm")
    with np.errstate(all="ignore"):
        ref = oracle.quiet_disk(wave, cube[0], n_eff, maps, grid, step)
        got = ctx.quiet_disk("plain64", wave, cube[0], n_eff, maps, grid, step)
        assert np.array_equal(got, ref, equal_nan=True)
        out = ctx.phase_integrate("plain64", wave, n_eff, grid, np.tile(temp, (n_phase, 1)), np.tile(bi, (n_phase, 1)),
                                  maps, dict(zip(names, cube), spot_sed=sed[0], fac_sed=sed[1]), step,
                                  Activity(5778, 663, 250, 20, 0))
        want = oracle.phase_integrate(wave, n_eff, grid, temp, bi, maps, *cube, *sed, step)
    for o, r in zip(out, want):
        for p in range(n_phase):
            assert np.array_equal(o[p], r, equal_nan=True)


@pytest.mark.parametrize("n,n_spec,top", [(3000, 5, 1e4), (1500, 1, 1e9), (2600, 2, 3.0)])
def test_plain_convolution_of_small_sums(ctx, n, n_spec, top):
    """Spectra whose terms 1 - A pass through zero, slowly and steeply, and stretches where they cancel:
    sums far below their terms."""
    rng = np.random.default_rng(n)
    step, sv = 0.01, _sigma_v(115000.0)
    wave = 5000.0 + step * np.arange(n)
    n_eff = n // 512 * 512
    x = np.arange(n)
    a = 1.0 + top * np.tanh((x - n // 2) / (1.0 + 40.0 * np.arange(n_spec)[:, None]))
    a[:, n // 4:n // 4 + 60] = 1.0 + 1e-9 * rng.uniform(-1, 1, (n_spec, 60))
    a[:, n // 3:n // 3 + 200] = 1.0 + top * (1.0 - 2.0 * (x[:200] % 2)) + 1e-7
    base = 2.0 + top * rng.uniform(0, 1, n)
    got, mm = ctx.lower_resolution("plain64", wave, base[None, :] - a, n_eff, sv, base=base, step_mult=step, step_exp=step)
    for s in range(n_spec):
        ref, _, ext = oracle.lower_resolution(wave, base - (base - a[s]), n_eff, sv, step_mult=step, step_exp=step)
        assert np.max(np.abs(got[s] - ref)) <= 1e-12 * np.max(np.abs(ref))
        assert np.allclose(mm[s], ext, rtol=1e-12, atol=0)


def _transposed_taps(wave, A, conv, mn, mx, g, n_eff, sv, wid, step):
    """The resolution gradient d out / d A against g over the whole reference window."""
    n = wave.size
    b = sv / C
    sig = -1 * wave[:n_eff] * (1 - np.sqrt((1 + b) / (1 - b)))
    i = np.arange(n_eff)
    inside = (i > wid) & (i + wid < n - 1)
    S = (g * conv).sum()
    gc = -(1 - mn) / mx * g
    gc[np.argmax(np.where(conv != 0, conv, -np.inf))] += S * (1 - mn) / mx ** 2
    ref = np.zeros(n)
    ref[np.argmin(A)] += S / mx
    for d in range(-wid, wid - 1):
        k = np.where(inside, step * np.exp(-d * d * step * step / (2 * sig * sig)) / (sig * np.sqrt(2 * np.pi)), 0)
        lo, hi = max(0, -d), min(n_eff, n - d)
        ref[lo + d:hi + d] -= (k * gc)[lo:hi]
    return ref, max(np.abs(gc).max(), abs(S / mx))


# the window is m - i = -wid .. wid - 2: without the central tap for wid = 1, without the upper one for wid = 2
@pytest.mark.parametrize("wid,window,step", [(1, 0.55, 0.01), (2, 1.1, 0.01), (3, 1.65, 0.01), (1, 50.0, 1.0)])
def test_resolution_of_narrow_windows(ctx, wid, window, step):
    """Forward and gradient of half widths of one to three pixels, with a base and without, against the
    oracle and the transposed taps in numpy (tolerances of the two tests above)."""
    n, n_eff, n_spec = 1100, 1024, 3
    rng = np.random.default_rng(wid)
    wave = 5000.0 + step * np.arange(n)
    sv = _sigma_v(115000.0)
    assert oracle.conv_halfwidth(wave, sv, window) == wid
    a = _spectra("disk", n, n_eff, n_spec, rng)
    base = a[0] * 1.5
    g = rng.standard_normal((n_spec, n_eff))
    kw = dict(window=window, step_mult=step, step_exp=step)
    for b in (base, None):
        spec = a if b is None else b[None, :] - a
        got, mm = ctx.lower_resolution("plain64", wave, spec, n_eff, sv, base=b, **kw)
        gs = ctx.lower_resolution_adjoint(wave, spec, n_eff, sv, g, base=b, **kw)[0]
        for s in range(n_spec):
            A = spec[s] if b is None else b - spec[s]
            ref, conv, (mn, mx) = oracle.lower_resolution(wave, A, n_eff, sv, window, step, step)
            assert np.allclose(mm[s], (mn, mx), rtol=1e-12, atol=0)
            assert np.max(np.abs(got[s] - ref)) <= 1e-12 * np.max(np.abs(ref))
            want, scale = _transposed_taps(wave, A, conv, mn, mx, g[s].copy(), n_eff, sv, wid, step)
            assert np.max(np.abs((gs[s] if b is None else -gs[s]) - want)) <= 1e-11 * scale


@pytest.mark.parametrize("factor", [2.5, 3.5])
def test_resolution_of_wavelengths_that_do_not_ascend(ctx, factor):
    """Pixels in the middle whose Gaussian is wider than at both ends of the grid: their taps reach
    further than the ends', also into blocks of pixels that the ends' reach from them does not touch
    (tolerances as above)."""
    n, n_eff, n_spec, step = 1900, 1536, 2, 0.01
    wide = [700, 740, 741, 1310]
    rng = np.random.default_rng(7)
    wave = 5000.0 + step * np.arange(n)
    wave[wide] *= factor
    sv = _sigma_v(115000.0)
    wid = oracle.conv_halfwidth(wave, sv, 50.0)
    a = _spectra("disk", n, n_eff, n_spec, rng)
    g = rng.standard_normal((n_spec, n_eff))
    g[:, wide] *= 1e6                # their far taps stand out
    kw = dict(step_mult=step, step_exp=step)
    got, mm = ctx.lower_resolution("plain64", wave, a, n_eff, sv, **kw)
    gs = ctx.lower_resolution_adjoint(wave, a, n_eff, sv, g, **kw)[0]
    for s in range(n_spec):
        ref, conv, (mn, mx) = oracle.lower_resolution(wave, a[s], n_eff, sv, **kw)
        assert np.max(np.abs(got[s] - ref)) <= 1e-12 * np.max(np.abs(ref))
        want, scale = _transposed_taps(wave, a[s], conv, mn, mx, g[s].copy(), n_eff, sv, wid, step)
        assert np.max(np.abs(gs[s] - want)) <= 1e-11 * scale


def _power_of_two_hits(rng, count):
    """(delta, lambda) whose shifted wavelength is 2^12 when l u is rounded to whole ulps of lambda, and
    half an ulp below in the reference's operations, which round finer there."""
    hits = []
    while len(hits) < count:
        d = -rng.uniform(1.0, 60.0)            # l' below l: the cell's u is positive
        b = d * 1000. / C
        u = 1 - np.sqrt((1 + b) / (1 - b))
        l0 = 4096.0 / (1 - u)
        for k in range(-3, 4):
            l = l0 + k * 2.0 ** -40
            t = int(l * 2 ** 40) * int(u * 2 ** 53)               # l u in units of ulp(l) 2^-53
            whole = int(l * 2 ** 40) - ((t + (1 << 52)) >> 53)
            ref = l + (-1.0 * l) * u
            if whole == 2 ** 52 and ref < 4096.0:
                hits.append((d, l))
                break
    return hits


@pytest.mark.parametrize("n", [700, 62 * 608 + 90])
def test_shifted_wavelengths_at_a_power_of_two(ctx, n):
    """Sources whose shifted wavelength comes to exactly 2^12: the sums stay the oracle's, bit for bit
    (the quiet sum and the integration, with few tiles and with many)."""
    from soap_gpu_gb300._lib import Activity
    rng = np.random.default_rng(12)
    step, n_mu, grid, at = 0.01, 2, 2, n // 2
    names = ("q_norm", "q_sed", "spot_norm", "fac_norm")
    for d, l in _power_of_two_hits(rng, 6):
        at -= (at - int(round((l - 4096.0) / step))) % 62 - 5    # early in a tile, whose middle lies above 2^12
        wave = l + step * (np.arange(n) - at)
        maps = dict(delta=np.array([d, -999.0, d, -999.0]), limb=np.array([0.9, -999.0, 0.7, -999.0]),
                    mu=np.array([0.9, -999.0, 0.6, -999.0]), lb=np.array([0.1, -999.0, 0.2, -999.0]),
                    region=np.array([0, 0, 1, 0], np.int32))
        cube = [1.0 + 0.5 * rng.uniform(-1, 1, (n_mu, n)) for _ in range(4)]
        sed = 0.3 + 0.1 * np.arange(n) / n, 1.0 + 0.1 * np.arange(n) / n
        ref = oracle.quiet_disk(wave, cube[0], n, maps, grid, step)
        assert np.array_equal(ctx.quiet_disk("plain64", wave, cube[0], n, maps, grid, step), ref)
        bi = np.array([0.0, -9999.0, 1.0, -9999.0])
        temp = np.array([5115.0, -9999.0, 5900.0, -9999.0])
        want = oracle.phase_integrate(wave, n, grid, temp, bi, maps, *cube, *sed, step)
        for n_phase in (1, 2):
            out = ctx.phase_integrate("plain64", wave, n, grid, np.tile(temp, (n_phase, 1)), np.tile(bi, (n_phase, 1)),
                                      maps, dict(zip(names, cube), spot_sed=sed[0], fac_sed=sed[1]), step,
                                      Activity(5778, 663, 250, 20, 0))
            for o, r in zip(out, want):
                assert all(np.array_equal(v, r) for v in o)


@pytest.mark.parametrize("kind", ["one", "stretch", "lines", "flat", "tiny"])
def test_plain_convolution_with_terms_of_zero(ctx, kind):
    """1 - A exactly zero at one pixel, over a stretch longer than a window, between lines, everywhere
    but at a few pixels, and beside terms of one ulp (tolerance as above; a spectrum of zeros alone
    keeps the sentinel)."""
    n, n_eff, step = 3000, 2560, 0.01
    rng = np.random.default_rng(5)
    wave, sv, x = 5000.0 + step * np.arange(n), _sigma_v(115000.0), np.arange(n)
    a = np.tile(1.0 - 0.5 * np.exp(-((x % 97) - 40.0) ** 2 / 18.0) * (1 + 0.1 * rng.uniform(-1, 1, n)), (3, 1))
    if kind == "one":
        a[:, [700, 1500]] = 1.0
    if kind == "stretch":
        a[:, 900:1400] = 1.0
    if kind == "lines":
        a = _spectra("unit", n, n_eff, 3, rng)
    if kind == "flat":
        a[:] = 1.0
        a[0, [640, 1300]], a[1, 2000] = 0.4, 2.0
    if kind == "tiny":
        a[:] = 1.0 + 2.0 ** -52 * (x % 3 - 1)
        a[1, 1000:1300] = 1.0
    got, mm = ctx.lower_resolution("plain64", wave, a, n_eff, sv, step_mult=step, step_exp=step)
    for s in range(3):
        ref, conv, ext = oracle.lower_resolution(wave, a[s], n_eff, sv, step_mult=step, step_exp=step)
        assert np.allclose(mm[s], ext, rtol=1e-12, atol=0)
        assert np.max(np.abs(got[s] - ref)) <= 1e-12 * np.max(np.abs(ref))
