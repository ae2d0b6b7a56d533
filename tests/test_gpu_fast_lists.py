"""The phase lists built from the region boxes (sorted per phase by runs of 64 and merges) against
those built from the maps by the cell order: the deficits are the same bits.  Phases of no cell, a few
cells, and one to several thousand.  And the exact extremum that the FP32 convolution's refinement finds,
several pixels per lane, at the remainders of its 1024-pixel blocks."""
import ctypes

import numpy as np
import pytest

from soap_gpu_gb300 import synth
from soap_gpu_gb300._lib import Star

from _cases import activity, cubes

pytestmark = pytest.mark.gpu


# (grid, sizes of the two regions): lists of tens of cells up to some 8000 of a 300 x 300 grid
@pytest.mark.parametrize("grid,sizes", [(17, (0.1, 0.08)), (60, (0.12, 0.3)), (150, (0.35, 0.2)), (300, (0.28, 0.1))])
def test_box_lists_equal_map_lists(ctx, grid, sizes):
    case = synth.small_case(seed=11, grid=grid, n=2100, n_phase=5, n_mu=6)
    case.regions = np.array([[20.0, 10.0, sizes[0], 0.0], [100.0, -15.0, sizes[1], 1.0]])
    inp = synth.generate(case)
    n_eff = 2048
    maps = ctx.disk_maps(case.grid, case.period, case.w_ratio, case.incl, case.radius_km, case.u1, case.u2,
                         inp.mu_boundary, inp.lb)
    cb = cubes(inp)
    cb["spot_sed"] = inp.spot_sed[0]
    cb["fac_sed"] = inp.fac_sed[0]
    act = activity(case)
    regions = [case.regions for _ in case.phases]
    star = Star(case.grid, case.period, case.w_ratio, case.incl, case.radius_km, case.u1, case.u2,
                (ctypes.c_double * 4)(*inp.lb))
    q_norm = ctx.quiet_disk("fast32", inp.wave, inp.q_norm, n_eff, maps, case.grid, case.step)
    q_sed = ctx.quiet_disk("fast32", inp.wave, inp.q_sed, n_eff, maps, case.grid, case.step)
    low, raw = ctx.phase_pipeline("fast32", inp.wave, n_eff, star, maps, cb, case.step, act, case.phases, regions,
                                  q_sed, q_norm, case.sigma_v, conv_step=case.step, want_raw=True)
    temp, bi = ctx.phase_maps(case.grid, case.incl, case.phases, regions, act)
    assert np.sum((bi >= -0.5) & (bi <= 1.5)) > 0
    flux, bconv, tot = ctx.phase_integrate("fast32", inp.wave, n_eff, case.grid, temp, bi, maps, cb, case.step, act)
    for k, spec in enumerate((tot, flux, bconv)):
        assert np.array_equal(raw[:, k], spec[:, :n_eff])


@pytest.mark.parametrize("n", [1100, 2047, 2049, 5123])
def test_refined_minimum_is_exact(ctx, n):
    """The minimum of base - spec in FP64, with plateaus that put many pixels within the FP32 bounds."""
    rng = np.random.default_rng(n)
    step = 0.01
    wave = 5000.0 + step * np.arange(n)
    x = np.arange(n)
    base = 1.7 - 0.6 * np.exp(-((x % 97) - 40.0) ** 2 / 18.0) + 1e-9 * rng.uniform(-1, 1, n)
    spec = (1e-3 * rng.uniform(0, 1, (7, n))).astype(np.float32).astype(np.float64)
    spec[3] = 0.0
    spec[4, n - 1] = 1.25   # the last pixel
    sigma_v = 299792458.0 / 115000.0 / (2 * np.sqrt(2 * np.log(2)))
    _, mm = ctx.lower_resolution("fast32", wave, spec, n // 512 * 512, sigma_v, base=base, step_mult=step,
                                 step_exp=step)
    assert np.array_equal(np.asarray(mm)[:, 0], (base[None, :] - spec).min(1))


@pytest.mark.parametrize("n_spec,n_v", [(1, 21), (5, 81), (40, 161)])
def test_ccf_normalise(ctx, n_spec, n_v):
    """The normalised CCFs of raw sums are soapgb_ccf's own, bit for bit."""
    torch = pytest.importorskip("torch")
    from soap_gpu_gb300.torch_ops import Ops
    rng = np.random.default_rng(n_v)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda:0")
    step, n, mask_step = 0.01, 6000, 0.01
    wave = 5000.0 + step * np.arange(n)
    lines = np.sort(rng.uniform(5003.0, 5057.0, 40))
    args = (dev(np.linspace(-20000.0, 20000.0, n_v)), dev(lines), dev(rng.uniform(0.1, 1.0, 40)), dev(wave), step,
            dev(1.0 - 0.5 * rng.uniform(0, 1, (n_spec, n))))
    kw = dict(wave_extend=100.0, mask_step=mask_step, index_old=int(100.0 / step))
    o = Ops(ctx)
    raw = o.ccf("plain64", *args, normalise=False, **kw)
    assert torch.equal(o.ccf_normalise(raw), o.ccf("plain64", *args, normalise=True, **kw))
