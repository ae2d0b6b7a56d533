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
