"""The collapsed quiet disk where its cell order and list change paths: grids of one tile of the
order and of several, their remainders, the largest grid ordered by ranks and the next one, lists
whose slopes lie in shared memory and not; equal slopes; all cells at rest; no visible cell; sizes
whose rows are not 16-byte aligned; two cubes of one disk (the batched form).

Tolerances: test_gpu_parity's of the forms, 2e-10 and 1e-6 of the spectrum's scale."""
import numpy as np
import pytest

import oracle
from _cases import oracle_maps, rel_err, small_inputs

pytestmark = pytest.mark.gpu
TOL = {"fast64": 2e-10, "fast32": 1e-6}


def _check(ctx, inp, maps, grid, n, n_eff):
    ref = oracle.quiet_disk(inp.wave, inp.q_norm, n_eff, maps, grid, inp.case.step)
    for form, tol in TOL.items():
        got = ctx.quiet_disk(form, inp.wave, inp.q_norm, n_eff, maps, grid, inp.case.step)
        assert np.all(got[n_eff:] == 0)
        assert rel_err(got, ref) <= tol, form


# 45^2 and 46^2: 2048 cells; 64^2 and 65^2: 4096; 362^2 and 363^2: 131072
@pytest.mark.parametrize("grid,n", [(4, 1100), (45, 2309), (46, 2047), (64, 1500), (65, 1025), (91, 1501),
                                    (362, 1030), (363, 1030)])
def test_quiet_disk_orders(ctx, grid, n):
    inp = small_inputs(grid=grid, n=n)
    _check(ctx, inp, oracle_maps(grid=grid, n=n), grid, n, (n // 512) * 512)


@pytest.mark.parametrize("delta", [0.0, 1.7, "two"])
def test_equal_slopes(ctx, delta):
    """One slope for all cells (two: of either sign), so that only the cell decides the order."""
    grid, n = 60, 1500
    inp = small_inputs(grid=grid, n=n)
    maps = dict(oracle_maps(grid=grid, n=n))
    d = np.where(np.arange(grid * grid) % 3 == 0, -2.1, 1.9) if delta == "two" else np.full(grid * grid, delta)
    maps["delta"] = d.reshape(np.shape(maps["delta"]))
    _check(ctx, inp, maps, grid, n, 1024)


def test_no_visible_cell(ctx):
    grid, n = 50, 1100
    inp = small_inputs(grid=grid, n=n)
    maps = dict(oracle_maps(grid=grid, n=n))
    maps["limb"] = np.full_like(maps["limb"], -999.0)
    for form in TOL:
        assert not ctx.quiet_disk(form, inp.wave, inp.q_norm, 1024, maps, grid, inp.case.step).any()
