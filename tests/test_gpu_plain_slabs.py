"""The plain form on maps of more cells than it holds constants of at a time."""
import numpy as np
import pytest

import oracle
from soap_gpu_gb300._lib import Activity

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("grid,n,n_phase", [(5000, 200, 1), (2100, 62 * 620, 2)])
def test_sums_over_slabs_of_cells(grid, n, n_phase):
    """A few thousand cells of a large map, among them the first and last of every slab of 2^22, with few
    tiles and with many: the oracle's sums, bit for bit; and the workspace stays below 2 GB where the
    constants of all 25 million cells take 5.6."""
    from soap_gpu_gb300.api import Context
    rng = np.random.default_rng(grid)
    gm, n_mu, step, n_eff = grid * grid, 2, 0.01, n - 3
    slab = 1 << 22
    edge = np.concatenate([np.r_[k - 2:k + 2] for k in range(slab, gm - 2, slab)])
    count = 3000 if n < 1000 else 150
    at = np.unique(np.r_[0, 1, edge, gm - 1, rng.integers(0, gm, count)])
    delta, limb, lb = np.full(gm, -999.0), np.full(gm, -999.0), np.zeros(gm)
    region = np.zeros(gm, np.int32)
    delta[at], limb[at] = rng.uniform(-3.0, 3.0, at.size), rng.uniform(0.3, 1.0, at.size)
    lb[at], region[at] = rng.uniform(-0.1, 0.2, at.size), rng.integers(0, n_mu, at.size)
    maps = dict(delta=delta, limb=limb, mu=limb, lb=lb, region=region)
    wave = 5000.0 + step * np.arange(n)
    cube = [1.0 + 0.3 * rng.uniform(-1, 1, (n_mu, n)) for _ in range(4)]
    sed = 0.3 + 0.1 * np.arange(n) / n, 1.0 + 0.1 * np.arange(n) / n
    bi = np.full(gm, -9999.0)
    bi[at[::2]], bi[at[1::2]] = 0.0, 1.0
    temp = np.where(bi == 0.0, 5115.0, np.where(bi == 1.0, 5900.0, -9999.0))
    dev = lambda a: torch.as_tensor(a, device="cuda:0")
    dm = {k: dev(v) for k, v in maps.items()}
    names = ("q_norm", "q_sed", "spot_norm", "fac_norm")
    cubes = dict({k: dev(c) for k, c in zip(names, cube)}, spot_sed=dev(sed[0]), fac_sed=dev(sed[1]))
    w, b, t = dev(wave), dev(np.tile(bi, (n_phase, 1))), dev(np.tile(temp, (n_phase, 1)))
    torch.cuda.synchronize()
    with Context(0) as ctx:
        free = torch.cuda.mem_get_info()[0]
        got = ctx.quiet_disk("plain64", w, cubes["q_norm"], n_eff, dm, grid, step)
        out = ctx.phase_integrate("plain64", w, n_eff, grid, t, b, dm, cubes, step, Activity(5778, 663, 250, 20, 0))
        ctx.synchronize()
        assert free - torch.cuda.mem_get_info()[0] < 2e9
    assert np.array_equal(got.cpu().numpy(), oracle.quiet_disk(wave, cube[0], n_eff, maps, grid, step))
    want = oracle.phase_integrate(wave, n_eff, grid, temp, bi, maps, *cube, *sed, step)
    for o, r in zip(out, want):
        for p in range(n_phase):
            assert np.array_equal(o[p].cpu().numpy(), r)
