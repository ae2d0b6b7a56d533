"""Threads with a context each."""
import threading

import numpy as np
import pytest

import oracle
from _cases import small_inputs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_calls_of_different_sizes_side_by_side():
    """Short and long spectra, small and larger grids: a kernel's limit of shared memory is the
    process's, and no thread's calls may lower it between another's setting and its launch."""
    from soap_gpu_gb300.api import Context
    inp = small_inputs()
    c = inp.case
    errors = []
    dev = lambda a: torch.as_tensor(a, device="cuda:0")

    def work(grid, n, rounds):
        try:
            rng = np.random.default_rng(grid)
            wave = dev(5000.0 + 0.01 * np.arange(n))
            maps = {k: dev(v) for k, v in oracle.disk_maps(grid, c.period, c.w_ratio, c.incl, c.radius_km, c.u1, c.u2,
                                                           inp.mu_boundary, inp.lb).items()}
            cube = dev(1.0 + 0.1 * rng.uniform(-1, 1, (len(inp.mu_boundary) + 1, 1024)))
            base = dev(1000.0 * (1.0 + 0.1 * rng.uniform(-1, 1, n)))
            spec = dev(10.0 * rng.uniform(0, 1, (1, n)))
            short = wave[:1024].contiguous()
            torch.cuda.synchronize()
            with Context(0) as ctx:
                first = None
                for _ in range(rounds):
                    for _ in range(10):
                        q = ctx.quiet_disk("fast32", short, cube, 1024, maps, grid, 0.01)
                    low, _ = ctx.lower_resolution("fast32", wave, spec, n, c.sigma_v, base=base, step_mult=0.01,
                                                  step_exp=0.01)
                    ctx.synchronize()
                    first = first or (q, low)
                    assert torch.equal(q, first[0]) and torch.equal(low, first[1])
        except Exception as e:   # noqa: BLE001 (reported below)
            errors.append(e)

    sizes = [(20, 4096), (64, 4096), (20, 170000), (64, 170000)] * 2
    threads = [threading.Thread(target=work, args=s + (150,)) for s in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
