"""Forms of the normalised CCF's call: one spectrum as a vector, in place, long spectra."""
import ctypes

import numpy as np
import pytest

from _cases import small_inputs
from test_gpu_ccf_adjoint import _ccf_setup, _dev

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _spectra(ctx, n_spec=3):
    inp = small_inputs()
    cs = _ccf_setup(ctx, inp, 4096)
    rng = np.random.default_rng(2)
    return cs, _dev(1.0 - 0.3 * rng.uniform(0, 1, (n_spec, cs.wave_trim.numel())) * inp.q_norm[0, 210:4096 - 210])


def test_normalised_ccf_of_one_spectrum(ctx):
    """A vector gives the row that it gives among others (the same operations: the same bits)."""
    from soap_gpu_gb300.differentiable import normalised_ccf
    cs, sp = _spectra(ctx)
    with torch.no_grad():
        rows = normalised_ccf(sp, cs)
        for s in range(sp.shape[0]):
            assert torch.equal(normalised_ccf(sp[s], cs), rows[s])


def test_gradient_of_one_spectrum(ctx):
    """Its gradient is the row's too, and the operator refuses shapes that its kernels would read past."""
    from soap_gpu_gb300.differentiable import normalised_ccf
    from soap_gpu_gb300.torch_ops import ops
    cs, sp = _spectra(ctx)
    w = _dev(np.random.default_rng(4).standard_normal((sp.shape[0], cs.vel.numel())))
    x = sp.clone().requires_grad_(True)
    (normalised_ccf(x, cs) * w).sum().backward()
    for s in range(sp.shape[0]):
        v = sp[s].clone().requires_grad_(True)
        (normalised_ccf(v, cs) * w[s]).sum().backward()
        assert torch.equal(v.grad, x.grad[s])
    args = (cs.vel, cs.line_wave, cs.line_weight, cs.wave_trim, cs.step)
    for g, raw in ((w[0], w[0]), (w[:, 1:].contiguous(), w[:, 1:].contiguous()), (w, w[:2].contiguous()), (w, None)):
        with pytest.raises(RuntimeError):
            ops(ctx).ccf_adjoint(*args, g, ccf_raw=raw, **cs.kwargs())


def test_normalise_in_place(ctx):
    """raw and ccf_out the same buffer, on the device and on the host: the values of separate buffers."""
    from soap_gpu_gb300 import _lib
    cs, sp = _spectra(ctx, 5)
    args = (cs.vel, cs.line_wave, cs.line_weight, cs.wave_trim, cs.step, sp)
    raw = ctx.ccf("plain64", *args, normalise=False, **cs.kwargs())
    want = ctx.ccf("plain64", *args, normalise=True, **cs.kwargs())
    lib = _lib.load()
    n_spec, n_v = raw.shape
    torch.cuda.synchronize()
    call = lambda src, mem, dst: lib.soapgb_ccf_normalise(ctx.h, n_spec, n_v, ctypes.c_void_p(src), mem, ctypes.c_void_p(dst))
    out, same = torch.empty_like(raw), raw.clone()
    torch.cuda.synchronize()
    assert call(raw.data_ptr(), _lib.DEVICE, out.data_ptr()) == 0
    assert call(same.data_ptr(), _lib.DEVICE, same.data_ptr()) == 0
    ctx.synchronize()
    assert torch.equal(out, want) and torch.equal(same, want)
    host = raw.cpu().numpy().copy()
    assert call(host.ctypes.data, _lib.HOST, host.ctypes.data) == 0
    assert np.array_equal(host, want.cpu().numpy())


def test_grid_longer_than_a_pitch(ctx):
    """A grid whose ends lie 2^31 bytes apart.  Both lines lie in its first part, which alone gives the
    same raw CCF and gradient."""
    n, part, step = (1 << 28) + 2, 1 << 20, 2.0 ** -17
    wave = torch.arange(n, dtype=torch.float64, device="cuda:0").mul_(step).add_(5000.0)
    spec = torch.ones((1, n), dtype=torch.float64, device="cuda:0")
    spec[0, :part] += _dev(0.1 * np.random.default_rng(1).standard_normal(part))
    lines = (_dev([5001.0, 5005.0]), _dev([0.5, 0.8]))
    vel, g = _dev([0.0]), _dev([[1.5]])
    kw = dict(normalise=False, wave_extend=10 * step, mask_step=step, index_old=10)
    got, want = (ctx.ccf("plain64", vel, *lines, wave[:m], step, spec[:, :m].contiguous(), **kw) for m in (n, part))
    assert float(want[0, 0]) > 0 and torch.equal(got, want)
    del spec
    got, want = (ctx.ccf_adjoint(vel, *lines, wave[:m], step, g, **kw) for m in (n, part))
    assert torch.equal(got[:, :part], want) and not got[0, part:].any()
