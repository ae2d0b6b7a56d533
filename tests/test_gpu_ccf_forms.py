"""Forms of the normalised CCF's call: one spectrum as a vector, in place, long spectra."""
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
