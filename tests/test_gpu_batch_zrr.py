"""psb_ctx_set_zrr applies to a batch that has stepped already: with the
register z pass switched off its next step is bit for bit the step of a batch
that never had it, and switching it on again brings the register pass back."""
import numpy as np
import pytest

from oracle import spectral_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("closure", ["smag", "dns"])
@pytest.mark.parametrize("precision", [64, 32])
def test_batch_follows_set_zrr(closure, precision):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import _capi
    from pyspectral_b200.ensemble import Batch
    N, runs = 32, 2
    cdt = torch.complex128 if precision == 64 else torch.complex64
    st = [torch.as_tensor(orc.isotropic_state(N, s, k0=3.0), device="cuda").to(cdt) for s in range(runs)]
    code = _capi.SMAG if closure == "smag" else _capi.DNS

    def make():
        ctx = _capi.Context(N, N, N, precision=precision)
        b = Batch(ctx, code, runs)
        own = [s.clone() for s in st]
        for r, q in enumerate(own):
            b.set_run(r, q, None, _capi.make_params(nu=1e-3, dt=2e-3))
        return ctx, b, own

    def step(ctx, b, own, zrr):
        ctx.set_zrr(zrr)
        for q, s in zip(own, st):
            q.copy_(s)
        b.step(1)
        torch.cuda.synchronize()
        return np.stack([q.cpu().numpy() for q in own])

    off = step(*make(), False)  # never had the register pass
    ctx, b, own = make()
    on = step(ctx, b, own, True)
    assert not np.array_equal(on, off)
    assert np.array_equal(step(ctx, b, own, False), off)
    assert np.array_equal(step(ctx, b, own, True), on)
