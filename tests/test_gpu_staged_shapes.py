"""Launch shapes given by hand at lengths that have register passes.

A staged shape runs the staged pass (other roundings than the register pass,
so not the same bits), with and without bulk tensor copies; the register
pass's own shape brings the register pass back.  64^3: padded length 96 in
every pass.  Bars: 1e-12 (FP64) and 2e-5 (FP32) against the oracle, relative,
max norm; bulk copies change no arithmetic (1e-14 and 1e-6: contraction of
separately compiled kernels)."""
import numpy as np
import pytest

from oracle import spectral_oracle as orc
from tests.helpers import rel

pytestmark = pytest.mark.gpu
N, NU, DT = 64, 1e-3, 2e-3


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-5)])
@pytest.mark.parametrize("tm", [0, 1])
@pytest.mark.parametrize("radices", [(8, 4, 3), (16, 6)])
def test_staged_shape_runs_the_staged_pass(tm, precision, tol, radices):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import Classes as C
    st = orc.isotropic_state(N, 4, k0=4.0).astype(np.complex64).astype(np.complex128)
    ref = (orc.rhs_smag if tm else orc.rhs_nosgs)(orc.Grid.periodic(N), st, orc.Params(nu=NU))[0]
    grid = C.gridclass.periodic(N)
    main = C.variables(0, tm, 0, 0, 0, 0, grid, st[0], st[1], st[2], 0.0, DT, NU, precision=precision)
    ctx, code = grid.ctx(precision), main.closure_code()

    def rhs():
        out = torch.empty_like(main.Q)
        ctx.rhs(code, main.Q, out, main.params())
        return out.cpu().numpy()

    default = rhs()
    assert rel(default, ref) < tol
    for k in (0, 1, 3, 4):
        ctx.autotune_clear(code)
        shapes = [None] * 5
        shapes[k] = {"tile": 2, "radices": list(radices)}
        ctx.set_tuned_shapes(code, shapes)
        got = {}
        for tma in (True, False):
            ctx.set_tma(tma)
            got[tma] = rhs()
            assert rel(got[tma], ref) < tol
            assert not np.array_equal(got[tma], default), (k, tma)
        ctx.set_tma(True)
        assert rel(got[True], got[False]) < (1e-14 if precision == 64 else 1e-6)
        own = ctx.tuned_shapes(code)
        ctx.autotune_clear(code)
        # the other passes' entries are the register passes' own shapes
        ctx.set_tuned_shapes(code, [sh if j != k else None for j, sh in enumerate(own)])
        assert np.array_equal(rhs(), default)
    ctx.autotune_clear(code)
    assert ctx.device_status() == 0
