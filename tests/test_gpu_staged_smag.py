"""Smagorinsky at padded lengths without a register pass: the staged y-inverse
pass forms one field per CTA, with the tiles a one-field pass has room for.
Oracle parity at 12, 486 and 576 points along y (and 486 along x) at the bars
of the other parity tests: 1e-12 (FP64) and 2e-5 (FP32, relative, max norm)."""
import numpy as np
import pytest

from oracle import spectral_oracle as orc
from tests.helpers import rel
from tests.test_gpu_reg_passes import NU, T0, gpu_rhs, grids, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (8, 324, 12), (12, 384, 8), (324, 8, 12)])
def test_staged_smagorinsky_matches_oracle(shape):
    st = state(shape, 31).astype(np.complex64).astype(np.complex128)
    ref = None
    for precision, tol in ((64, 1e-12), (32, 2e-5)):
        got, g = gpu_rhs(shape, 1, st, precision)
        ref = orc.rhs_smag(g, st, orc.Params(nu=NU, t=T0))[0] if ref is None else ref
        assert rel(got, ref) < tol


@pytest.mark.parametrize("precision", [64, 32])
def test_smagorinsky_y_pass_takes_one_field_tiles(precision):
    """A tile of 16 columns is 50 KB (FP64) for one field of 96 points; it is
    accepted, as for the other closures' y passes."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import _capi
    grid, _ = grids((64, 64, 64))
    ctx = grid.ctx(precision)
    want = {"tile": 16, "radices": [8, 4, 3]}
    ctx.set_tuned_shapes(_capi.SMAG, [None, want, None, None, None])
    assert ctx.tuned_shapes(_capi.SMAG)[1] == want
