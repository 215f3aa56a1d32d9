"""FP32 fields of magnitude 1e15: the right-hand side (quadratic) is within the
range of a float, and so are the products on the way when the fields are formed
at their physical size.  Against the oracle in 64
bits at the bar of the other FP32 tests, 2e-5 relative, max norm."""
import numpy as np
import pytest

from oracle import spectral_oracle as orc
from tests.helpers import rel

pytestmark = pytest.mark.gpu
N, NU, DT = 32, 1e-3, 2e-3


@pytest.mark.parametrize("tm", [0, 1])
def test_navier_stokes_fp32_large_fields(tm):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import Classes as C
    st = (3e16 * orc.isotropic_state(N, 2, k0=3.0)).astype(np.complex64).astype(np.complex128)
    grid = C.gridclass.periodic(N)
    main = C.variables(0, tm, 0, 0, 0, 0, grid, st[0], st[1], st[2], 0.0, DT, NU, precision=32)
    out = torch.empty_like(main.Q)
    grid.ctx(32).rhs(main.closure_code(), main.Q, out, main.params())
    got = out.cpu().numpy().astype(np.complex128)
    ref = (orc.rhs_smag if tm else orc.rhs_nosgs)(orc.Grid.periodic(N), st, orc.Params(nu=NU))[0]
    assert np.isfinite(got).all()
    assert rel(got, ref) < 2e-5


def test_mhd_fp32_large_fields():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import mpi as M
    grid = M.gridclass.periodic(N)
    phys = 1e15 * np.random.default_rng(5).standard_normal((6, N, N, N))
    main = M.variables("MHD", 0, 0, 0, 0, grid, *phys, t=0.0, dt=DT, nu=NU, precision=32, forcing=False)
    st = main.Q.cpu().numpy().astype(np.complex128)
    ref = orc.rhs_mhd(orc.MHDGrid(N, N, N, N // 2), st, NU)[0]
    M.computeRHS_MHD(main, grid, None)
    got = main.Q.cpu().numpy().astype(np.complex128)
    assert np.isfinite(got).all()
    assert rel(got, ref) < 2e-5
