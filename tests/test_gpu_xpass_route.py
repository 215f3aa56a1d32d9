"""The x pass on either side of the line between its staged and its register
form (csrc/psb_ctx.cuh, x_pass_in_registers), against the CPU oracle at the
bars of the other parity tests: 1e-12 (FP64), 2e-5 (FP32), relative, max norm.

Small grids run the staged pass, (N, 64, 64) and larger the register pass:
DNS and Smagorinsky at 3N/2 points, the t-model's two stages at 2N.  The
register pass is also asked for by its own shape on grids below the line, at
every length it has up to 384 points."""
import numpy as np
import pytest

from oracle import spectral_oracle as orc
from tests.helpers import rel
from tests.test_gpu_reg_passes import DT, NU, T0, gpu_rhs, grids, state

pytestmark = pytest.mark.gpu
RHS = {0: orc.rhs_nosgs, 1: orc.rhs_smag, 2: orc.rhs_tmodel}
# radices of the register x pass (psb_xreg.cuh PSB_REG_X)
OWN = {18: (6, 3), 24: (6, 4), 36: (9, 4), 48: (12, 4), 54: (9, 2, 3), 72: (6, 3, 4), 96: (8, 3, 4), 108: (9, 3, 4),
       144: (9, 4, 4), 162: (9, 6, 3), 192: (8, 6, 4), 216: (9, 6, 4), 288: (9, 8, 4), 324: (9, 9, 4), 384: (12, 8, 4)}


@pytest.mark.parametrize("N", [12, 24, 36, 48, 64, 72, 96, 108, 128, 144])
@pytest.mark.parametrize("tm", [0, 1, 2])
def test_x_pass_on_wide_grids_matches_oracle(N, tm):
    shape = (N, 64, 64) if tm < 2 else (N, 48, 48)
    st = state(shape, 3 + N).astype(np.complex64).astype(np.complex128)
    g = grids(shape)[1]
    ref = RHS[tm](g, st, orc.Params(nu=NU, t=T0))[0]
    for precision, tol in ((64, 1e-12), (32, 2e-5)):
        assert rel(gpu_rhs(shape, tm, st, precision)[0], ref) < tol


@pytest.mark.parametrize("L", sorted(OWN))
@pytest.mark.parametrize("tm", [0, 1])
@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-5)])
def test_register_x_pass_by_its_own_shape_matches_oracle(L, tm, precision, tol):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import Classes as C
    shape = (2 * L // 3, 8, 12)
    st = state(shape, L).astype(np.complex64).astype(np.complex128)
    grid, g = grids(shape)
    main = C.variables(0, tm, 0, 0, 0, 0, grid, st[0], st[1], st[2], T0, DT, NU, precision=precision)
    ctx, code = grid.ctx(precision), main.closure_code()
    want = {"tile": 4 if precision == 64 else 8, "radices": list(OWN[L])}
    ctx.set_tuned_shapes(code, [None, None, None, None, want])
    assert ctx.tuned_shapes(code)[4] == want
    out = torch.empty_like(main.Q)
    ctx.rhs(code, main.Q, out, main.params())
    assert rel(out.cpu().numpy(), RHS[tm](g, st, orc.Params(nu=NU, t=T0))[0]) < tol


@pytest.mark.parametrize("shape,precision,tol", [((64, 128, 96), 64, 1e-12), ((144, 128, 128), 32, 2e-5)])
def test_mhd_register_x_pass_matches_oracle(shape, precision, tol):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import mpi as M
    a1, a2, a3 = (np.arange(n) * (2 * np.pi / n) for n in shape)
    y, x, z = np.meshgrid(a2, a1, a3)
    grid = M.gridclass(*shape, x, y, z, min(shape) // 2)
    phys = np.random.default_rng(3).standard_normal((6,) + shape)
    main = M.variables("MHD", 0, 0, 0, 0, grid, *phys, t=T0, dt=DT, nu=0.03, precision=precision)
    st = main.Q.cpu().numpy().astype(np.complex128)
    ref = orc.rhs_mhd(orc.MHDGrid(*shape, min(shape) // 2), st, 0.03, force=main.force.cpu().numpy().astype(np.complex128))
    M.computeRHS_MHD(main, grid, None)
    assert rel(main.Q.cpu().numpy(), ref[0] if isinstance(ref, tuple) else ref) < tol
