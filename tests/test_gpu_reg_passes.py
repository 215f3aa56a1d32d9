"""Register passes (csrc/psb_reg.cuh) at every transform length they serve.

A grid with one long axis runs that axis's padded lengths 3N/2 (DNS) and 2N
(t-model) through the inverse and forward passes along x or y, ragged column
tiles included (k3 counts of 6 and 13, below a tile's columns); the right-hand
sides are held to the CPU oracle at the bars of the other parity tests: 1e-12
(FP64) and 2e-5 (FP32, fields rounded to FP32 on entry), relative, max norm.
"""
import numpy as np
import pytest

from oracle import spectral_oracle as orc
from tests.helpers import rel

pytestmark = pytest.mark.gpu
NU, DT, T0 = 1e-3, 2e-3, 0.4


def grids(shape):
    from pyspectral_b200 import Classes as C
    L = 2 * np.pi
    a1, a2, a3 = (np.arange(n) * (L / n) for n in shape)
    y, x, z = np.meshgrid(a2, a1, a3)
    kc = min(shape) // 2
    return C.gridclass(*shape, x, y, z, kc), orc.Grid(*shape, L / shape[0], L / shape[1], L / shape[2], kc)


def state(shape, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((3,) + tuple(shape))
    return np.stack([np.fft.rfftn(a) for a in x]) / np.sqrt(np.prod(shape))


def gpu_rhs(shape, tm, st, precision):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import Classes as C
    grid, g = grids(shape)
    main = C.variables(0, tm, 0, 0, 0, 0, grid, st[0], st[1], st[2], T0, DT, NU, precision=precision)
    main.computeRHS(main, grid, None, None)
    return main.Q.cpu().numpy().astype(np.complex128), g


@pytest.mark.parametrize("N", [12, 16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("tm", [0, 2])
def test_register_axis_passes_match_oracle(N, axis, tm):
    shape = (N, 8, 12) if axis == 0 else (8, N, 12)
    st = state(shape, 5 + N)
    fn = orc.rhs_nosgs if tm == 0 else orc.rhs_tmodel
    got, g = gpu_rhs(shape, tm, st, 64)
    ref = fn(g, st, orc.Params(nu=NU, t=T0))[0]
    assert rel(got, ref) < 1e-12
    st32 = st.astype(np.complex64).astype(np.complex128)
    got, _ = gpu_rhs(shape, tm, st32, 32)
    assert rel(got, fn(g, st32, orc.Params(nu=NU, t=T0))[0]) < 2e-5


@pytest.mark.parametrize("N", [16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256])
@pytest.mark.parametrize("tm", [0, 1, 2])
def test_register_z_pass_matches_oracle(N, tm):
    """Every real length of the register z pass (3N/2: DNS and Smagorinsky; 2N:
    t-model, its spectra kept to k3 = N inclusive) on 18 x 12 or 24 x 16
    pencils: ragged last tiles."""
    shape = (12, 8, N)
    st = state(shape, 7 + N)
    fn = {0: lambda g, s, p: orc.rhs_nosgs(g, s, p)[0], 1: lambda g, s, p: orc.rhs_smag(g, s, p)[0],
          2: lambda g, s, p: orc.rhs_tmodel(g, s, p)[0]}[tm]
    got, g = gpu_rhs(shape, tm, st, 64)
    assert rel(got, fn(g, st, orc.Params(nu=NU, t=T0))) < 1e-12
    st32 = st.astype(np.complex64).astype(np.complex128)
    got, _ = gpu_rhs(shape, tm, st32, 32)
    assert rel(got, fn(g, st32, orc.Params(nu=NU, t=T0))) < 2e-5


@pytest.mark.parametrize("N", [24, 32, 64, 96, 128, 192])
@pytest.mark.parametrize("precision", [64, 32])
def test_register_passes_of_mhd_match_oracle(N, precision):
    """MHD products and their linearisation (transforms of N and 2N points)."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import mpi as M
    shape = (12, 8, N)
    a1, a2, a3 = (np.arange(n) * (2 * np.pi / n) for n in shape)
    y, x, z = np.meshgrid(a2, a1, a3)
    grid = M.gridclass(*shape, x, y, z, 6)
    phys = np.random.default_rng(3 + N).standard_normal((6,) + shape)
    main = M.variables("MHD", 0, 0, 0, 0, grid, *phys, t=T0, dt=DT, nu=0.03, precision=precision, closure="tmodel",
                       Ct=0.13)
    g = orc.MHDGrid(*shape, 6)
    st = main.Q.cpu().numpy().astype(np.complex128)
    ref = orc.rhs_mhd_tmodel(g, st, 0.03, 0.13, T0, force=main.force.cpu().numpy().astype(np.complex128))[0]
    M.computeRHS_MHD(main, grid, None)
    assert rel(main.Q.cpu().numpy().astype(np.complex128), ref) < (1e-12 if precision == 64 else 2e-5)


@pytest.mark.parametrize("N", [16, 32, 48, 64, 72, 108, 128, 144])
@pytest.mark.parametrize("precision,tol", [(64, 1e-4), (32, 5e-4)])
def test_register_z_pass_learned_matches_oracle(N, precision, tol):
    """The learned closure on the register z pass against the BF16-emulating
    oracle, at the bars of the other learned tests (BF16 roundings of features
    that differ in the last bits)."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import mlp_oracle as mo
    from pyspectral_b200 import Classes as C
    from pyspectral_b200.learned import MLPModel
    shape = (12, 8, N)
    rng = np.random.default_rng(9 + N)
    k = np.sqrt(np.add.outer(np.add.outer(np.fft.fftfreq(12, 1 / 12) ** 2, np.fft.fftfreq(8, 1 / 8) ** 2),
                             np.fft.rfftfreq(N, 1 / N) ** 2))
    st = np.stack([np.fft.rfftn(a) for a in rng.standard_normal((3,) + shape)]) * np.exp(-0.25 * k)
    st = (st / np.sqrt(np.prod(shape))).astype(np.complex64).astype(np.complex128)
    grid, g = grids(shape)
    model = MLPModel.load()
    delta = 2 * np.pi / 64
    main = C.variables(0, "learned", 0, 0, 0, 0, grid, st[0], st[1], st[2], 0.0, DT, NU, precision=precision,
                       model=model, les_delta=delta)
    main.computeRHS(main, grid, None, None)
    ref = mo.rhs_learned(g, st, NU, model.params.cpu().numpy().astype(np.float64),
                         model.norm.cpu().numpy().astype(np.float64), delta, act=model.act_name)
    assert rel(main.Q.cpu().numpy().astype(np.complex128), ref) < tol
