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
