"""The dynamic tau-model's coefficient where its sums change shape: 18 modes (one
block, mostly idle), a ragged last block, and more modes than one round of the grid
of blocks (37,888).

Bar: each of the three sums runs over n modes of fields good to 1e-12 of their
largest value (the bar of the other FP64 parity tests), so it is off by at most
1e-12 sqrt(n) of its own size for fields without a preferred phase; the quotient
multiplies the error of its denominator by (|a| + |b|) / |a - b + 1e-5|.
"""
import numpy as np
import pytest

from oracle import spectral_oracle as orc
from tests.test_gpu_reg_passes import DT, NU, T0, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 32, 72])
def test_dynamic_tau_matches_oracle(N):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import Classes as C
    kc = N // 2
    kf = int(kc * 2.0 / 3.0)
    st = state((N, N, N), 11 + N)
    grid = C.gridclass.periodic(N, kc=kc)
    main = C.variables(0, "Dynamic tau-model", 0, 0, 0, 0, grid, st[0], st[1], st[2], T0, DT, NU, precision=64)
    main.computeRHS(main, grid, None, None)
    L = 2 * np.pi / N
    _, _, _, tau, (_, _, a, b) = orc.rhs_dtaumodel(orc.Grid(N, N, N, L, L, L, kc), st, orc.Params(nu=NU, t=T0))
    a, b = abs(a), abs(b)
    n = (2 * kf - 1) ** 2 * kf
    bar = 1e-12 * np.sqrt(n) * (1 + (a + b) / abs(a - b + 1e-5))
    assert abs(main.tau - tau) < bar * abs(tau)
