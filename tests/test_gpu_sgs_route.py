"""psb_sgs_dns: the z pass is two register launches where the length has a
register form and one staged launch of both sets of products elsewhere (12^3:
18 points), or when the register form is switched off.  The stress and the
force are those of the oracle either way."""
import numpy as np
import pytest

from oracle import spectral_oracle as orc
from tests.helpers import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,zrr,launches", [(12, True, 1), (16, True, 2), (16, False, 1)])
@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-5)])
def test_sgs_dns_z_launches(N, zrr, launches, precision, tol):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from pyspectral_b200 import Classes as C
    st = orc.isotropic_state(N, 5, k0=3.0).astype(np.complex64).astype(np.complex128)
    grid = C.gridclass.periodic(N, kc=N // 4)
    ctx = grid.ctx(precision)
    ctx.set_zrr(zrr)
    q = torch.as_tensor(st, device="cuda").to(torch.complex128 if precision == 64 else torch.complex64).contiguous()
    w0, tau = torch.empty_like(q), torch.empty((6,) + tuple(q.shape[1:]), dtype=q.dtype, device="cuda")
    ctx.sgs_dns(q, w0, tau)
    ctx.timing(True)
    ctx.sgs_dns(q, w0, tau)
    torch.cuda.synchronize()
    assert [r[0] for r in ctx.timing_records()].count("z-fused") == launches
    ctx.timing(False)
    ref, tref = orc.sgs_dns(orc.Grid.periodic(N, kc=N // 4), st)
    assert rel(w0.cpu().numpy(), ref) < tol
    assert rel(tau.cpu().numpy(), tref) < tol
