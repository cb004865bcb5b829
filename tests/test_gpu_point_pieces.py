"""Point tables for a part of the grid at a time: the same bits as whole ones."""

import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu
FORM = "8*exp(-(x**2+y**2+(z-1.5*sin(4*t))**2)/0.64)+0.3*sin(10*t)*z**2+0.1*x*y*z"


# a last piece of one tile and of many, tiles of one line and of several, compiled sides too
@pytest.mark.parametrize("n", [6, 18, 32, 35, 64, 105, 130])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_pieces_equal_whole_tables(cuda, n, dtype):
    from gpe_simulator_b200 import Plan
    from gpe_simulator_b200.plan import launch_count
    x, k = ssf.get_grids(n, 12.0)
    kw = dict(dtype=dtype, kind="real", beta=50.0, dt=1e-3, static_expr="x**2+2*z**2", dynamic_expr=FORM)
    whole, parts = Plan(n, x, k, **kw), Plan(n, x, k, point_pieces=True, **kw)
    X = torch.from_numpy(x).cuda()
    v = torch.complex(torch.cos(X)[None, :, None].expand(n, n, n).contiguous(),
                      -20 * torch.clamp(X.abs() - 4, min=0)[None, None, :].expand(n, n, n).contiguous())
    a = torch.from_numpy(ssf.noisy_gaussian(x, seed=n)).to(dtype).cuda()
    b = a.clone()
    for static in (None, v.contiguous()):
        for p in (whole, parts):
            p.set_static_potential(static)
        before = launch_count(parts)
        whole.step(a, 3, 5)
        parts.step(b, 3, 5)
        assert launch_count(parts) - before > 3 * 5 or n == 6
        whole.step_at(a, 0.3)
        parts.step_at(b, 0.3)
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))
        d, e = whole.diagnostics(a, t=0.2, nk=True), parts.diagnostics(a, t=0.2, nk=True)
        assert all(d[q] == e[q] for q in ("N", "E_kin", "E_pot", "E_int"))
