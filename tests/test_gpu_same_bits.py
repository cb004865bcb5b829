"""The sweep paths that promise each other's bits, with phases up to and beyond the short series and
array potentials: packed against scalar arithmetic at 256, where any product fused otherwise in one
of them shows once in some 1e10 operations."""

import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 256])
@pytest.mark.parametrize("kind", ["imaginary", "real"])
@pytest.mark.parametrize("beta", [0.0, 800.0])
@pytest.mark.parametrize("dt", [4e-3, 2e-2])
def test_paths(cuda, n, kind, beta, dt):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 12.0)
    X = torch.from_numpy(x).cuda()
    v = (5 * torch.cos(X))[None, :, None].expand(n, n, n).contiguous()
    loss = -300 * torch.clamp(X.abs() - 3, min=0)[:, None, None].expand(n, n, n)
    psi = torch.from_numpy(ssf.noisy_gaussian(x, seed=n)).to(torch.complex64).cuda()
    arrays = [None, v] if kind == "imaginary" else [None, v.to(torch.complex128), torch.complex(v, loss.contiguous())]
    for array in arrays:
        out = []
        for path in ("default", "plane", "tma"):
            p = Plan(n, x, k, dtype=torch.complex64, kind=kind, beta=beta, dt=dt, path=path,
                     static_expr="x**2+1.44*y**2+2.25*z**2")
            p.set_static_potential(array)
            a = psi.clone()
            p.step(a, 4, 1)
            assert p.status() == 0
            out.append(torch.view_as_real(a))
        assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
