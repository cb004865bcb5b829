"""The streaming norm and the angular momentum on the run-time-length sweeps, against the
generic sweeps and exact sums.  FP64 sums of at most 2e6 terms, compensated: 1e-14."""

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu


def plan(n, dtype, generic=False):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 10.0)
    return Plan(n, x, k, dtype=dtype, kind="real", beta=10.0, dt=1e-3, generic_only=generic), x


# fewer points than a block's round, one round exactly, ragged ends, several rounds per block
@pytest.mark.parametrize("n", [2, 7, 13, 16, 32, 45, 128])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_norm(cuda, n, dtype):
    p, x = plan(n, dtype)
    rng = np.random.default_rng(n)
    a = torch.from_numpy(rng.standard_normal((n, n, n)) + 1j * rng.standard_normal((n, n, n))).to(dtype).cuda()
    v = torch.view_as_real(a).double()
    want = float((v * v).sum()) * (x[1] - x[0]) ** 3
    assert abs(p.norm(a) - want) <= 1e-13 * want
    # a view that is aligned to its elements only
    flat = torch.empty(n ** 3 + 1, dtype=dtype, device=cuda)
    b = flat[1:].view(n, n, n)
    b.copy_(a)
    assert p.norm(b) == p.norm(a)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_norm_reports_non_finite(cuda, bad):
    p, _ = plan(32, torch.complex64)
    a = torch.ones((32, 32, 32), dtype=torch.complex64, device=cuda)
    a[31, 31, 31] = bad
    assert not np.isfinite(p.norm(a))
    assert p.status() & 1


@pytest.mark.parametrize("n", [7, 16, 30, 64, 105, 128])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_angular_momentum(cuda, n, dtype):
    """A flow exp(i 0.3 x y): Lz = 0.3 (<x^2> - <y^2>); the sums against the generic sweeps."""
    p, x = plan(n, dtype)
    g, _ = plan(n, dtype, generic=True)
    X, Y = x[:, None, None], x[None, :, None]
    psi = ssf.noisy_gaussian(x, sigma=1.3, seed=n) * np.exp(0.3j * X * Y) * np.exp(-0.1 * Y ** 2)
    a = torch.from_numpy(psi).to(dtype).cuda()
    got, want = p.angular_momentum(a), g.angular_momentum(a)
    # size of the terms the two sums cancel from
    size = float(np.sum(np.abs(psi) ** 2)) * (x[1] - x[0]) ** 3 * np.pi / (x[1] - x[0]) * np.abs(x).max()
    assert abs(got - want) <= 1e-13 * size
