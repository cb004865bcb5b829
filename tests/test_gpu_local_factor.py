"""The complex128 local factors of the register-resident sweeps: series inside
|phase| <= 1/2, library functions beyond, and two half-steps with an absorber as one
rotation; and the renormalisation's quotient.

Tolerances: a half-step's factor is within 2 ulp and its product rounds once, the
transforms add a few ulp per sweep, so a handful of steps stays below 64 eps = 1.4e-14
of the state's norm (generic sweeps and oracle differ by the same amount from exact).
"""

import math

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def rel(a, b):
    return float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b))


def plans(n, kind, dt, **kw):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 8.0)
    mk = lambda g: Plan(n, x, k, dtype=torch.complex128, kind=kind, beta=40.0, dt=dt,  # noqa: E731
                        generic_only=g, **kw)
    return mk(False), mk(True), x


# constant offsets put every phase V dt/2 next to the series' end, on it, and far beyond
@pytest.mark.parametrize("phase", [1e-9, 0.4999, 0.5, 0.5001, 3.0, 40.0])
@pytest.mark.parametrize("kind", ["imaginary", "real"])
def test_factor_across_the_series_range(cuda, phase, kind):
    dt = 1e-3
    fast, generic, x = plans(32, kind, dt, static_expr=f"{2 * phase / dt!r}+0.3*x**2")
    a = torch.from_numpy(ssf.noisy_gaussian(x, seed=4)).cuda()
    b = a.clone()
    fast.step(a, 3)
    generic.step(b, 3)
    assert rel(a, b) < 64 * EPS * max(1.0, phase)


@pytest.mark.parametrize("gamma", [0.0, 1e-3, 300.0, 2000.0])
def test_absorber_in_the_fused_half_steps(cuda, gamma):
    """Im V dt/2 from nothing to beyond the series (2000 * 5e-4 = 1), inside one call."""
    n, dt = 48, 1e-3
    fast, generic, x = plans(n, "real", dt, static_expr="0.3*x**2+y**2")
    X = torch.from_numpy(x).cuda()
    edge = torch.clamp(X.abs() - 2.0, min=0.0)[:, None, None].expand(n, n, n)
    v = torch.complex(5 * torch.cos(X)[None, :, None].expand(n, n, n).contiguous(), (-gamma * edge).contiguous())
    for p in (fast, generic):
        p.set_static_potential(v.contiguous())
    a = torch.from_numpy(ssf.noisy_gaussian(x, seed=5)).cuda()
    b = a.clone()
    fast.step(a, 4)
    generic.step(b, 4)
    assert rel(a, b) < 64 * EPS


@pytest.mark.parametrize("scale", [1.0, 3.7e-3, 1.1e5])
def test_renormalisation_is_the_quotient(cuda, scale):
    fast, _, x = plans(32, "imaginary", 1e-3)
    a = torch.from_numpy(ssf.noisy_gaussian(x, seed=6)).cuda() * scale
    # (divided by NumPy: torch multiplies by a Python scalar's reciprocal)
    want = torch.view_as_real(a).cpu().numpy() / math.sqrt(fast.norm(a))
    fast.normalise(a)
    assert np.array_equal(torch.view_as_real(a).cpu().numpy(), want)
