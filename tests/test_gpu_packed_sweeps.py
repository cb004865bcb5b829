"""The 256- and 512-point complex64 sweeps with two lines per thread, against the generic sweeps:
steps with every potential form, states aligned to their elements only (the 16-byte accesses
fall back), phases beyond the short series.  A complex64 sweep rounds each value a few times
at 6e-8: two steps (ten sweeps) stay within 2e-6 of the norm."""

import math

import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu
L = 24.0


@pytest.fixture(params=[256, 512])
def n(request):
    return request.param


def rel(a, b):
    """Norm of the difference over the norm, plane by plane (no full-size temporaries)."""
    d = sum(float(torch.linalg.vector_norm(x - y)) ** 2 for x, y in zip(a, b))
    return math.sqrt(d / sum(float(torch.linalg.vector_norm(y)) ** 2 for y in b))


def state(cuda, n, offset=0):
    x, _ = ssf.get_grids(n, L)
    X = torch.from_numpy(x).to(cuda)
    g = torch.exp(-X ** 2 / 8)
    flat = torch.empty(n ** 3 + offset, dtype=torch.complex64, device=cuda)
    psi = flat[offset:].view(n, n, n)
    psi.copy_((g[:, None, None] * g[None, :, None] * g[None, None, :]
               * torch.polar(torch.ones_like(X), 0.4 * X)[:, None, None]).to(torch.complex64))
    return psi


def pair(n, kind, dt, **kw):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, L)
    return [Plan(n, x, k, dtype=torch.complex64, kind=kind, beta=30.0, dt=dt, generic_only=g,
                 static_expr="x**2+1.44*y**2+2.25*z**2", **kw) for g in (False, True)]


# dt = 2e-3 puts the corners' phases (V dt/2 up to 1.3) beyond both series
@pytest.mark.parametrize("kind", ["imaginary", "real"])
@pytest.mark.parametrize("dt", [1e-4, 2e-3])
@pytest.mark.parametrize("offset", [0, 1])
def test_steps(cuda, n, kind, dt, offset):
    from gpe_simulator_b200 import Beam
    kw = dict(beam=Beam(20.0, 0.5, 2.0, 1.0, 0.02), k_cut=60.0) if kind == "real" else {}
    new, old = pair(n, kind, dt, **kw)
    a = state(cuda, n, offset)
    b = a.clone()
    new.step(a, 2, 3)
    old.step(b, 2, 3)
    assert rel(a, b) < 2e-6
    assert new.status() == 0


def test_array_potential_with_loss(cuda, n):
    new, old = pair(n, "real", 1e-4)
    x, _ = ssf.get_grids(n, L)
    X = torch.from_numpy(x).to(cuda)
    edge = torch.clamp(X.abs() - 8.0, min=0.0)
    v = torch.zeros((n, n, n), dtype=torch.complex128, device=cuda)
    v.real.add_(5 * torch.cos(X)[None, :, None])
    v.imag.sub_(300.0 * edge[:, None, None])
    for p in (new, old):
        p.set_static_potential(v)
    del v
    a = state(cuda, n)
    b = a.clone()
    new.step(a, 2)
    old.step(b, 2)
    assert rel(a, b) < 2e-6


def test_transform_round_trip(cuda, n):
    new, old = pair(n, "real", 1e-4)
    a = state(cuda, n)
    f, g = new.fft(a), old.fft(a)
    assert rel(f, g) < 1e-6
    assert rel(new.fft(f, inverse=True), a) < 1e-6
