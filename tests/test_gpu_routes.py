"""Routes that other tests reach at one end of their range only: the largest sides of the
run-time-length sweeps, batches on the packed and the run-time-length sweeps, and point tables
together with array potentials.  The reference is the generic Stockham sweeps
(``generic_only``) or a plan of its own.

Tolerances: a complex64 sweep rounds each value a few times at 6e-8, so ten sweeps stay within
2e-6 of the norm; complex128 within 64 eps."""

import math

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu
TOL = {torch.complex64: 2e-6, torch.complex128: 64 * np.finfo(np.float64).eps}
TRAP = "x**2+1.44*y**2+2.25*z**2"


def rel(a, b):
    """Norm of the difference over the norm, plane by plane (no full-size temporaries)."""
    d = sum(float(torch.linalg.vector_norm(x - y)) ** 2 for x, y in zip(a, b))
    return math.sqrt(d / sum(float(torch.linalg.vector_norm(y)) ** 2 for y in b))


def state(x, dtype, device):
    """A moving Gaussian without symmetry between the axes, plane by plane."""
    n = len(x)
    X = torch.from_numpy(x).to(device)
    gz = torch.exp(-(X - 0.3) ** 2 / 5) * torch.polar(torch.ones_like(X), 0.7 * X)
    gy = torch.exp(-(X + 0.2) ** 2 / 7) * torch.polar(torch.ones_like(X), -0.2 * X)
    plane = (gy[:, None] * gz[None, :]).to(torch.complex128)
    psi = torch.empty((n, n, n), dtype=dtype, device=device)
    for i in range(n):
        psi[i] = plane * math.exp(-x[i] ** 2 / 6) * complex(math.cos(0.4 * x[i]), math.sin(0.4 * x[i]))
    return psi


def pair(n, dtype, kind, L=24.0, **kw):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, L)
    kw = dict(dict(dtype=dtype, kind=kind, beta=30.0, dt=1e-4, static_expr=TRAP), **kw)
    return Plan(n, x, k, **kw), Plan(n, x, k, generic_only=True, **kw), x


def test_512_complex128(cuda):
    """Stirred steps, then a lossy array potential with a cutoff, and n(k)."""
    from gpe_simulator_b200 import Beam
    n, dt = 512, torch.complex128
    new, old, x = pair(n, dt, "real", beam=Beam(20.0, 0.5, 2.0, 1.0, 0.02), k_cut=60.0)
    a = state(x, dt, cuda)
    b = a.clone()
    new.step(a, 2, 5)
    old.step(b, 2, 5)
    assert rel(a, b) < TOL[dt]
    d, e = new.diagnostics(b, t=0.01, nk=True), old.diagnostics(b, t=0.01, nk=True)
    np.testing.assert_allclose(d["Nk"], e["Nk"], rtol=1e-10, atol=1e-13 * np.abs(e["Nk"]).max())
    assert np.array_equal(d["counts"], e["counts"])
    assert all(abs(d[q] - e[q]) <= 1e-12 * abs(e[q]) for q in ("N", "E_kin", "E_pot", "E_int", "mu"))
    X = torch.from_numpy(x).to(cuda)
    v = torch.zeros((n, n, n), dtype=dt, device=cuda)
    v.real.add_(5 * torch.cos(X)[None, :, None])
    v.imag.sub_(300.0 * torch.clamp(X.abs() - 8.0, min=0.0)[:, None, None])
    for p in (new, old):
        p.set_static_potential(v)
    del v
    new.step(a, 2, 7)
    old.step(b, 2, 7)
    assert rel(a, b) < 2 * TOL[dt]


# 1000 = 10^3; 1024 takes a radix of 16 and eight-byte rows of four lines
@pytest.mark.parametrize("n", [1000, 1024])
def test_largest_sides_complex64(cuda, n):
    new, old, x = pair(n, torch.complex64, "imaginary")
    a = state(x, torch.complex64, cuda)
    f, g = new.fft(a), old.fft(a)
    assert all(torch.equal(torch.view_as_real(p), torch.view_as_real(q)) for p, q in zip(f, g))
    del f, g
    b = a.clone()
    new.step(a, 1)
    old.step(b, 1)
    assert rel(a, b) < TOL[torch.complex64]


# a member aligned to its elements only takes the narrow loads for its whole group
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [256, 512])
@pytest.mark.parametrize("kind", ["imaginary", "real"])
def test_packed_sweeps_in_a_batch(cuda, n, kind, offset):
    from gpe_simulator_b200 import Beam, Plan
    from gpe_simulator_b200.batch import Batch, Instance
    beam = Beam(20.0, 0.5, 2.0, 1.0, 0.02) if kind == "real" else None
    insts = [Instance(n=n, simulation_range=24.0, beta=b, dt=1e-4, static_expr=TRAP, kind=kind, beam=beam)
             for b in (30.0, 60.0)]
    psis = []
    for i in range(2):
        flat = torch.empty(n ** 3 + offset * i, dtype=torch.complex64, device=cuda)
        psis.append(flat[offset * i:].view(n, n, n))
        psis[i].copy_(state(insts[i].x, torch.complex64, cuda))
    want = psis[0].clone()
    batch = Batch(insts, torch.complex64)
    batch.bind(psis)
    batch.step(2)
    diag = batch.diagnostics()
    for i, inst in enumerate(insts):
        plan = Plan(n, inst.x, inst.k, dtype=torch.complex64, kind=kind, beta=inst.beta, dt=inst.dt, static_expr=TRAP,
                    beam=beam)
        alone = want.clone()
        if kind == "real":
            for s in range(2):
                plan.step(alone, 1, s)
        else:
            plan.step(alone, 2)
        assert torch.equal(torch.view_as_real(alone), torch.view_as_real(psis[i]))
        d = plan.diagnostics(alone, t=2 * inst.dt if kind == "real" else 0.0)
        assert [d[q] for q in ("N", "E_kin", "E_pot", "E_int", "E", "mu")] == list(diag[i])


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_real_time_batch_on_run_time_length_sweeps(cuda, dtype):
    from gpe_simulator_b200 import Plan
    from gpe_simulator_b200.batch import Batch, initial_states, stirring_instances
    insts = stirring_instances(rates=(0.25, 1.0), gs=(500.0,), grids=((35, 12.0), (60, 16.0), (105, 16.0)))
    states = initial_states(insts, dtype, seed0=40)
    work = [s.clone() for s in states]
    batch = Batch(insts, dtype)
    batch.bind(work)
    batch.step(5)
    diag = batch.diagnostics()
    for i, inst in enumerate(insts):
        plan = Plan(inst.n, inst.x, inst.k, dtype=dtype, kind="real", beta=inst.beta, dt=inst.dt,
                    static_expr=inst.static_expr, beam=inst.beam)
        alone = states[i].clone()
        for s in range(5):
            plan.step(alone, 1, s)
        assert torch.equal(alone, work[i])
        d = plan.diagnostics(alone, t=5 * inst.dt)
        assert np.allclose([d["N"], d["E"], d["mu"]], diag[i, [0, 4, 5]], rtol=1e-12, atol=0)


@pytest.mark.parametrize("n", [32, 35, 60])
@pytest.mark.parametrize("loss", [0.0, 30.0])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_point_tables_with_arrays_and_cutoff(cuda, n, dtype, loss):
    # (no mode of exactly the cutoff's length: rounding decides those, path by path)
    new, old, x = pair(n, dtype, "real", L=10.0, dt=1e-3, k_cut=0.71 * math.pi * n / 10.0,
                       dynamic_expr="8*exp(-(x**2+y**2+(z-1.5*sin(4*t))**2)/0.64)+0.2*x*z*cos(t)")
    X = torch.from_numpy(x).to(cuda)
    edge = torch.clamp(X.abs() - 3.0, min=0.0)[:, None, None].expand(n, n, n)
    v = torch.complex(3 * torch.sin(X)[None, None, :].expand(n, n, n).contiguous(), (-loss * edge).contiguous())
    for p in (new, old):
        p.set_static_potential(v.contiguous())
    a = state(x, dtype, cuda)
    b = a.clone()
    new.step(a, 3, 20)
    old.step(b, 3, 20)
    assert rel(a, b) < 1.5 * TOL[dtype]
    d, e = new.diagnostics(b, t=0.2), old.diagnostics(b, t=0.2)
    bound = 1e-6 if dtype == torch.complex64 else 1e-12
    assert abs(d["E_pot"] - e["E_pot"]) <= bound * max(abs(e["E_pot"]), abs(e["N"]))
