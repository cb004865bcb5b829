"""The sweeps that take the grid side at run time, against the generic Stockham sweeps
(``generic_only``) of the same plan: two to four phases, every radix, ragged tiles, all
potential forms, and the batched launches.

Tolerances: a complex64 sweep rounds each value a few times at 6e-8, so the ten sweeps of
two steps keep two roundings of the same step within 2e-6 of the norm; complex128 within
64 eps.  Transforms and reductions in complex64 keep the Stockham passes' rounding: equal
bit for bit (the FP64 sums over them up to their order, 1e-12).
"""

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu

TOL = {torch.complex64: 2e-6, torch.complex128: 64 * np.finfo(np.float64).eps}
# radices of the steps' phases: 2..16 all occur, two phases up to 15 x 15, three, tiles
# smaller and larger than a row, sides below and above the two-blocks-per-SM line
SIDES = [6, 18, 22, 26, 30, 35, 39, 63, 77, 81, 100, 105, 121, 125, 130, 143, 168, 169, 182, 196, 200, 216, 225]


def rel(a, b):
    d = a.to(torch.complex128) - b.to(torch.complex128)
    return float(torch.linalg.vector_norm(d) / torch.linalg.vector_norm(b.to(torch.complex128)))


def pair(n, dtype, kind, **kw):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 10.0)
    mk = lambda g: Plan(n, x, k, dtype=dtype, kind=kind, beta=50.0, dt=1e-3,  # noqa: E731
                        static_expr="x**2+1.44*y**2+2.25*z**2", generic_only=g, **kw)
    return mk(False), mk(True), x


def state(x, dtype, seed):
    return torch.from_numpy(ssf.noisy_gaussian(x, sigma=1.2, seed=seed)).to(dtype).cuda()


@pytest.mark.parametrize("n", SIDES)
@pytest.mark.parametrize("kind", ["imaginary", "real"])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_steps_match_generic_sweeps(cuda, n, kind, dtype):
    from gpe_simulator_b200 import Beam
    kw = dict(beam=Beam(20.0, 0.8, 1.5, 1.0, 0.002)) if kind == "real" else {}
    new, old, x = pair(n, dtype, kind, **kw)
    a = state(x, dtype, n)
    b = a.clone()
    new.step(a, 2, 1)
    old.step(b, 2, 1)
    assert rel(a, b) < TOL[dtype]
    assert new.status() == 0
    new.step_at(a, 0.3)
    old.step_at(b, 0.3)
    assert rel(a, b) < 1.5 * TOL[dtype]


@pytest.mark.parametrize("n", [30, 105, 125])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_array_line_and_cutoff_potentials(cuda, n, dtype):
    """Complex static array, a dynamic formula without z terms, momentum cutoff."""
    from gpe_simulator_b200.plan import launch_count
    new, old, x = pair(n, dtype, "real", dynamic_expr="0.5*sin(3*t)*x+2*exp(-(y-cos(t))**2)",
                          k_cut=0.7 * np.pi * n / 10.0)
    X = torch.from_numpy(x).cuda()
    edge = torch.clamp(X.abs() - 3.0, min=0.0)[:, None, None].expand(n, n, n)
    v = torch.complex(3 * torch.sin(X)[None, None, :].expand(n, n, n).contiguous(), (-200.0 * edge).contiguous())
    for p in (new, old):
        p.set_static_potential(v.contiguous())
    a = state(x, dtype, 7)
    b = a.clone()
    before = launch_count(new)
    new.step(a, 3)
    assert launch_count(new) - before == 2 + 5 * 3     # four sweeps per step, a line table per z sweep
    old.step(b, 3)
    assert rel(a, b) < 1.5 * TOL[dtype]


@pytest.mark.parametrize("n", [18, 30, 77, 105, 130, 162, 200, 216])
def test_complex64_transforms_keep_their_rounding(cuda, n):
    new, old, x = pair(n, torch.complex64, "real", nk_bins=50)
    a = state(x, torch.complex64, n + 1)
    f, g = new.fft(a), old.fft(a)
    assert torch.equal(torch.view_as_real(f), torch.view_as_real(g))
    assert torch.equal(torch.view_as_real(new.fft(f, inverse=True)), torch.view_as_real(old.fft(g, inverse=True)))
    d, e = new.diagnostics(a, nk=True), old.diagnostics(a, nk=True)
    np.testing.assert_allclose(d["Nk"], e["Nk"], rtol=1e-12, atol=1e-14 * np.abs(e["Nk"]).max())
    assert np.array_equal(d["counts"], e["counts"])
    for key in ("N", "E_kin", "E_int", "E_pot"):
        assert abs(d[key] - e[key]) <= 1e-7 * abs(e[key])


@pytest.mark.parametrize("n", [30, 105, 200])
def test_complex128_transforms_and_sums(cuda, n):
    new, old, x = pair(n, torch.complex128, "real")
    a = state(x, torch.complex128, n + 2)
    f, g = new.fft(a), old.fft(a)
    assert rel(f, g) < TOL[torch.complex128]
    assert rel(new.fft(f, inverse=True), a) < TOL[torch.complex128]
    d, e = new.diagnostics(a, nk=True), old.diagnostics(a, nk=True)
    np.testing.assert_allclose(d["Nk"], e["Nk"], rtol=1e-10, atol=1e-13 * np.abs(e["Nk"]).max())
    assert all(abs(d[key] - e[key]) <= 1e-12 * abs(e[key]) for key in ("N", "E_kin", "E_pot", "E_int", "mu"))


def test_histogram_beyond_shared_memory(cuda):
    """More bins than a tile's shared memory holds run on the generic sweeps as before."""
    new, old, x = pair(30, torch.complex64, "real", nk_bins=12000)
    a = state(x, torch.complex64, 3)
    np.testing.assert_allclose(new.diagnostics(a, nk=True)["Nk"], old.diagnostics(a, nk=True)["Nk"], rtol=1e-12,
                               atol=1e-18)


def test_four_phases(cuda):
    """625 = 5^4 takes four phases; one imaginary-time step."""
    new, old, x = pair(625, torch.complex64, "imaginary")
    assert new.n == 625
    g = torch.exp(-torch.from_numpy(x).cuda() ** 2 / 2).to(torch.float32)
    a = (g[:, None, None] * g[None, :, None] * g[None, None, :]).to(torch.complex64)
    b = a.clone()
    new.step(a, 1)
    old.step(b, 1)
    worst = max(float(torch.linalg.vector_norm(a[i] - b[i])) for i in range(0, 625, 48))
    assert worst < TOL[torch.complex64] * float(torch.linalg.vector_norm(b[312])) * 4


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_batched_equals_alone(cuda, dtype):
    from gpe_simulator_b200.batch import Batch, Instance, initial_states
    from gpe_simulator_b200.plan import Plan
    insts = [Instance(n=n, simulation_range=10.0, beta=100.0 + n, dt=5e-4, static_expr="x**2+y**2+2*z**2")
             for n in (30, 50, 50, 105)]
    psis = initial_states(insts, dtype=dtype)
    alone = [p.clone() for p in psis]
    batch = Batch(insts, dtype=dtype)
    batch.bind(psis)
    batch.step(3)
    diag = batch.diagnostics()
    for i, (inst, p, q) in enumerate(zip(insts, alone, psis)):
        plan = Plan(inst.n, inst.x, inst.k, dtype=dtype, kind="imaginary", beta=inst.beta, dt=inst.dt,
                    static_expr=inst.static_expr)
        for _ in range(3):
            plan.step(p, 1)
        # (lagged against immediate renormalisation: the batch carries the scale into the next step)
        assert rel(p, q) < TOL[dtype]
        d = plan.diagnostics(q)
        assert [d[k] for k in ("N", "E_kin", "E_pot", "E_int", "E", "mu")] == list(diag[i])
