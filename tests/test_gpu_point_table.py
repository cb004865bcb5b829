"""Dynamic potentials with z terms, tabulated per point, against the oracle and the generic
sweeps' per-point evaluation: hoisted and residual subtrees, budgets of slots, rows and z
values exceeded, both precisions, fused and single steps, diagnostics.

Tolerances: complex128 within 256 eps of the oracle after a few steps (x**2 as a product
instead of pow and hoisting differ from it by an ulp of the potential); complex64 within
2e-6 (rounding of ten sweeps)."""

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu
TOL = {torch.complex64: 2e-6, torch.complex128: 256 * np.finfo(np.float64).eps}

FORMULAS = [
    "0.5*sin(4*t)*z**2+0.3*x*z*cos(t)",
    "8*exp(-(x**2+y**2+(z-1.5*sin(4*t))**2)/0.64)+0.3*sin(10*t)*z**2",
    "z", "z*t", "x*y*z", "sqrt(abs(x*z))+tanh(y*z)-log(2+z*z*x*x)/3+tan(0.1*x*z)",
    # more t-only, row and z subtrees than there are slots
    "+".join(f"sin({k}*t)*cos({k}*x+0.1*t)*sin({k}*z)*x*z" for k in range(1, 13)),
    # deep nesting (the stack's bound) around a z term
    "+".join(["z*x"] + [f"0.01*(x+z)**{k}" for k in range(2, 8)]),
]


def rel(a, b):
    d = a.to(torch.complex128) - b.to(torch.complex128)
    return float(torch.linalg.vector_norm(d) / torch.linalg.vector_norm(b.to(torch.complex128)))


@pytest.mark.parametrize("expr", FORMULAS)
@pytest.mark.parametrize("n", [18, 32, 35])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_steps_match_generic_and_oracle(cuda, expr, n, dtype):
    from gpe_simulator_b200 import Plan
    from gpe_simulator_b200.plan import launch_count
    L, dt = 6.0, 1e-3
    x, k = ssf.get_grids(n, L)
    kw = dict(dtype=dtype, kind="real", beta=50.0, dt=dt, static_expr="x**2+2*z**2", dynamic_expr=expr)
    new, old = Plan(n, x, k, **kw), Plan(n, x, k, generic_only=True, **kw)
    psi0 = ssf.noisy_gaussian(x, seed=n)
    a = torch.from_numpy(psi0).to(dtype).cuda()
    start = a.cpu().numpy().astype(np.complex128)
    b = a.clone()
    before = launch_count(new)
    new.step(a, 4, 3)
    assert launch_count(new) - before == 5 * 4       # 17 sweeps and 3 table launches
    old.step(b, 4, 3)
    m = ssf.Model(n=n, simulation_range=L, kind="real", beta=50.0, dt=dt, static_expr="x**2+2*z**2", dynamic_expr=expr)
    want = torch.from_numpy(ssf.run(start, m, 4, step0=3)).cuda()
    assert rel(a, want) < TOL[dtype]
    assert rel(a, b) < 1.5 * TOL[dtype]
    # single steps at arbitrary times, a repeated time, and diagnostics after another call
    for t in (0.37, 0.37, 0.0):
        new.step_at(a, t)
        old.step_at(b, t)
    new.step(a, 1, 9)
    old.step(b, 1, 9)
    assert rel(a, b) < 3 * TOL[dtype]
    d, e = new.diagnostics(b, t=0.2, nk=True), old.diagnostics(b, t=0.2, nk=True)
    assert abs(d["E_pot"] - e["E_pot"]) <= 1e-6 * max(abs(e["E_pot"]), abs(e["N"])) if dtype == torch.complex64 \
        else abs(d["E_pot"] - e["E_pot"]) <= 1e-12 * max(abs(e["E_pot"]), abs(e["N"]))
    np.testing.assert_allclose(d["Nk"], e["Nk"], rtol=1e-9, atol=1e-13 * np.abs(e["Nk"]).max())
