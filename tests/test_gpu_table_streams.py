"""One plan on several streams: the tables of its dynamic potential are used by one call at a
time, and a captured call shares none."""

import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu
Z_FORM = "8*exp(-(x**2+y**2+(z-1.5*sin(4*t))**2)/0.64)+0.3*sin(10*t)*z**2"     # tabulated per point
XY_FORM = "8*exp(-((x-cos(4*t))**2+(y-sin(4*t))**2)/0.64)"                     # tabulated per line


def plan(n, expr, **kw):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 12.0)
    return Plan(n, x, k, dtype=torch.complex128, kind="real", beta=50.0, dt=1e-3, static_expr="x**2+2*z**2",
                dynamic_expr=expr, **kw), x


@pytest.mark.parametrize("n, expr", [(60, Z_FORM), (64, Z_FORM), (60, XY_FORM), (64, XY_FORM)])
def test_steps_and_diagnostics_side_by_side(cuda, n, expr):
    p, x = plan(n, expr)
    a = torch.from_numpy(ssf.noisy_gaussian(x, seed=1)).cuda()
    b = torch.from_numpy(ssf.noisy_gaussian(x, seed=2)).cuda()
    want_a, want_b = a.clone(), b.clone()
    p.step(want_a, 60, 0)
    p.step(want_b, 60, 500)
    e_pot = p.diagnostics(b, t=0.77)["E_pot"]
    torch.cuda.synchronize()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        a1, b1 = a.clone(), b.clone()
        torch.cuda.synchronize()
        with torch.cuda.stream(one):
            p.step(a1, 60, 0)
        with torch.cuda.stream(two):
            got = p.diagnostics(b, t=0.77)["E_pot"]
        with torch.cuda.stream(one):
            p.step_at(a1.clone(), 0.4)
        with torch.cuda.stream(two):
            p.step(b1, 60, 500)
        torch.cuda.synchronize()
        assert got == e_pot
        assert torch.equal(a1, want_a) and torch.equal(b1, want_b)


@pytest.mark.parametrize("n, expr", [(60, Z_FORM), (64, Z_FORM), (60, XY_FORM)])
def test_captured_steps(cuda, n, expr):
    p, x = plan(n, expr)
    g, _ = plan(n, expr, generic_only=True)
    psi0 = torch.from_numpy(ssf.noisy_gaussian(x, seed=3)).cuda()
    want, psi = psi0.clone(), psi0.clone()
    g.step(want, 2, 7)
    g.step_at(want, 0.3)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p.step(psi, 2, 7)
        p.step_at(psi, 0.3)
    psi.copy_(psi0)
    graph.replay()
    p.diagnostics(want, t=0.1)        # (a call of the plan beside the replay)
    torch.cuda.synchronize()
    assert torch.equal(psi, want)
