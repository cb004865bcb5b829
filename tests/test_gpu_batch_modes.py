"""Batches whose instances differ in their accuracy mode: each keeps its own."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# a side with compiled sweeps and one whose sweeps take it at run time; the instance that is
# created first decided for the whole group
@pytest.mark.parametrize("n", [32, 24])
@pytest.mark.parametrize("modes", [("", "exact_local"), ("exact_local", ""), ("", "generic_only", "exact_local")])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_modes_of_one_size(cuda, monkeypatch, n, modes, dtype):
    from gpe_simulator_b200 import batch as mod
    from gpe_simulator_b200.plan import Plan
    fill = mod._fill_desc

    def fill_mode(d, inst, *rest):
        fill(d, inst, *rest)
        if inst.mode:
            setattr(d, inst.mode, 1)

    monkeypatch.setattr(mod, "_fill_desc", fill_mode)
    insts = [mod.Instance(n=n, simulation_range=10.0, beta=300.0, dt=2e-3, static_expr="x**2+y**2+2*z**2")
             for _ in modes]
    for inst, mode in zip(insts, modes):
        inst.mode = mode
    psis = mod.initial_states(insts, dtype)
    alone = [p.clone() for p in psis]
    b = mod.Batch(insts, dtype)
    b.bind(psis)
    b.step(4)
    diag = b.diagnostics()
    for inst, mode, p, q, d in zip(insts, modes, alone, psis, diag):
        plan = Plan(n, inst.x, inst.k, dtype=dtype, kind="imaginary", beta=inst.beta, dt=inst.dt,
                    static_expr=inst.static_expr, **({mode: True} if mode else {}))
        plan.step(p, 4)
        assert torch.equal(p, q)
        want = plan.diagnostics(q)
        assert [want[k] for k in ("N", "E_kin", "E_pot", "E_int", "E", "mu")] == list(d)
