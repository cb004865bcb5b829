"""Batches whose instances of one size differ in accuracy mode or shell binning."""

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


@pytest.mark.parametrize("bins", [(0, 3000), (3000, 0)])
def test_shell_binnings_of_one_size(cuda, monkeypatch, bins):
    """The Stockham x sweep of a prime side bins into shared memory behind its tile: the launch
    makes room for the instance with the most shells."""
    from gpe_simulator_b200 import batch as mod
    from gpe_simulator_b200.plan import Plan
    fill = mod._fill_desc

    def fill_bins(d, inst, *rest):
        fill(d, inst, *rest)
        d.nk_bins = inst.bins

    monkeypatch.setattr(mod, "_fill_desc", fill_bins)
    insts = [mod.Instance(n=13, simulation_range=10.0, beta=300.0, dt=2e-3, static_expr="x**2+y**2+2*z**2")
             for _ in bins]
    for inst, nb in zip(insts, bins):
        inst.bins = nb
    psis = mod.initial_states(insts, torch.complex64)
    b = mod.Batch(insts, torch.complex64)
    b.bind(psis)
    b.step(2)
    diag = b.diagnostics()
    for inst, q, d in zip(insts, psis, diag):
        plan = Plan(13, inst.x, inst.k, dtype=torch.complex64, kind="imaginary", beta=inst.beta, dt=inst.dt,
                    static_expr=inst.static_expr, nk_bins=inst.bins)
        want = plan.diagnostics(q)
        assert [want[k] for k in ("N", "E_kin", "E_pot", "E_int", "E", "mu")] == list(d)
