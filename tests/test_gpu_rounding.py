"""Rounding of complex128 steps: without potential, interaction and kinetic factor a step is
the transforms there and back, so what it does to the state is its error."""

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu


# radices with a split of two coprime factors (6, 10, 12, 14, 15), primes, compiled sides
@pytest.mark.parametrize("n", [35, 36, 42, 48, 60, 66, 77, 84, 96, 105])
def test_round_trips_are_as_exact_as_the_generic_sweeps(cuda, n):
    """The generic sweeps' radices are at most 5, 7, 11, 13, 8 and 16 with table twiddles.  Both
    errors are sums of some hundred independent roundings per value, whose spread over
    orders of operation is about 10%."""
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 24.0)
    psi = torch.from_numpy(ssf.noisy_gaussian(x, sigma=1.4, seed=n)).cuda()
    err = []
    for generic in (False, True):
        p = Plan(n, x, k, dtype=torch.complex128, kind="real", beta=0.0, dt=1e-3, kinetic_coeff=0.0, generic_only=generic)
        a = psi.clone()
        p.step(a, 5)
        err.append(float(torch.linalg.vector_norm(a - psi) / torch.linalg.vector_norm(psi)))
    assert err[0] <= 1.15 * err[1]
    assert err[1] < 16 * np.finfo(np.float64).eps
