"""Sums over the state keep every element: a few values of 1e8 among ones, whose squares (1e16)
leave no bits for a one that is added to them in plain FP64."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
BIG = 1.0e8


def plan(n, dtype, **kw):
    from gpe_simulator_b200 import Plan
    x = np.arange(n, dtype=np.float64)            # dx = 1: the sums are exact integers
    k = 2 * np.pi * np.fft.fftfreq(n, 1.0)
    return Plan(n, x, k, dtype=dtype, kind="real", beta=1.0, dt=1e-3, **kw)


def state(n, dtype, every):
    psi = torch.ones((n, n, n), dtype=dtype)
    psi[:, :, ::every] = BIG
    big = n * n * len(range(0, n, every))
    return psi.cuda(), big, n ** 3 - big


def ulps(got, want):
    """Distance from an exact integer sum in units of its last place as a double."""
    return abs(int(got) - want) / float(np.spacing(float(want)))


# half a unit from rounding the whole sum, and up to one from its partial sums: t equal tiles
# round to half a unit of sum / t each, in the same direction, t * ulp(sum / t) / 2 <= ulp(sum)
BOUND = 1.5


@pytest.mark.parametrize("n", [13, 48, 60, 64, 105])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_norm(cuda, n, dtype):
    a, big, ones = state(n, dtype, 12)
    assert ulps(plan(n, dtype).norm(a), big * 10 ** 16 + ones) <= BOUND


@pytest.mark.parametrize("n", [13, 60, 105])     # Stockham and run-time-length sweeps
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_diagnostics(cuda, n, dtype):
    a, big, ones = state(n, dtype, n)             # z = 0 only: the first element of every line's first butterfly
    d = plan(n, dtype, static_expr="2").diagnostics(a)
    assert ulps(d["N"], big * 10 ** 16 + ones) <= BOUND
    assert ulps(d["E_pot"], 2 * (big * 10 ** 16 + ones)) <= BOUND
