"""A plan with thousands of n(k) bins: the same shells, and little more time to make."""

import time

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu


def make(n, bins):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 10.0)
    torch.cuda.synchronize()
    t = time.perf_counter()
    p = Plan(n, x, k, dtype=torch.complex64, kind="real", beta=1.0, dt=1e-3, nk_bins=bins)
    return p, time.perf_counter() - t, k


@pytest.mark.parametrize("bins", [2, 50, 777, 5000])
@pytest.mark.parametrize("n", [13, 32, 60])
def test_counts(cuda, n, bins):
    p, _, k = make(n, bins)
    width = np.sqrt(3.0) * (n // 2) * abs(k[1] - k[0]) / (bins - 1)
    kk = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    shell = np.minimum(np.floor(np.sqrt(kk) / width + 0.5).astype(np.int64), bins - 1)
    a = torch.ones((n, n, n), dtype=torch.complex64, device=cuda)
    assert np.array_equal(p.diagnostics(a, nk=True)["counts"], np.bincount(shell.ravel(), minlength=bins))


def test_time(cuda):
    """Least of 15: ten halvings per bin, 5000 bins, at most 20 ns each on the host, is 1 ms."""
    few, many = (min(make(32, bins)[1] for _ in range(15)) for bins in (50, 5000))
    assert many - few < 1e-3
