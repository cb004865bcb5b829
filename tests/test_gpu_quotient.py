"""The renormalisation's quotient of signed zeros and of components down to its remainder's
underflow (2^-968, about 3e-292)."""

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32])
def test_signed_zeros_and_small_components(cuda, n):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 8.0)
    p = Plan(n, x, k, dtype=torch.complex128, kind="imaginary", beta=0.0, dt=1e-3)
    rng = np.random.default_rng(n)
    v = rng.uniform(1.0, 10.0, (n, n, n, 2)) * 10.0 ** rng.integers(-290, 3, (n, n, n, 2)).astype(float)
    v *= rng.choice([-1.0, 1.0], v.shape)
    v[::3, ::2, :, 1] = -0.0
    v[1::3, ::2, :, 1] = 0.0
    a = torch.view_as_complex(torch.from_numpy(v)).cuda()
    want = v / np.sqrt(p.norm(a))
    p.normalise(a)
    got = torch.view_as_real(a).cpu().numpy()
    assert np.array_equal(got.view(np.int64), want.view(np.int64))
