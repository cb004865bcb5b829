"""Modes of exactly the cutoff's length on the run-time-length x sweeps: kept or dropped by the
rounding of fma(kx, kx, fma(ky, ky, kz kz)), the same in both precisions."""

from fractions import Fraction

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c)))


def tied_cutoff(k):
    """The modes of one exact length, and a cutoff between their rounded k^2."""
    m = np.rint(k / k[1]).astype(np.int64)
    exact = m[:, None, None] ** 2 + m[None, :, None] ** 2 + m[None, None, :] ** 2
    length, count = np.unique(exact, return_counts=True)
    for s in length[np.argsort(-count)]:
        ties = np.argwhere(exact == s)
        kk = np.array([fma(k[i], k[i], fma(k[j], k[j], k[l] * k[l])) for i, j, l in ties])
        for c in np.sqrt(np.unique(kk)):
            kept = kk <= float(c) * float(c)
            if 0 < kept.sum() < len(kept):
                return float(c), exact, s, ties, kept


@pytest.mark.parametrize("n", [18, 35, 75])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_modes_on_the_sphere(cuda, n, dtype):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 10.0)
    cut, exact, s, ties, kept = tied_cutoff(k)
    want = exact < s
    want[tuple(ties.T)] = kept
    rng = np.random.default_rng(n)
    f = np.exp(2j * np.pi * rng.random((n, n, n)))            # every mode of size 1
    psi = torch.from_numpy(np.fft.ifftn(f)).to(dtype).cuda()
    p = Plan(n, x, k, dtype=dtype, kind="real", beta=0.0, dt=1e-3, kinetic_coeff=0.0, k_cut=cut)
    p.step(psi, 1)
    got = np.abs(np.fft.fftn(psi.cpu().numpy().astype(np.complex128)))
    assert np.array_equal(got > 0.5, want)
