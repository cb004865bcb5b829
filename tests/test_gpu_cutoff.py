"""Modes on the cutoff sphere: kept or dropped as the reference's k^2 > k_cut^2 in NumPy's
rounding, whatever sweeps a side takes and whichever axis the components lie on."""

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu


def tied_cutoff(k):
    """A cutoff whose square falls between the rounded k^2 of modes of one exact length."""
    m = np.rint(k / k[1]).astype(np.int64)
    exact = (m[:, None, None] ** 2 + m[None, :, None] ** 2 + m[None, None, :] ** 2)
    kk = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    best = None
    for s in np.unique(exact):
        v = np.unique(kk[exact == s])
        for c in np.sqrt(v[:-1]):
            cut = float(c) * float(c)
            kept = int((kk[exact == s] <= cut).sum())
            split = min(kept, int((exact == s).sum()) - kept)
            if split and (best is None or split > best[0]):
                best = (split, float(c))
    return best[1], kk, exact


# Stockham (one radix), run-time-length and compiled x sweeps
@pytest.mark.parametrize("n, dtype", [(13, torch.complex128), (16, torch.complex64), (18, torch.complex128),
                                      (35, torch.complex64), (35, torch.complex128), (32, torch.complex64),
                                      (48, torch.complex128), (64, torch.complex64)])
@pytest.mark.parametrize("L", [10.0, 7.3])
def test_modes_on_the_sphere(cuda, n, dtype, L):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, L)
    cut, kk, exact = tied_cutoff(k)
    rng = np.random.default_rng(n)
    f = rng.standard_normal((n, n, n)) + 1j * rng.standard_normal((n, n, n)) + 3.0
    psi = torch.from_numpy(np.fft.ifftn(f)).to(dtype).cuda()
    p = Plan(n, x, k, dtype=dtype, kind="real", beta=0.0, dt=1e-3, kinetic_coeff=0.0, k_cut=cut)
    p.step(psi, 1)
    got = np.abs(np.fft.fftn(psi.cpu().numpy().astype(np.complex128)))
    keep = kk <= cut * cut
    assert 0 < keep.sum() < keep.size and len(np.unique(keep[exact == exact[keep].max()])) == 2
    # a kept mode is about 3 in size, a dropped one a rounding of the transforms
    assert np.array_equal(got > 0.5 * np.abs(f), keep)
