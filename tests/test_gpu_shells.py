"""Modes per shell and shell sums: the square-root-free shell rule against NumPy's expression,
for shells wide and narrow, bins that one, two, four and eight copies of the histogram fit
for, and bins only global memory holds.  Counts are integers: equal.  A shell's sum has FP64
rounding only (order): 1e-12."""

import numpy as np
import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu


def shells(k, n, nbins):
    dk = abs(k[1] - k[0])
    w = np.sqrt(3.0) * (n // 2) * dk / (nbins - 1) if nbins else dk
    nb = nbins or int(np.floor(np.sqrt(3) * (n // 2) + 0.5)) + 1
    kk = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    return np.minimum(np.floor(np.sqrt(kk) / w + 0.5).astype(np.int64), nb - 1), nb


@pytest.mark.parametrize("n,nbins", [(32, 0), (32, 2), (32, 7), (32, 400), (32, 3000), (35, 0), (35, 256), (48, 1000),
                                     (50, 1500), (50, 2500), (50, 12000), (13, 0), (128, 256)])
@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128])
def test_counts_and_sums(cuda, n, nbins, dtype):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 7.3)
    plan = Plan(n, x, k, dtype=dtype, kind="real", beta=0.0, dt=1e-3, nk_bins=nbins)
    sh, nb = shells(k, n, nbins)
    rng = np.random.default_rng(n + nbins)
    f = torch.from_numpy(rng.standard_normal((n, n, n)) + 1j * rng.standard_normal((n, n, n))).to(dtype).cuda()
    dx3, m = (x[1] - x[0]) ** 3, n ** 3
    if nbins <= 3000:
        w = torch.view_as_real(f).double().square().sum(-1).cpu().numpy()
        want = np.bincount(sh.ravel(), w.ravel(), nb) * dx3 / m
        nk, counts = plan.shells(f)
        assert np.array_equal(counts, np.bincount(sh.ravel(), minlength=nb))
        np.testing.assert_allclose(nk, want, rtol=1e-12, atol=1e-15 * want.max())
    d = plan.diagnostics(f, nk=True)
    assert np.array_equal(d["counts"], np.bincount(sh.ravel(), minlength=nb))
    psi_k = plan.fft(f)
    w = torch.view_as_real(psi_k).double().square().sum(-1).cpu().numpy()
    want = np.bincount(sh.ravel(), w.ravel(), nb) * dx3 / m
    np.testing.assert_allclose(d["Nk"], want, rtol=1e-12 if dtype == torch.complex128 else 1e-5,
                               atol=1e-12 * want.max())
