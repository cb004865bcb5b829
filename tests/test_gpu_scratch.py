"""Device memory that diagnostics take: the work state, and histograms only where n(k) is asked for."""

import pytest
import torch

from oracle import ssf

pytestmark = pytest.mark.gpu
SLACK = 6 << 20          # allocation granules (2 MB) of the buffers counted


# run-time-length sweeps whose z tiles outnumber the x tiles, and a compiled side
@pytest.mark.parametrize("n, dtype", [(200, torch.complex128), (216, torch.complex64), (256, torch.complex64)])
def test_diagnostics_scratch(cuda, n, dtype):
    from gpe_simulator_b200 import Plan
    x, k = ssf.get_grids(n, 12.0)
    p = Plan(n, x, k, dtype=dtype, kind="real", beta=10.0, dt=1e-3, nk_bins=1024)
    a = torch.ones((n, n, n), dtype=dtype, device=cuda)
    state = a.numel() * a.element_size()
    lines = 16 if dtype == torch.complex64 else 8
    hists = n * -(-n // lines) * 1024 * 8 * 5 // 4       # one per x tile (tiles of a row evened out)
    p.norm(a)
    free = torch.cuda.mem_get_info()[0]
    p.diagnostics(a)
    plain = free - torch.cuda.mem_get_info()[0]
    assert plain <= state + SLACK
    p.diagnostics(a, nk=True)
    assert free - torch.cuda.mem_get_info()[0] <= state + hists + SLACK
