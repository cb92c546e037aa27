"""Mixed-path forward FFT with rows prefetched ahead: the same results for every batch and alignment.

Large batches take two row pairs a warp and, with rows of 512 points or more,
prefetch the grid rows of a CTA further on, if the grid is 16-byte aligned.  A prefetch changes no result, so
the whole batch, the same batch at an 8-byte offset (no prefetch) and its
parts (one row pair a warp) are equal bit for bit.  The batch sizes leave the
last CTAs partly filled and the prefetches of the last CTAs past the end.
"""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,I,J,batch", [(21, 64, 32, 1203), (42, 128, 64, 601), (170, 512, 256, 61),
                                         (341, 1024, 512, 13)])
def test_forward_same_with_prefetch(N, I, J, batch):
    pkg = importlib.import_module("dennou-ccm_gb300")
    P = pkg.ShtPlan(N, I, J, precision=pkg.SHT_MIXED, max_batch=batch)
    gen = torch.Generator(device="cuda").manual_seed(N)
    n = batch * J * I
    store = torch.empty(n + 1, dtype=torch.float64, device="cuda")
    store[:n] = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
    grid = store[:n].view(batch, J, I)
    assert grid.data_ptr() % 16 == 0
    st = torch.cuda.current_stream()

    def forward(g, b):
        out = torch.full((b, P.ncoef, 2), float("nan"), dtype=torch.float64, device="cuda")
        P.forward_dev(g, out, b, st)
        return out

    whole = forward(grid, batch)
    part = 3
    for b0 in (0, batch // 2, batch - part):
        assert torch.equal(forward(grid[b0:b0 + part].contiguous(), part), whole[b0:b0 + part])
    moved = torch.empty(n + 1, dtype=torch.float64, device="cuda")[1:]
    moved.copy_(store[:n])
    assert moved.data_ptr() % 16 == 8
    assert torch.equal(forward(moved.view(batch, J, I), batch), whole)
    torch.cuda.synchronize()
    assert P.status()[0] == 0
