"""Mixed-path transforms of batches that leave CTAs and 16-byte runs partly filled.

A field-level's result does not depend on the batch it comes in, so every
ragged batch equals its field-levels transformed one by one, bit for bit: the
last run of a batch, CTAs of 8 and 16 warps, one and two row pairs a warp, and
plans larger than the call.
"""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["SHT_MIXED", "SHT_MIXED_FP16"])
@pytest.mark.parametrize("N,I,J,batches", [(21, 64, 32, (1, 3, 6, 9)), (127, 384, 192, (2, 5, 27)),
                                           (255, 768, 384, (1, 5, 9)), (341, 1024, 512, (3, 5, 9, 11))])
def test_ragged_batch(prec, N, I, J, batches):
    pkg = importlib.import_module("dennou-ccm_gb300")
    most = max(batches)
    P = pkg.ShtPlan(N, I, J, precision=getattr(pkg, prec), max_batch=most)
    gen = torch.Generator(device="cuda").manual_seed(N)
    grid = torch.randn(most, J, I, dtype=torch.float64, device="cuda", generator=gen)
    grid *= torch.logspace(-3, 3, most, dtype=torch.float64, device="cuda")[:, None, None]
    st = torch.cuda.current_stream()

    def new(*shape):
        return torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")

    spec, back = new(most, P.ncoef, 2), new(most, J, I)
    for b in range(most):
        P.forward_dev(grid[b:b + 1], spec[b:b + 1], 1, st)
        P.inverse_dev(spec[b:b + 1], back[b:b + 1], 1, st)
    assert torch.isfinite(spec).all() and torch.isfinite(back).all()
    for n in batches:
        s, g = new(n, P.ncoef, 2), new(n, J, I)
        P.forward_dev(grid[:n], s, n, st)
        assert torch.equal(s, spec[:n]), n
        P.inverse_dev(spec[:n], g, n, st)
        assert torch.equal(g, back[:n]), n
    torch.cuda.synchronize()
    assert P.status()[0] == 0
