"""SPML's real layout read and written by the FP64 transforms themselves.

The smaller truncations take no permutation pass.  The arithmetic is that of
the native layout, so the results equal the permuted ones bit for bit, at
sizes on both sides of the rules (N, and N + 1 times the batch) and at the
edges of the packs' lane groups.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,I,J,batch", [(1, 64, 2, 3), (21, 64, 32, 70), (63, 192, 96, 33), (64, 192, 96, 2),
                                         (85, 256, 128, 95), (85, 256, 128, 96), (127, 384, 192, 1),
                                         (128, 384, 192, 5), (255, 768, 320, 2), (256, 768, 320, 2)])
def test_equals_permuted(dccm, cuda, N, I, J, batch):
    torch = cuda
    P = dccm.ShtPlan(N, I, J, max_batch=batch)
    gen = torch.Generator(device="cuda").manual_seed(N + batch)
    wa = torch.randn(batch, P.nwa, dtype=torch.float64, device="cuda", generator=gen)
    nan = float("nan")

    def new(*shape):
        return torch.full(shape, nan, dtype=torch.float64, device="cuda")

    spec, grid, want = new(batch, P.ncoef, 2), new(batch, J, I), new(batch, J, I)
    P.spec_from_wa_dev(wa, spec, batch)
    P.inverse_dev(spec, want, batch)
    P.xya_wa_dev(wa, grid, batch)
    assert torch.equal(grid, want)
    back, want_wa = new(batch, P.nwa), new(batch, P.nwa)
    P.forward_dev(want, spec, batch)
    P.wa_from_spec_dev(spec, want_wa, batch)
    P.wa_xya_dev(want, back, batch)
    assert torch.equal(back, want_wa)
    torch.cuda.synchronize()
    assert P.status()[0] == 0


def test_first_call_prepares_captured_calls(dccm, cuda):
    """A first call of any size sets the plan's tables up for captured ones."""
    torch = cuda
    N, I, J, most = 85, 256, 128, 120  # 120 field-levels are permuted, 2 are not
    P = dccm.ShtPlan(N, I, J, max_batch=most)
    gen = torch.Generator(device="cuda").manual_seed(5)
    wa = torch.randn(most, P.nwa, dtype=torch.float64, device="cuda", generator=gen)
    grid = torch.zeros(most, J, I, dtype=torch.float64, device="cuda")
    spec = torch.zeros(most, P.ncoef, 2, dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()
    P.xya_wa_dev(wa, grid, 2, st)
    st.synchronize()
    small = grid[:2].clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        P.xya_wa_dev(wa, grid, most, torch.cuda.current_stream())
        P.spec_from_wa_dev(wa, spec, most, torch.cuda.current_stream())
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(grid[:2], small)
    assert torch.equal(spec[:, 0, 0], wa[:, 0])
    assert P.status()[0] == 0
