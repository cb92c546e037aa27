"""Spectra at any address that holds doubles.

An FP64 plan takes spectra that start at an odd multiple of 8 bytes (a part
of a larger array of doubles) both ways, with the results of the same values at a
16-byte boundary: sizes on both sides of the packs' lane groups, ragged
batches, and through an ensemble.
"""
import pytest

pytestmark = pytest.mark.gpu


def _moved(torch, x):
    """x's values 8 bytes past a 16-byte boundary."""
    store = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)
    y = store[1:].view(x.shape)
    y.copy_(x)
    assert y.data_ptr() % 16 == 8 and x.data_ptr() % 16 == 0
    return y


@pytest.mark.parametrize("N,I,J,batch", [(1, 64, 2, 1), (21, 64, 32, 7), (63, 192, 96, 3), (64, 192, 96, 65),
                                         (127, 384, 192, 2), (128, 384, 192, 5)])
def test_fp64_takes_any_double(dccm, cuda, N, I, J, batch):
    torch = cuda
    P = dccm.ShtPlan(N, I, J, max_batch=batch)
    gen = torch.Generator(device="cuda").manual_seed(N)
    spec = torch.randn(batch, P.ncoef, 2, dtype=torch.float64, device="cuda", generator=gen)

    def new(*shape):
        return torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")

    want, got = new(batch, J, I), new(batch, J, I)
    P.inverse_dev(spec, want, batch)
    P.inverse_dev(_moved(torch, spec), got, batch)
    assert torch.equal(got, want)
    back, out = new(batch, P.ncoef, 2), _moved(torch, new(batch, P.ncoef, 2))
    P.forward_dev(want, back, batch)
    P.forward_dev(_moved(torch, want), out, batch)
    assert torch.equal(out, back)
    assert P.status()[0] == 0


def test_fp64_ensemble(dccm, cuda):
    torch = cuda
    sizes = [(21, 64, 32, 3), (42, 128, 64, 2)]
    E = dccm.Ensemble(sizes, dccm.SHT_FP64)
    n = [b for *_, b in sizes]
    spec = [torch.randn(b, (N + 1) * (N + 2) // 2, 2, dtype=torch.float64, device="cuda") for N, I, J, b in sizes]
    grids = [[torch.zeros(b, J, I, dtype=torch.float64, device="cuda") for N, I, J, b in sizes] for _ in range(2)]
    E.inverse_dev(spec, grids[0], n)
    E.inverse_dev([_moved(torch, s) for s in spec], grids[1], n)
    for a, b in zip(*grids):
        assert torch.equal(a, b)


@pytest.mark.parametrize("prec", ["SHT_MIXED", "SHT_MIXED_FP16"])
def test_others_refuse(dccm, cuda, prec):
    """Kernels that take spectra as 16-byte pairs: the host refuses other
    addresses, launches nothing on them, and the plan works on."""
    torch = cuda
    N, I, J, B = 42, 128, 64, 2
    P = dccm.ShtPlan(N, I, J, getattr(dccm, prec), B)
    E = dccm.Ensemble([(N, I, J, B)], getattr(dccm, prec))
    gen = torch.Generator(device="cuda").manual_seed(3)
    spec = torch.randn(B, P.ncoef, 2, dtype=torch.float64, device="cuda", generator=gen)
    grid = torch.zeros(B, J, I, dtype=torch.float64, device="cuda")
    wa = torch.zeros(B, P.nwa, dtype=torch.float64, device="cuda")
    moved = _moved(torch, spec)
    op = dccm.spec_op(dccm.SPEC_LAPLACIAN, 1.0)
    calls = {
        "inverse": lambda s: P.inverse_dev(s, grid, B),
        "forward": lambda s: P.forward_dev(grid, s, B),
        "ensemble inverse": lambda s: E.inverse_dev([s], [grid], [B]),
        "ensemble forward": lambda s: E.forward_dev([grid], [s], [B]),
        "from wa": lambda s: P.spec_from_wa_dev(wa, s, B),
        "to wa": lambda s: P.wa_from_spec_dev(s, wa, B),
        "operator in": lambda s: dccm.spec_apply_dev(N, op, s, spec, B),
        "operator out": lambda s: dccm.spec_apply_dev(N, op, spec, s, B),
    }
    keep = moved.clone()
    for name, call in calls.items():
        with pytest.raises(dccm.DccmError) as e:
            call(moved)
        assert e.value.status == -1, name
        call(spec.clone())
    torch.cuda.synchronize()
    assert torch.equal(moved, keep)
    assert P.status()[0] == 0
