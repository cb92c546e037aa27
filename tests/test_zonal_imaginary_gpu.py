"""Synthesis takes the real part of s_n^0 alone.

The imaginary parts of the zonal coefficients are zero by convention and the
synthesis does not use them (g = Re F_0 + ...), so whatever they hold the
grid is the same, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["SHT_FP64", "SHT_MIXED"])
@pytest.mark.parametrize("N,I,J", [(21, 64, 32), (85, 256, 128), (170, 512, 256)])
@pytest.mark.parametrize("value", [1.0, 1e20, -1e300, np.inf, np.nan])
def test_ignored(dccm, synth, prec, N, I, J, value):
    s = synth.spectra(N, 2, seed=N)
    plan = dccm.ShtPlan(N, I, J, getattr(dccm, prec), 2)
    want = plan.inverse(s)
    s[1, :N + 1:3].imag = value
    assert np.array_equal(plan.inverse(s), want)


@pytest.mark.parametrize("value", [1e20, np.nan])
def test_ignored_at_any_address(dccm, cuda, synth, value):
    torch = cuda
    N, I, J = 42, 128, 64
    plan = dccm.ShtPlan(N, I, J, dccm.SHT_FP64, 1)
    s = synth.spectra(N, 1, seed=1)
    want = torch.zeros(1, J, I, dtype=torch.float64, device="cuda")
    got = torch.zeros_like(want)
    plan.inverse_dev(torch.from_numpy(s.view(np.float64)).cuda(), want, 1)
    s[0, :N + 1].imag = value
    moved = torch.empty(2 * plan.ncoef + 1, dtype=torch.float64, device="cuda")[1:]
    moved.copy_(torch.from_numpy(s.view(np.float64).ravel()))
    plan.inverse_dev(moved, got, 1)
    assert torch.equal(got, want)
